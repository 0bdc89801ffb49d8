"""Performance cases: the work a user of graptor_gb300 has it do, through its public
entry points.

Kinds of case:

* ``iterate``   -- a resident :class:`Problem` advanced by ``iters`` primal-dual
  iterations, u, K u and lambda read back on the device (2-D and 3-D, every
  coupling, both data terms, TGV and TV).
* ``call``      -- one call of the drop-in ``Reconstructionapproach3d`` with host
  arrays: set-up, data upload, operator norm, iterations, float64 results.
* ``gap``       -- the body of a solve to a gap tolerance: iterations, then the FP64
  primal-dual gap.
* ``subsample`` -- the two-resolution solver.
* ``predict``   -- the warm-start network applied to one volume.
* ``train``     -- one training step of that network (forward, backward, Adam).
"""
import ctypes
import math
import os

import numpy as np
import torch

import graptor_gb300
from graptor_gb300 import _lib as L
from graptor_gb300 import solver
from graptor_gb300 import radon_tgv_primal_dual_3d as r3
from graptor_gb300.radon_tgv_primal_dual_3dsubsample import Subsampling
from graptor_gb300.warmstart import UNet3D

r3.progress = False
WEIGHTS = os.path.join(os.path.dirname(graptor_gb300.__file__), "weights", "unet_tgv_kl_c2_p500.npz")
PEAKS = (1e4, 20.0, 20.0, 20.0)       # Poisson peak counts: channel 0 dense, the others sparse
MU = {"KL": (0.2, 5e-4, 5e-4, 5e-4), "L2": (0.2, 0.02, 0.02, 0.02)}
ALPHA = (4.0, 1.0)
METHOD = {"FROB": "Frobenius 3D Reconstruction", "UNCORR": "Uncorrelated 3D Reconstruction",
          "NUCL": "Nuclear 3D Reconstruction"}


def _iterate(name, dim, N, Nz, C, nang, data, reg, cpl, iters, step=1.0):
    d = {"kind": "iterate", "dim": dim, "N": N, "Nz": Nz, "C": C, "nang": nang, "data": data, "reg": reg,
         "coupling": cpl, "step": step, "iters": iters}
    return dict(d, name=name) if name else d


def listed():
    return [
        # one 2-D slice, the single-channel workload: latency of an iteration
        _iterate("slice_2d_128", 2, 128, 1, 1, 60, "KL", "TGV", "UNCORR", 100),
        # several coupled 2-D slices of an odd detector, quadratic data term, TV
        _iterate("slices_2d_odd_tv", 2, 177, 5, 3, 45, "L2", "TV", "FROB", 50),
        # the small 3-D problem that is solved to a gap tolerance (10^5 iterations)
        _iterate("volume_64x16x2", 3, 64, 16, 2, 71, "KL", "TGV", "FROB", 100),
        # odd image, slice and channel counts (one chunk of a ragged section)
        _iterate("volume_odd_101x13x3", 3, 101, 13, 3, 45, "L2", "TGV", "UNCORR", 50, 2.0),
        # nuclear-norm coupling
        _iterate("volume_nuclear_128x30x3", 3, 128, 30, 3, 71, "L2", "TGV", "NUCL", 8),
        # the headline workload: 3-D, four channels, Frobenius coupling
        _iterate("volume_256x60x4", 3, 256, 60, 4, 71, "KL", "TGV", "FROB", 20),
        # a large section: state well beyond the L2 cache
        _iterate("volume_512x96x4", 3, 512, 96, 4, 141, "KL", "TGV", "FROB", 4),
        # a whole reconstruction call as the command line makes it for one section
        {"name": "call_128x32x2", "kind": "call", "N": 128, "Nz": 32, "C": 2, "nang": 71, "data": "KL", "reg": "TGV",
         "coupling": "FROB", "step": 1.0, "iters": 100},
        # iterations between two gap checks of a solve to a tolerance (quadratic data
        # term: the gap is finite from the start)
        {"name": "gap_128x32x2", "kind": "gap", "N": 128, "Nz": 32, "C": 2, "nang": 71, "data": "L2", "reg": "TGV",
         "coupling": "FROB", "step": 1.0, "iters": 50, "before": 150},
        # a channel measured at half the resolution of the other
        {"name": "subsample_128x30", "kind": "subsample", "N": 128, "Nz": 30, "nang": 71, "data": "KL", "reg": "TGV",
         "coupling": "FROB", "iters": 16},
        # the network's prediction for one 128^2 x 32 volume of two channels
        {"name": "predict_128x32", "kind": "predict", "B": 1, "D": 32, "H": 128, "W": 128},
        # one training step on four random crops
        {"name": "train_4x16x64x64", "kind": "train", "B": 4, "D": 16, "H": 64, "W": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(N, Nz, C, nang, iters):
    return N * N * Nz * C * (nang + 60.0) * iters


def draw(rng):
    kind = rng.choice(["iterate"] * 7 + ["call", "gap", "subsample", "predict", "train"])
    most = _cost(512, 96, 4, 141, 4)
    if kind == "predict" or kind == "train":
        B = rng.randint(1, 2) if kind == "predict" else rng.randint(1, 4)
        D, H, Wd = 4 * rng.randint(2, 8), 4 * rng.randint(8, 32), 16 * rng.randint(2, 8)
        if kind == "train":
            D, H, Wd = min(D, 16), min(H, 64), min(Wd, 64)
        return {"kind": kind, "B": B, "D": D, "H": H, "W": Wd}
    while True:
        nang = rng.randint(30, 141)
        data, reg = rng.choice(["KL", "L2"]), rng.choice(["TGV", "TGV", "TGV", "TV"])
        cpl = rng.choice(["FROB", "FROB", "UNCORR"])
        step = rng.choice([1.0, 1.0, 2.0])
        if kind == "iterate":
            dim = rng.choice([2, 3, 3, 3])
            N, C = _log_int(rng, 48, 512), rng.randint(1, 4)
            Nz = _log_int(rng, 1, 12) if dim == 2 else _log_int(rng, 4, 96)
            if dim == 3 and rng.random() < 0.12:
                cpl, data = "NUCL", "L2"
            iters = rng.choice([4, 10, 16, 20, 50, 100])
            if cpl == "NUCL":
                iters = min(iters, 10)
            if _cost(N, Nz, C, nang, iters) > most or N * N * Nz * C > 512 * 512 * 96 * 4:
                continue
            return _iterate(None, dim, N, Nz, C, nang, data, reg, cpl, iters, step if dim == 3 else 1.0)
        N, Nz, C = rng.randint(48, 192), rng.randint(4, 48), rng.randint(1, 3)
        if kind == "call":
            return {"kind": kind, "N": N, "Nz": Nz, "C": C, "nang": nang, "data": data, "reg": reg, "coupling": cpl,
                    "step": step, "iters": rng.choice([20, 50, 100])}
        if kind == "gap":
            return {"kind": kind, "N": min(N, 128), "Nz": min(Nz, 32), "C": C, "nang": min(nang, 90), "data": "L2",
                    "reg": "TGV", "coupling": cpl, "step": 1.0, "iters": 50, "before": 150}
        return {"kind": kind, "N": 2 * (N // 2), "Nz": 2 * (Nz // 2), "nang": nang, "data": data, "reg": reg,
                "coupling": cpl, "iters": rng.choice([8, 16])}


# ---------------------------------------------------------------------------- inputs
def _angles(nang):
    """Tilt series of +-70 degrees in the solver's convention (radians, shifted by pi / 2)."""
    return np.linspace(-70.0, 70.0, nang) * np.pi / 180.0 + np.pi / 2.0


def _volume(N, Nz, C, seed):
    """Ellipsoid phantom [N*N][C*Nz] (slice fastest) on the GPU: the channels share the
    ellipsoids, channel 0 carries all of them, the others a few each."""
    rng = np.random.default_rng(seed)
    g = (torch.arange(N, device="cuda", dtype=torch.float32) - (N - 1) / 2.0) / (N / 2.0)
    gz = (torch.arange(Nz, device="cuda", dtype=torch.float32) - (Nz - 1) / 2.0) / max(Nz / 2.0, 1.0)
    Y, X = torch.meshgrid(g, g, indexing="ij")
    vol = torch.zeros((N, N, C, Nz), device="cuda")
    for k in range(12):
        cx, cy = rng.uniform(-0.5, 0.5, 2)
        cz, cc = rng.uniform(-0.4, 0.4), rng.uniform(0.3, 0.9)
        a, b = rng.uniform(0.08, 0.4, 2)
        th = rng.uniform(0, math.pi)
        val = rng.uniform(0.1, 1.0, C)
        keep = rng.random(C) < 0.25
        keep[0] = True
        keep[1:] |= k == 0
        xr = (X - cx) * math.cos(th) + (Y - cy) * math.sin(th)
        yr = (Y - cy) * math.cos(th) - (X - cx) * math.sin(th)
        m = ((xr / a) ** 2 + (yr / b) ** 2)[:, :, None] + (((gz - cz) / cc) ** 2)[None, None, :] <= 1.0
        for c in range(C):
            if keep[c]:
                vol[:, :, c, :][m] = float(val[c])
    return vol.reshape(N * N, C * Nz)


def _sinogram(N, Nz, C, nang, seed):
    """Poisson data [C*Nz, nang, N] (host float32): line integrals of seeded ellipsoids (the
    channels share them, channel 0 carries all, the others a few each) with counts of the
    channel's peak."""
    rng = np.random.default_rng(seed)
    ang = torch.from_numpy(_angles(nang)).cuda().reshape(1, nang, 1)
    t = ((torch.arange(N, device="cuda", dtype=torch.float64) - (N - 1) / 2.0) / (N / 2.0)).reshape(1, 1, N)
    gz = ((torch.arange(Nz, device="cuda", dtype=torch.float64) - (Nz - 1) / 2.0) / max(Nz / 2.0, 1.0)).reshape(Nz, 1, 1)
    g = torch.zeros((C, Nz, nang, N), device="cuda")
    for k in range(12):
        cx, cy = rng.uniform(-0.5, 0.5, 2)
        cz, cc = rng.uniform(-0.4, 0.4), rng.uniform(0.3, 0.9)
        a, b = rng.uniform(0.08, 0.4, 2)
        th = rng.uniform(0, math.pi)
        val = rng.uniform(0.1, 1.0, C)
        keep = rng.random(C) < 0.25
        keep[0] = True
        keep[1:] |= k == 0
        sz = (1.0 - ((gz - cz) / cc) ** 2).clamp_min(0.0)  # the slice's squared scale of both half axes
        r2 = (a * torch.cos(ang - th)) ** 2 + (b * torch.sin(ang - th)) ** 2
        tau = t - cx * torch.cos(ang) - cy * torch.sin(ang)
        length = (N / 2.0) * 2 * a * b * (sz * r2 - tau * tau).clamp_min(0.0).sqrt() / r2
        for c in range(C):
            if keep[c]:
                g[c] += float(val[c]) * length.float()
    gen = torch.Generator("cuda").manual_seed(seed + 104729)
    for c in range(C):
        scale = PEAKS[c] / g[c].max().clamp_min(1e-20)
        g[c] = torch.poisson(g[c] * scale, generator=gen) / PEAKS[c]
    return g.reshape(C * Nz, nang, N).cpu().numpy()


def _subs_data(case, seed):
    N, Nz, nang = case["N"], case["Nz"], case["nang"]
    f = _sinogram(N, Nz, 2, nang, seed).reshape(2, Nz, nang, N)
    f1 = f[1]
    lo = 0.25 * (f1[0::2, :, 0::2] + f1[1::2, :, 0::2] + f1[0::2, :, 1::2] + f1[1::2, :, 1::2])
    refnew, refold = [(N - 1) / 2.0, (Nz - 1) / 2.0], [(N / 2 - 1) / 2.0, (Nz / 2 - 1) / 2.0]
    return f[0], np.ascontiguousarray(lo, np.float32), refold, refnew


def _network_input(case, seed):
    """(x bfloat16 [B][2][D][H][W], target float32): normalised phantom volumes as the
    network meets them, the input blurred by noise, the target clean."""
    B, D, H, Wd = case["B"], case["D"], case["H"], case["W"]
    N = max(H, Wd)
    gen = torch.Generator("cuda").manual_seed(seed)
    t = torch.stack([_volume(N, D, 2, 1000 * seed + b).reshape(N, N, 2, D).permute(2, 3, 0, 1)[:, :, :H, :Wd]
                     for b in range(B)]).contiguous()
    t = t / t.mean(dim=(2, 3, 4), keepdim=True).clamp_min(1e-3)
    x = (t + 0.1 * t.std() * torch.randn(t.shape, generator=gen, device="cuda")).clamp_min(0)
    return x.to(torch.bfloat16), t


def _problem(case, seed):
    dim, N, Nz, C, nang = case.get("dim", 3), case["N"], case["Nz"], case["C"], case["nang"]
    prob = solver.Problem(dim, N, Nz, C, N, _angles(nang), ALPHA, MU[case["data"]][:C], case["data"], case["reg"],
                          case["coupling"], case["step"])
    prob.set_data(_sinogram(N, Nz, C, nang, seed))
    return prob


def _device_fields(prob, fields):
    return {k: torch.empty(prob._shape(k), device="cuda") for k in fields}


def _read(handle, out):
    for k, t in out.items():
        L.check(L.lib().gt_get_state_device(handle, L.FIELDS[k], ctypes.c_void_p(t.data_ptr())))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        prob = _problem(case, seed)
        out = _device_fields(prob, ("u", "ku", "lambda"))
        torch.cuda.synchronize()
        return {"case": case, "prob": prob, "out": out}
    if kind == "gap":
        prob = _problem(case, seed)
        prob.run(case["before"]).synchronize()
        return {"case": case, "prob": prob}
    if kind == "call":
        N, Nz, C, nang = case["N"], case["Nz"], case["C"], case["nang"]
        f = _sinogram(N, Nz, C, nang, seed).reshape(C, Nz, nang, N)
        return {"case": case, "sino": [np.ascontiguousarray(f[c].transpose(1, 0, 2)) for c in range(C)]}
    if kind == "subsample":
        f0, f1, refold, refnew = _subs_data(case, seed)
        N, Nz = case["N"], case["Nz"]
        ang = _angles(case["nang"])
        sub = Subsampling(N, Nz, 1, 1, N // 2, Nz // 2, ang, ang, ALPHA, MU[case["data"]][:2], 2.0, refold, refnew,
                          case["data"], case["reg"], case["coupling"])
        sub.set_data(f0, f1)
        fields = {"u": (2 * Nz, N, N), "v": (3, 2 * Nz, N, N)}
        out = {k: torch.empty(s, device="cuda") for k, s in fields.items()}
        torch.cuda.synchronize()
        return {"case": case, "sub": sub, "out": out}
    net = UNet3D.load(WEIGHTS)
    x, target = _network_input(case, seed)
    out = torch.empty_like(target)
    if kind == "train":
        net.train_step(x, target, lr=0.0)  # the buffers of a training run; no weight moves
        net.step_count = 0
        net.m.zero_()
        net.v.zero_()
    else:
        net.buffers(case["B"], case["D"], case["H"], case["W"])
    torch.cuda.synchronize()
    return {"case": case, "net": net, "x": x, "target": target, "out": out}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "iterate":
        prob = state["prob"]
        prob.run(case["iters"])
        return _read(prob._h, state["out"])
    if kind == "gap":
        return state["prob"].solve_to_gap(tol=0.0, check_every=case["iters"], max_iters=case["iters"])
    if kind == "call":
        u, ku = r3.Reconstructionapproach3d(state["sino"], _angles(case["nang"]), ALPHA,
                                            MU[case["data"]][:case["C"]], case["iters"], 0, [0, 0.1], case["step"],
                                            case["data"], METHOD[case["coupling"]], case["reg"], [0, 1, [0]])
        return {"solution": u, "sinogram": ku}
    if kind == "subsample":
        sub = state["sub"]
        sub.run(case["iters"])
        return _read(L.lib().gt_subs_problem(sub._h), state["out"])
    net, x, out = state["net"], state["x"], state["out"]
    if kind == "predict":
        net.residual_base(x, out)
        return net.forward(x, out)
    loss = net.train_step(x, state["target"], lr=1e-4)
    return {"loss": loss, "grad": net.grad, "weights": net.master}


# ---------------------------------------------------------------------------- work
def _solver_work(dim, N, Nz, C, nang, reg, iters):
    """Per iteration: every field the update rules read and write once (K u, lambda and f
    per bin, u, ubar, p, pbar, v, w per voxel-channel), two taps per pixel and angle
    in each projection."""
    V, S = float(N) * N * Nz * C, float(N) * nang * Nz * C
    per_v = {(3, "TGV"): 172, (2, "TGV"): 108, (3, "TV"): 48, (2, "TV"): 40}[(dim, reg)]
    per_f = {(3, "TGV"): 180, (2, "TGV"): 90, (3, "TV"): 45, (2, "TV"): 35}[(dim, reg)]
    return {"bytes": iters * (per_v * V + 16 * S), "flops": iters * (8.0 * V * nang + per_f * V + 12 * S)}


def _conv_flops(case):
    vox = case["B"] * case["D"] * case["H"] * case["W"]
    c1, c2, c3 = 16, 32, 64
    full = 27 * (2 * c1 + c1 * c1 + (c1 + c2) * c1 + c1 * c1) + c1 * 2
    half = 27 * (c1 * c2 + c2 * c2 + (c2 + c3) * c2 + c2 * c2)
    quarter = 27 * (c2 * c3 + c3 * c3)
    return 2.0 * vox * (full + half / 8.0 + quarter / 64.0)


def work(case):
    kind = case["kind"]
    if kind in ("iterate", "gap", "call"):
        w = _solver_work(case.get("dim", 3), case["N"], case["Nz"], case["C"], case["nang"], case["reg"], case["iters"])
        V, S = float(case["N"]) ** 2 * case["Nz"] * case["C"], float(case["N"]) * case["nang"] * case["Nz"] * case["C"]
        if kind == "gap":    # two checks: u, p, v, w, lambda and f read once each
            w["bytes"] += 2 * (4 * (13 if case["reg"] == "TGV" else 4) * V + 8 * S)
            w["flops"] += 2 * (8.0 * V * case["nang"] + 150 * V)
        if kind == "call":   # data in, float64 results out
            w["bytes"] += 8 * V + 12 * S
        return w
    if kind == "subsample":
        return _solver_work(3, case["N"], case["Nz"], 2, case["nang"], case["reg"], case["iters"])
    vox = float(case["B"] * case["D"] * case["H"] * case["W"])
    if kind == "predict":
        return {"bytes": 12 * vox + 2 * 353730, "flops": _conv_flops(case)}
    return {"bytes": 12 * vox + 28 * 353730, "flops": 3 * _conv_flops(case)}


# ---------------------------------------------------------------------------- exact values
# The iteration in float64, written from the model: u, p primal, v, w, lambda dual,
# fields [.., C, Nz, N(y), N(x)].
def _matrix(angles, N, nd):
    """Projection matrix [nang*nd, N*N] of the hat weights (1 - |t - i|)+, float64, on the GPU."""
    ang = np.asarray(angles, np.float64)
    X, Y = np.cos(ang), np.sin(ang)
    vert = np.abs(X) < 1.0 / (10 * nd)
    X[vert] = 0.0
    Y[vert] = np.round(np.sin(ang[vert]))
    off = (nd - 1) / 2.0 - X * (N - 1) / 2.0 - Y * (N - 1) / 2.0
    yy, xx = torch.meshgrid(*(torch.arange(N, device="cuda", dtype=torch.float64),) * 2, indexing="ij")
    pix = torch.arange(N * N, device="cuda")
    rows, cols, vals = [], [], []
    for j in range(ang.size):
        t = (xx * X[j] + yy * Y[j] + off[j]).reshape(-1)
        fl = t.floor()
        for k, w in ((fl, 1.0 - (t - fl)), (fl + 1, t - fl)):
            ok = (k >= 0) & (k < nd) & (w > 0)
            rows.append(j * nd + k[ok].long())
            cols.append(pix[ok])
            vals.append(w[ok])
    idx = torch.stack([torch.cat(rows), torch.cat(cols)])
    val = torch.cat(vals)
    shape = (ang.size * nd, N * N)
    R = torch.sparse_coo_tensor(idx, val, shape).coalesce().to_sparse_csr()
    RT = torch.sparse_coo_tensor(idx.flip(0), val, shape[::-1]).coalesce().to_sparse_csr()
    return R, RT


def _fwd(a, dim, h=1.0):
    """Forward difference along an axis, zero at its end."""
    o = torch.zeros_like(a)
    n = a.shape[dim]
    o.narrow(dim, 0, n - 1).copy_((a.narrow(dim, 1, n - 1) - a.narrow(dim, 0, n - 1)) / h)
    return o


def _fwd_adj(a, dim, h=1.0):
    """Minus the adjoint of _fwd."""
    o = a / h
    n = a.shape[dim]
    o.narrow(dim, n - 1, 1).zero_()
    if n > 1:
        o.narrow(dim, 1, n - 1).sub_(a.narrow(dim, 0, n - 1) / h)
    return o


def _bwd(a, dim, h=1.0):
    """Backward difference along an axis, zero at its start."""
    o = torch.zeros_like(a)
    n = a.shape[dim]
    o.narrow(dim, 1, n - 1).copy_((a.narrow(dim, 1, n - 1) - a.narrow(dim, 0, n - 1)) / h)
    return o


def _bwd_adj(a, dim, h=1.0):
    """Minus the adjoint of _bwd."""
    o = -a / h
    n = a.shape[dim]
    o.narrow(dim, 0, 1).zero_()
    if n > 1:
        o.narrow(dim, 0, n - 1).add_(a.narrow(dim, 1, n - 1) / h)
    return o


class _Exact:
    def __init__(self, dim, N, Nz, C, angles, data, reg, coupling, step, mu, lsqr=None):
        self.dim, self.N, self.Nz, self.C, self.nang = dim, N, Nz, C, len(angles)
        self.data, self.reg, self.coupling = data, reg, coupling
        self.ax = [3, 2, 1][:dim]  # x, y, z axes of [C, Nz, y, x]
        self.h = [1.0, 1.0, step][:dim]
        self.R, self.RT = _matrix(angles, N, N)
        self.mu = torch.tensor(list(mu), dtype=torch.float64, device="cuda").reshape(C, 1, 1, 1)
        self.sigma = self.tau = 1.0 / math.sqrt(lsqr or (17.0 if dim == 3 else 0.5 * (18 + math.sqrt(33))))
        q = 1.4142 ** 2
        self.b = [1, 1, 1, q, q, 1.0 if coupling == "UNCORR" else q] if dim == 3 else \
            [1, 1, q if coupling == "UNCORR" else 4.0]
        self.m = [1, 1, 1, 2, 2, 2] if dim == 3 else [1, 1, 2]
        self.pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)] if dim == 3 else [(0, 0), (1, 1), (0, 1)]

        def z(k):
            return torch.zeros((k, C, Nz, N, N), dtype=torch.float64, device="cuda")
        self.u, self.ubar = z(1)[0], z(1)[0]
        self.v = z(dim)
        if reg == "TGV":
            self.p, self.pbar, self.w = z(dim), z(dim), z(len(self.pairs))

    def proj(self, u):
        C, Nz, N = u.shape[0], u.shape[1], u.shape[2]
        return (self.R @ u.reshape(C * Nz, N * N).t().contiguous()).t().reshape(C, Nz, self.nang, N)

    def back(self, g):
        C, Nz = g.shape[0], g.shape[1]
        return (self.RT @ g.reshape(C * Nz, -1).t().contiguous()).t().reshape(C, Nz, self.N, self.N)

    def norm_estimate(self):
        """sqrt of the power iteration's sum ratio on R^T R from the all-ones image."""
        x = torch.ones((self.N * self.N, 1), dtype=torch.float64, device="cuda")
        s = 0.0
        for _ in range(31):
            s, prev = float(x.sum()), s
            if abs(s - prev) <= 1e-12 * s:
                break
            x = self.RT @ (self.R @ (x / s))
        return math.sqrt(s)

    def setup(self, f, ne):
        self.f, self.ne = f, ne
        self.a0, self.a1 = ALPHA[0] / ne ** 2, ALPHA[1] / ne ** 2
        self.lam = torch.zeros_like(f)

    def ball(self, x, radius, weights, coupling):
        if coupling == "NUCL":
            A = x.permute(2, 3, 4, 1, 0)
            U, s, Vh = torch.linalg.svd(A, full_matrices=False)
            A = (U * s.clamp_max(radius)[..., None, :]) @ Vh
            return A.permute(4, 3, 0, 1, 2).contiguous()
        wt = torch.tensor(weights, dtype=torch.float64, device="cuda").reshape(-1, 1, 1, 1, 1)
        n2 = (wt * x * x).sum(0, keepdim=True)
        if coupling != "UNCORR":
            n2 = n2.sum(1, keepdim=True)
        return x / (n2.sqrt() / radius).clamp_min(1.0)

    def eps(self, p):
        d = [[_bwd(p[k], a, h) for a, h in zip(self.ax, self.h)] for k in range(self.dim)]
        return torch.stack([d[i][i] if i == j else 0.5 * (d[j][i] + d[i][j]) for i, j in self.pairs])

    def eps_div(self, w):
        at = {}
        for k, (i, j) in enumerate(self.pairs):
            at[i, j] = at[j, i] = k
        return torch.stack([sum(_bwd_adj(w[at[i, j]], self.ax[j], self.h[j]) for j in range(self.dim))
                            for i in range(self.dim)])

    def grad(self, u):
        return torch.stack([_fwd(u, a, h) for a, h in zip(self.ax, self.h)])

    def div(self, v):
        return sum(_fwd_adj(v[k], self.ax[k], self.h[k]) for k in range(self.dim))

    def dual_data(self, lam, ku, f, mu):
        sg = self.sigma / self.ne
        s = lam + sg * ku
        if self.data == "KL":
            t = s - mu
            return s - 0.5 * (t + (t * t + 4 * sg * f * mu).sqrt())
        return (s - sg * f) * (mu / (self.sigma + mu))

    def data_step(self):
        """lambda from ubar; returns R^T lambda."""
        self.ku = self.proj(self.ubar)
        self.lam = self.dual_data(self.lam, self.ku, self.f, self.mu)
        return self.back(self.lam)

    def iterate(self, n):
        tgv = self.reg == "TGV"
        for _ in range(n):
            self.v = self.v + self.sigma * (self.grad(self.ubar) - (self.pbar if tgv else 0.0))
            self.v = self.ball(self.v, self.a1, [1.0] * self.dim, self.coupling)
            if tgv:
                self.w = self.w + self.sigma * self.eps(self.pbar)
                self.w = self.ball(self.w, self.a0, self.b, "UNCORR" if self.coupling == "UNCORR" else "FROB")
            kt = self.data_step() / self.ne
            un = (self.u + self.tau * (self.div(self.v) - kt)).clamp_min(0.0)
            self.ubar, self.u = 2 * un - self.u, un
            if tgv:
                pn = self.p + self.tau * (self.v + self.eps_div(self.w))
                self.pbar, self.p = 2 * pn - self.p, pn
        return self

    def feasible(self, f):
        """Data zeroed on the bins that no pixel reaches."""
        one = self.R @ torch.ones((self.N * self.N, 1), dtype=torch.float64, device="cuda")
        return f * (one.reshape(self.nang, self.N) > 0)

    def gap(self):
        ne, mu, f = self.ne, self.mu, self.f
        ru = self.proj(self.u)
        if self.data == "KL":
            t = torch.where(f > 0, f * (f / ru.clamp_min(0)).log(), torch.zeros_like(f))
            data = float((mu * (torch.where(f > 0, ru - f, ru) + t)).sum() / ne)
            fstar = float(torch.where(f > 0, -(mu * f) * torch.log1p(-self.lam / mu), torch.zeros_like(f)).sum() / ne)
        else:
            data = float((mu / (2 * ne ** 2) * (ru - f) ** 2).sum())
            fstar = float((self.lam * f / ne).sum() + (self.lam ** 2 / (2 * mu)).sum())

        def norms(e, wt):
            n2 = (torch.tensor(wt, dtype=torch.float64, device="cuda").reshape(-1, 1, 1, 1, 1) * e * e).sum(0)
            return n2.sqrt() if self.coupling == "UNCORR" else n2.sum(0).sqrt()
        reg = self.a1 * float(norms(self.grad(self.u) - self.p, [1.0] * self.dim).sum())
        reg += self.a0 * float(norms(self.eps(self.p), [m * m / b for m, b in zip(self.m, self.b)]).sum())
        vt = -self.eps_div(self.w)
        top = float(norms(vt, [1.0] * self.dim).max())
        theta = min(1.0, self.a1 / top) if top > 0 else 1.0
        umax = float(self.u.max())
        U = 2 * umax if umax > 0 else 1.0
        box = U * float((self.back(self.lam) / ne - theta * self.div(vt)).clamp_max(0.0).sum())
        P, D = reg + data, box - fstar
        return {"primal": P, "dual": D, "gap": P - D, "relative": (P - D) / abs(P), "theta": theta, "U": U,
                "data": data, "fstar": fstar, "iterations": None}


class _ExactSubs(_Exact):
    """Channel 0 on the fine detector, channel 1 binned by M (area weights of the coarse
    pixels over (detector, slice), the same for every angle)."""

    def binning(self, refold, refnew, nd1, nz1):
        N, Nz = self.N, self.Nz
        M = torch.zeros((nz1 * nd1, Nz * N), dtype=torch.float64)
        for j in range(nz1):
            for i in range(nd1):
                x, y = 2.0 * (i - refold[0]) + refnew[0], 2.0 * (j - refold[1]) + refnew[1]
                for jj in range(math.ceil(y - 1.499999), math.floor(y + 1.499999) + 1):
                    for ii in range(math.ceil(x - 1.499999), math.floor(x + 1.499999) + 1):
                        wx = min(x + 1 - ii, 0.5) + min(ii - x + 1, 0.5)
                        wy = min(y + 1 - jj, 0.5) + min(jj - y + 1, 0.5)
                        M[j * nd1 + i, min(max(jj, 0), Nz - 1) * N + min(max(ii, 0), N - 1)] += wx * wy / 4.0
        self.M, self.nd1, self.nz1 = M.cuda(), nd1, nz1

    def bin(self, g):   # [Nz, nang, N] -> [nz1, nang, nd1]
        t = g.permute(0, 2, 1).reshape(self.Nz * self.N, self.nang)
        return (self.M @ t).reshape(self.nz1, self.nd1, self.nang).permute(0, 2, 1)

    def unbin(self, g):
        t = g.permute(0, 2, 1).reshape(self.nz1 * self.nd1, self.nang)
        return (self.M.t() @ t).reshape(self.Nz, self.N, self.nang).permute(0, 2, 1)

    def norm_estimate(self):
        x = torch.ones((2, self.Nz, self.N, self.N), dtype=torch.float64, device="cuda")
        nrm = 0.0
        for _ in range(30):
            nrm = float(x.norm())
            g = self.proj(x / nrm)
            x = self.back(torch.stack([g[0], self.unbin(self.bin(g[1]))]))
        return math.sqrt(nrm)

    def setup(self, f, ne):
        self.f0, self.f1, self.ne = f[0], f[1], ne
        self.a0, self.a1 = ALPHA[0] / ne ** 2, ALPHA[1] / ne ** 2
        self.l0, self.l1 = torch.zeros_like(f[0]), torch.zeros_like(f[1])

    def data_step(self):
        g = self.proj(self.ubar)
        self.l0 = self.dual_data(self.l0, g[0], self.f0, float(self.mu[0]))
        self.l1 = self.dual_data(self.l1, self.bin(g[1]), self.f1, float(self.mu[1]))
        return self.back(torch.stack([self.l0, self.unbin(self.l1)]))


def _exact_problem(case, seed):
    dim, N, Nz, C, nang = case.get("dim", 3), case["N"], case["Nz"], case["C"], case["nang"]
    e = _Exact(dim, N, Nz, C, _angles(nang), case["data"], case["reg"], case["coupling"], case["step"],
               MU[case["data"]][:C])
    f = torch.from_numpy(_sinogram(N, Nz, C, nang, seed)).cuda().double().reshape(C, Nz, nang, N)
    e.setup(e.feasible(f), e.norm_estimate())
    return e


def _exact_network(case, seed):
    """Output of the network in float64 (bfloat16 weights and input, no rounding of
    activations) with its parameters as leaves."""
    net = UNet3D.load(WEIGHTS)
    F = torch.nn.functional
    flat = net.master.double().cpu().numpy()
    wts = {}
    for name, (o, ob, ci, co, k) in net.offsets.items():
        w = torch.from_numpy(flat[o:ob]).reshape(co, ci, k, k, k).cuda().to(torch.bfloat16).double()
        wts[name] = (w.requires_grad_(), torch.from_numpy(flat[ob:ob + co]).cuda().requires_grad_())
    x, target = _network_input(case, seed)

    def conv(name, a, act=True):
        w, b = wts[name]
        y = F.conv3d(a, w, b, padding=w.shape[2] // 2)
        return F.relu(y) if act else y

    def up(a):
        return F.interpolate(a, scale_factor=2, mode="nearest")
    xd = x.double()
    e1 = conv("enc1b", conv("enc1a", xd))
    e2 = conv("enc2b", conv("enc2a", F.avg_pool3d(e1, 2)))
    bt = conv("botb", conv("bota", F.avg_pool3d(e2, 2)))
    d2 = conv("dec2b", conv("dec2a", torch.cat([e2, up(bt)], 1)))
    d1 = conv("dec1b", conv("dec1a", torch.cat([e1, up(d2)], 1)))
    return net, wts, xd + conv("head", d1, False), target


def exact(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        if case["coupling"] == "NUCL":
            # the reference's spectral projection is its own formula, not the exact one
            return None
        e = _exact_problem(case, seed).iterate(case["iters"])
        S, N, nang = case["C"] * case["Nz"], case["N"], case["nang"]
        return {"u": e.u.reshape(S, N, N), "ku": e.ku.reshape(S, nang, N), "lambda": e.lam.reshape(S, nang, N)}
    if kind == "call":
        if case["coupling"] == "NUCL":
            return None
        e = _exact_problem(case, seed).iterate(case["iters"])
        return {"solution": e.u.permute(0, 3, 2, 1).contiguous(), "sinogram": e.ku.permute(0, 2, 1, 3).contiguous()}
    if kind == "gap":
        return _exact_problem(case, seed).iterate(case["before"] + case["iters"]).gap()
    if kind == "subsample":
        f0, f1, refold, refnew = _subs_data(case, seed)
        N, Nz, nang = case["N"], case["Nz"], case["nang"]
        e = _ExactSubs(3, N, Nz, 2, _angles(nang), case["data"], case["reg"], case["coupling"], 1.0,
                       MU[case["data"]][:2], 36.0)
        e.binning(refold, refnew, N // 2, Nz // 2)
        one = (e.R @ torch.ones((N * N, 1), dtype=torch.float64, device="cuda")).reshape(nang, N) > 0
        e.setup((torch.from_numpy(f0).cuda().double() * one, torch.from_numpy(f1).cuda().double() * one[:, :N // 2]),
                e.norm_estimate())
        e.iterate(case["iters"])
        return {"u": e.u.reshape(2 * Nz, N, N), "v": e.v.reshape(3, 2 * Nz, N, N)}
    with torch.set_grad_enabled(kind == "train"):
        net, wts, out, target = _exact_network(case, seed)
        if kind == "predict":
            return out
        loss = ((out - target.double()) ** 2).mean()
        loss.backward()
    grad = torch.zeros(net.nparams, dtype=torch.float64, device="cuda")
    for name, (o, ob, ci, co, k) in net.offsets.items():
        w, b = wts[name]
        grad[o:ob], grad[ob:ob + co] = w.grad.reshape(-1), b.grad
    step = 1e-4 * grad / (grad.abs() + 1e-8)  # Adam's first step: m / (sqrt(v) + eps), bias-corrected
    return {"loss": loss.detach(), "grad": grad, "weights": net.master.double() - step}
