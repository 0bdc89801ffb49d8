"""Paths that leave the padding slices out of their work: the fused batch mode, and the start of
the dual from the primal with its repair of missed rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fused_batch_of_padded_slice_counts():
    """Members of 3, 5, 6, 9, 39 and 90 slices (4, 8, 8, 12, 40 and 92 in memory), and of 5 and 39 in images too
    small for the padding, against each alone."""
    from graptor_gb300.solver import Batch, Problem
    sizes = [(17, 3, 1), (100, 5, 1), (91, 2, 3), (74, 9, 1), (36, 13, 3), (24, 45, 2), (18, 5, 1), (15, 13, 3)]
    specs, data = [], []
    for k, (N, Nz, C) in enumerate(sizes):
        ang = np.deg2rad(np.linspace(-80, 85, 9 + k))
        specs.append(dict(dim=3, N=N, Nz=Nz, C=C, nd=19 + k, angles=ang, alpha=(4.0, 1.0), mu=[0.2] * C,
                          discrepancy="KL" if k % 2 else "L2", normest=11.0))
        data.append(np.abs(np.random.default_rng(k).standard_normal((Nz * C, ang.size, 19 + k))).astype(np.float32))
    with Batch(specs) as b:
        for k, f in enumerate(data):
            b[k].set_data(f)
        b.set_mode(1)
        b.run(11).synchronize()
        for k, f in enumerate(data):
            with Problem(**specs[k]) as p:
                p.set_data(f).run(11).synchronize()
                for name in ("u", "ku", "lambda", "v", "w", "p"):
                    np.testing.assert_array_equal(b[k].get(name), p.get(name), err_msg=f"{k} {name}")


@pytest.mark.parametrize("Nz,full", [(3, 4), (5, 8), (6, 8), (37, 40)])
def test_dual_from_primal_of_padded_slice_counts(Nz, full):
    """2-D slices do not see each other: the first Nz of `full` slices give the same iterates in both
    problems, after a repair of missed rays too, and nothing of the padding reaches the movement."""
    from graptor_gb300.solver import Problem
    N, nd = 100, 110
    ang = np.deg2rad(np.linspace(-80, 85, 13))
    rng = np.random.default_rng(Nz)
    f = np.abs(rng.standard_normal((full, ang.size, nd))).astype(np.float32)
    u = rng.random((full, N, N)).astype(np.float32)
    u[:, :, :40] = 0  # rays that the image misses
    got = []
    for n in (Nz, full):
        with Problem(2, N, n, 1, nd, ang, (4, 1), [0.2], "KL", "TGV", "UNCORR", 1.0, 11.0) as p:
            p.set_data(f[:n])
            p.set("w", np.ones((3, n, N, N), np.float32))  # leaves the staging buffer full
            p.set("w", np.zeros((3, n, N, N), np.float32))
            p.set("u", u[:n])
            p.get("v")
            p.dual_from_primal(repair=True)
            a = [p.get(k)[..., :Nz, :, :] for k in ("u", "lambda")]
            p.snapshot()
            p.run(4).synchronize()
            b = {k: p.get(k) for k in ("u", "p", "v", "w", "lambda")}
            got.append(a + [b[k][..., :Nz, :, :] for k in b])
            if n == Nz:
                p.restart()
                p.snapshot()
                before = b
                p.run(3).synchronize()
                primal, dual = p.movement()
                d = {k: float(((p.get(k).astype(np.float64) - before[k]) ** 2).sum()) for k in b}
                assert abs(primal - np.sqrt(d["u"] + d["p"])) <= 1e-12 * primal
                assert abs(dual - np.sqrt(d["v"] + d["w"] + d["lambda"])) <= 1e-12 * dual
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("case", [(2, 100, 5, 1, "TV", "UNCORR"), (3, 91, 2, 3, "TGV", "FROB"), (3, 84, 1, 7, "TGV", "UNCORR"),
                                  (3, 74, 9, 1, "TV", "FROB"), (3, 37, 13, 3, "TGV", "UNCORR"), (3, 36, 13, 3, "TGV", "FROB"),
                                  (3, 30, 11, 5, "TGV", "FROB"), (3, 17, 3, 1, "TGV", "FROB")],
                         ids=lambda c: "-".join(map(str, c)))
def test_padding_slices_reach_no_result(case):
    """5, 6, 7, 9, 39 and 55 slices in images from the size at which they are padded, and 3; iterates against the
    CPU oracle, the movement against the fields read back."""
    from graptor_gb300 import phantom
    from graptor_gb300.solver import Problem
    from oracle import oracle as O
    dim, N, Nz, C, reg, cpl = case
    nd, nang, ne = N, 9, 16.0
    rng = np.random.default_rng(N + Nz)
    ang = phantom.angles_deg(nang)
    ofs = O.radon_struct(ang, N, nd)
    f = phantom.poisson(O.radon(np.abs(rng.standard_normal((C * Nz, N, N))).astype(np.float32), ofs, nd), 200.0, 1)
    mu = rng.uniform(0.1, 0.5, C)
    fields = ("u", "p", "v", "w", "lambda") if reg == "TGV" else ("u", "v", "lambda")
    with Problem(dim, N, Nz, C, nd, ang, (3.0, 1.5), mu, "KL", reg, cpl, 1.0, ne) as p:
        p.set_data(f)
        assert C * Nz == 3 or p.tuning["fwd_cfg"] > 0  # padded: more than the one shape
        p.run(7).synchronize()
        a = {k: p.get(k).astype(np.float64) for k in fields}
        p.snapshot()
        p.run(5).synchronize()
        b = {k: p.get(k).astype(np.float64) for k in fields}
        ku = p.get("ku")
        primal, dual = p.movement()
    d = {k: float(((a[k] - b[k]) ** 2).sum()) for k in fields}
    assert abs(primal - np.sqrt(d["u"] + d.get("p", 0.0))) <= 1e-12 * primal
    assert abs(dual - np.sqrt(d["v"] + d.get("w", 0.0) + d["lambda"])) <= 1e-12 * dual
    o = O.Solver(dim, N, Nz, C, nd, ofs, f, (3.0, 1.5), mu, ne, O.KL, O.TGV if reg == "TGV" else O.TV,
                 {"UNCORR": O.UNCORR, "FROB": O.FROB}[cpl], stepsize=1.0).run(12)
    for got, want in ((b["u"], o.u), (b["lambda"], o.lam), (ku, o.ku), (b["v"], o.v)):
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
