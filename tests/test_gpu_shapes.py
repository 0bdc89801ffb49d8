"""Projector launch shapes on geometries where their tables and tiles can go wrong: images
whose side is not a multiple of the tile, detectors wider and narrower than the
image, rays along the axes and the diagonals, slice counts around a warp's chunk.
Every shape must give the one-pixel / one-ray shapes' iterates bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEOMETRIES = [
    # N, nd, angles in degrees, Nz, C
    (17, 17, (0, 30, 45, 90, 135, 180, 270), 4, 1),
    (18, 31, (-85, -45, 0, 1, 44.9, 89.99, 90.01), 16, 1),
    (23, 9, (10, 20, 45, 100, 170), 33, 4),
    (5, 5, (3, 93), 128, 2),
    (31, 2, (0, 12, 77, 90), 65, 4),
    (1, 1, (0, 45), 8, 1),
    (33, 40, tuple(range(-90, 90, 9)), 96, 4),
]


def _iterates(N, nd, deg, Nz, C, shapes):
    from graptor_gb300.solver import Problem
    rng = np.random.default_rng(N * 1000 + nd)
    ang = np.deg2rad(np.asarray(deg, np.float64))
    f = np.abs(rng.standard_normal((C * Nz, ang.size, nd))).astype(np.float32)
    out = []
    with Problem(3, N, Nz, C, nd, ang, (4, 1), [0.2] * C, normest=11.0, autotune=False) as p:
        for fwd, bp in shapes:
            p.set_data(f, feasible=False)
            p.set_tuning(fwd, bp)
            p.run(5).synchronize()
            out.append({k: p.get(k) for k in ("u", "ku", "lambda")})
    return out


@pytest.mark.parametrize("geometry", GEOMETRIES, ids=lambda g: f"{g[0]}-{g[1]}-{g[3] * g[4]}")
def test_back_projection_shapes_agree(geometry):
    got = _iterates(*geometry, shapes=[(0, 4)] + [(0, b) for b in (9, 10, 11, 12, 18, 19)])
    for g in got[1:]:
        for k in g:
            np.testing.assert_array_equal(g[k], got[0][k], err_msg=k)


@pytest.mark.parametrize("geometry", GEOMETRIES, ids=lambda g: f"{g[0]}-{g[1]}-{g[3] * g[4]}")
def test_forward_projection_shapes_agree(geometry):
    got = _iterates(*geometry, shapes=[(0, 4)] + [(s, 4) for s in (5, 6, 7, 9, 10, 11)])
    for g in got[1:]:
        for k in g:
            np.testing.assert_array_equal(g[k], got[0][k], err_msg=k)


def test_pair_shapes_keep_infinities_to_their_rays():
    """A pixel that only one ray of a pair takes must not reach the other ray through its
    zero weight when it is infinite or NaN."""
    from graptor_gb300.solver import Problem
    N, Nz, C = 24, 8, 1
    ang = np.deg2rad(np.array([20.0, 63.0, 90.0, 131.0]))
    f = np.abs(np.random.default_rng(8).standard_normal((Nz, ang.size, N))).astype(np.float32)
    u = np.random.default_rng(9).random((Nz, N, N)).astype(np.float32)
    u[0, 5, 7], u[3, 20, 2], u[6, 11, 11] = np.inf, np.nan, -np.inf
    got = []
    with Problem(3, N, Nz, C, N, ang, (4, 1), [0.2], normest=11.0, autotune=False) as p:
        for fwd in (0, 10, 11):
            p.set_data(f)
            p.set_tuning(fwd, 4)
            p.set("ubar", u)
            p.run(1).synchronize()
            got.append(p.get("ku"))
    assert not np.isfinite(got[0]).all()
    for g in got[1:]:
        np.testing.assert_array_equal(g, got[0])


@pytest.mark.parametrize("dim,N,nd,Nz", [(2, 33, 33, 1), (2, 40, 70, 2), (2, 64, 64, 1), (2, 20, 5, 4)])
def test_staged_forward_projection_matches_oracle(dim, N, nd, Nz):
    """One, two and four slices take the staged kernel; detectors around the 32 rays of a
    block and around chunks of its entries."""
    from graptor_gb300 import phantom
    from graptor_gb300.solver import Problem
    from oracle import oracle as O
    ang = phantom.angles_deg(9)
    ofs = O.radon_struct(ang, N, nd)
    f = np.abs(np.random.default_rng(N).standard_normal((Nz, ang.size, nd))).astype(np.float32)
    with Problem(dim, N, Nz, 1, nd, ang, (3.0, 1.5), [0.3], "L2", "TGV", "UNCORR", 1.0, 13.0) as p:
        p.set_data(f).run(20).synchronize()
        u, lam = p.get("u"), p.get("lambda")
    o = O.Solver(dim, N, Nz, 1, nd, ofs, f, (3.0, 1.5), np.array([0.3]), 13.0, O.L2, O.TGV, O.UNCORR, stepsize=1.0).run(20)
    assert np.linalg.norm(u - o.u) <= 1e-5 * np.linalg.norm(o.u)
    assert np.linalg.norm(lam - o.lam) <= 1e-5 * np.linalg.norm(o.lam)


@pytest.mark.parametrize("N,nd,deg", [(1, 1, (10,)), (19, 19, (0, 45, 90, 135)), (40, 23, (-70, -20, 3, 70, 89.99)),
                                      (64, 90, tuple(range(20, 161, 10))), (33, 33, tuple(range(0, 180)))])
def test_operator_norm_matches_fp64_power_iteration(N, nd, deg):
    """The fixed-point projectors of the norm estimate (rounding about 1e-13 in the weights)
    against the power iteration with the exact FP64 matrix; it stops when two
    consecutive sums agree to 1e-8.  More than 128 angles: a second chunk of the table."""
    from graptor_gb300.solver import Problem
    from oracle import fp64 as F
    ang = np.deg2rad(np.asarray(deg, np.float64))
    R = F.radon_matrix(ang, N, nd)
    x = np.ones(N * N)
    for _ in range(30):
        s = x.sum()
        x = R.T @ (R @ (x / s))
    with Problem(2, N, 1, 1, nd, ang, (4, 1), [0.2], "L2", "TGV", "UNCORR", autotune=False) as p:
        p.set_data(np.ones((1, ang.size, nd), np.float32))
        ne = p.scalars["normest"]
    want = np.sqrt(x.sum())
    assert abs(ne - want) <= 1e-6 * want, (ne, want)


@pytest.mark.parametrize("dim,N,nd,Nz,C,reg,cpl,disc", [
    (2, 33, 33, 1, 1, "TGV", "UNCORR", "KL"), (2, 30, 41, 2, 1, "TV", "FROB", "L2"), (2, 17, 17, 1, 4, "TGV", "FROB", "L2"),
    (3, 21, 21, 7, 1, "TGV", "FROB", "KL"), (3, 24, 19, 5, 3, "TGV", "UNCORR", "L2"), (3, 26, 26, 8, 4, "TV", "FROB", "KL")])
def test_two_launch_iteration_equals_separate_launches(dim, N, nd, Nz, C, reg, cpl, disc):
    """The two-launch form of small problems (whichever form the tuning picks) against schedule
    0, with the primal weight and the precise primal mode, over runs that end inside and at a graph chunk."""
    from graptor_gb300.solver import Problem
    ang = np.deg2rad(np.linspace(-80, 85, 13))
    f = np.abs(np.random.default_rng(N).standard_normal((C * Nz, ang.size, nd))).astype(np.float32)
    fields = ("u", "ubar", "v", "lambda", "ku") + (("p", "pbar", "w") if reg == "TGV" else ())
    got = []
    for forced in (False, True):
        with Problem(dim, N, Nz, C, nd, ang, (4, 1), [0.2] * C, disc, reg, cpl, 1.0, 11.0) as p:
            if forced:
                p.set_schedule(0)
            p.set_data(f)
            p.set_precise_primal()
            p.run(5).synchronize()
            p.set_primal_weight(3.0)
            p.run(37).synchronize()
            got.append({k: p.get(k) for k in fields + ("ulo",)})
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
