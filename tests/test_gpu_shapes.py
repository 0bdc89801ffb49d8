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
