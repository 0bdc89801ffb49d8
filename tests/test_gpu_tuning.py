"""Forced launch shapes: what gt_get_tuning returns is accepted by gt_set_tuning for every slice
count, and every projector shape gives the same iterates on slice counts that are padded in memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(N, nd, nang, Nz, C, **kw):
    from graptor_gb300.solver import Problem
    rng = np.random.default_rng(N + Nz)
    f = np.abs(rng.standard_normal((C * Nz, nang, nd))).astype(np.float32)
    ang = np.deg2rad(np.linspace(-80, 85, nang))
    return f, Problem(3, N, Nz, C, nd, ang, (4, 1), [0.2] * C, normest=11.0, **kw)


@pytest.mark.parametrize("autotune", [True, False])
@pytest.mark.parametrize("Nz,C", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (2, 3), (13, 3), (16, 2), (45, 2)])
def test_tuned_shapes_can_be_set(Nz, C, autotune):
    f, p = _problem(100, 22, 9, Nz, C, autotune=autotune)
    with p:
        p.set_data(f)
        t = p.tuning
        p.set_tuning(t["fwd_cfg"], t["bp_cfg"])
        assert {k: p.tuning[k] for k in ("fwd_cfg", "bp_cfg")} == {k: t[k] for k in ("fwd_cfg", "bp_cfg")}
        for bad in ((20, 0), (0, 20), (-1, 0), (0, -1)):
            with pytest.raises(ValueError):
                p.set_tuning(*bad)


@pytest.mark.parametrize("N,nd,Nz,C", [(93, 25, 3, 2), (37, 3, 13, 3), (24, 23, 45, 2), (21, 31, 43, 3), (20, 14, 65, 2)])
def test_projector_shapes_agree_on_padded_slice_counts(N, nd, Nz, C):
    """6, 39, 90, 129 and 130 slices (8, 40, 92, 132 and 132 in memory), an odd and an even number of bins,
    pairs of bins fewer than a group and not a multiple of one."""
    f, p = _problem(N, nd, 11, Nz, C, autotune=False)
    got = []
    with p:
        for fwd, bp in [(0, 4)] + [(s, 4) for s in (5, 6, 7, 8, 9, 10, 11)] + [(0, s) for s in (9, 10, 11, 12, 18, 19)]:
            p.set_data(f).set_tuning(fwd, bp)
            p.run(5).synchronize()
            got.append({k: p.get(k) for k in ("u", "ku", "lambda")})
    for g in got[1:]:
        for k in g:
            np.testing.assert_array_equal(g[k], got[0][k], err_msg=k)


@pytest.mark.parametrize("N,nd,Nz,C", [(17, 5, 20, 4), (18, 31, 24, 4), (24, 24, 32, 4), (25, 25, 27, 3)])
def test_flat_pair_shape_on_edges_and_infinities(N, nd, Nz, C):
    """Forward shape 8 at 80 to 128 slices: fewer than four pairs of bins, numbers of pairs that are not a
    multiple of four, and infinite and NaN pixels that only one ray of a pair takes."""
    f, p = _problem(N, nd, 9, Nz, C, autotune=False)
    u = np.random.default_rng(9).random((C * Nz, N, N)).astype(np.float32)
    u[0, 5, 7], u[3, 12, 2], u[C * Nz - 1, 11, 11] = np.inf, np.nan, -np.inf
    got = []
    with p:
        for fwd in (0, 8, 9, 11):
            p.set_data(f).set_tuning(fwd, 4)
            p.run(3).synchronize()
            a = p.get("ku")
            p.set("ubar", u)
            p.run(1).synchronize()
            got.append((a, p.get("ku")))
    assert not np.isfinite(got[0][1]).all() and np.isfinite(got[0][0]).all()
    for a, b in got[1:]:
        np.testing.assert_array_equal(a, got[0][0])
        np.testing.assert_array_equal(b, got[0][1])


FORM = """
import numpy as np
from graptor_gb300.solver import Problem
ang = np.deg2rad(np.linspace(-80, 85, 11))
for schedule in (0, None, None):
    with Problem(2, 24, 1, 1, 24, ang, (4, 1), [0.2], normest=11.0) as p:
        if schedule is not None:
            p.set_schedule(schedule)
        p.set_data(np.ones((1, 11, 24), np.float32)).run(3).synchronize()
"""


def test_a_chosen_schedule_does_not_stand_for_later_problems():
    """The first problem of a size has its schedule set and its form of the iteration not timed: the second
    one times it, the third takes the result."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FORM], cwd=root, env=dict(os.environ, GRAPTOR_TUNE_LOG="1"),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert r.stderr.count("two launches:") == 1, r.stderr


@pytest.mark.parametrize("N,nd,nang,Nz,C,fwd,bp", [
    (19, 12, 41, 52, 1, 9, 10), (13, 13, 3, 113, 4, 9, 10), (20, 40, 11, 65, 2, 9, 10),  # small images, many slices
    (64, 64, 20, 92, 1, 9, 10), (64, 64, 20, 64, 3, 9, 10),  # below 2^18 threads per projector
    (64, 65, 64, 64, 2, 11, 10), (72, 72, 60, 48, 4, 9, 10), (64, 70, 84, 64, 4, 11, 19),  # above one or both
    (64, 70, 88, 64, 4, 10, 19), (112, 112, 10, 48, 4, 9, 18)])  # 3000 warps with 8 slices per lane
def test_default_shapes_of_small_images_with_many_slices(N, nd, nang, Nz, C, fwd, bp):
    """Both sides of the lines of the default shapes: the shapes as stated there, and the iterates of the
    default and of the tuned shapes those of the one-ray and one-pixel kernels."""
    got = []
    for autotune, forced in ((False, True), (False, False), (True, False)):
        f, p = _problem(N, nd, nang, Nz, C, autotune=autotune)
        with p:
            p.set_data(f)
            if forced:
                p.set_tuning(0, 4)
            elif not autotune:
                assert (p.tuning["fwd_cfg"], p.tuning["bp_cfg"]) == (fwd, bp)
            p.run(4).synchronize()
            got.append([p.get(k) for k in ("u", "ku", "lambda")])
    for g in got[1:]:
        for a, b in zip(g, got[0]):
            np.testing.assert_array_equal(a, b)
