"""The two-launch form of small problems (schedule 3), forced, against separate launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reg,disc", [("TGV", "KL"), ("TV", "L2")])
@pytest.mark.parametrize("cpl", ["UNCORR", "FROB"])
@pytest.mark.parametrize("dim,N,nd,Nz,C", [
    (2, 33, 33, 1, 1), (2, 30, 41, 2, 1), (2, 21, 5, 1, 3), (2, 17, 17, 1, 4),
    (3, 21, 21, 1, 1), (3, 24, 19, 2, 1), (3, 19, 40, 3, 1), (3, 26, 26, 4, 1), (3, 18, 18, 1, 2), (3, 20, 20, 2, 2),
    (3, 15, 22, 1, 3), (3, 23, 23, 1, 4)])
def test_two_launch_iteration_equals_separate_launches(dim, N, nd, Nz, C, reg, cpl, disc):
    """1, 2, 3 (padded) and 4 slices in every split into slices and channels, with the primal weight, the
    step size and the precise primal mode, over runs that end inside and at a graph chunk."""
    from graptor_gb300.solver import Problem
    ang = np.deg2rad(np.linspace(-80, 85, 35))  # 33 to 35: more than one group of staged angles
    f = np.abs(np.random.default_rng(N).standard_normal((C * Nz, ang.size, nd))).astype(np.float32)
    fields = ("u", "ubar", "v", "lambda", "ku") + (("p", "pbar", "w") if reg == "TGV" else ())
    got = []
    for schedule in (0, 3):
        with Problem(dim, N, Nz, C, nd, ang, (4, 1), [0.2] * C, disc, reg, cpl, 1.5 if dim == 3 else 1.0, 11.0) as p:
            p.set_schedule(schedule)
            p.set_data(f)
            assert p.tuning["schedule"] == schedule
            assert (p.launches_per_iteration == 2) == (schedule == 3)
            p.run(7).synchronize()
            got.append({k: p.get(k) for k in fields})
            p.set_precise_primal()
            p.run(5).synchronize()
            p.set_primal_weight(3.0)
            p.run(37).synchronize()
            got[-1].update({k + " precise": p.get(k) for k in fields + ("ulo",)})
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)


def test_schedule_3_is_refused_where_it_does_not_apply():
    from graptor_gb300.solver import Problem
    ang = np.deg2rad(np.linspace(-80, 85, 5))
    for Nz, C, cpl in ((5, 1, "FROB"), (4, 2, "FROB"), (1, 5, "UNCORR"), (1, 2, "NUCL")):
        with Problem(3, 9, Nz, C, 9, ang, (4, 1), [0.2] * C, coupling=cpl, normest=11.0) as p:
            with pytest.raises(ValueError):
                p.set_schedule(3)
    with Problem(3, 9, 4, 1, 9, ang, (4, 1), [0.2], normest=11.0) as p:
        p.set_schedule(3)
        p.set_data(np.ones((4, 5, 9), np.float32))
        p.set_tuning(9, 10)  # the shapes asked for are the ones that run
        assert p.tuning["schedule"] == 1 and p.launches_per_iteration > 2
