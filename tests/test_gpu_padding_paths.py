"""Paths that leave the padding slices out of their work: the fused batch mode, and the start of
the dual from the primal with its repair of missed rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fused_batch_of_padded_slice_counts():
    """Members of 3, 5, 6, 9, 39 and 90 slices (4, 8, 8, 12, 40 and 92 in memory) against each alone."""
    from graptor_gb300.solver import Batch, Problem
    sizes = [(3, 1), (5, 1), (2, 3), (9, 1), (13, 3), (45, 2)]
    specs, data = [], []
    for k, (Nz, C) in enumerate(sizes):
        ang = np.deg2rad(np.linspace(-80, 85, 9 + k))
        specs.append(dict(dim=3, N=17 + k, Nz=Nz, C=C, nd=19 + k, angles=ang, alpha=(4.0, 1.0), mu=[0.2] * C,
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
    N, nd = 19, 23
    ang = np.deg2rad(np.linspace(-80, 85, 13))
    rng = np.random.default_rng(Nz)
    f = np.abs(rng.standard_normal((full, ang.size, nd))).astype(np.float32)
    u = rng.random((full, N, N)).astype(np.float32)
    u[:, :, :7] = 0  # rays that the image misses
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
