"""Slice counts that are not a multiple of 4 (padded with zero slices in device memory):
the padding must not reach any result.  Iterates against the CPU oracle, the
movement of a restart against the fields read back, and schedule 2 (its second buffer
set) against plain iterations, at the counts where the padding starts and ends."""
import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # dim, Nz, C, regularisation, coupling: S = 1, 2 (no padding), 3, 5, 6, 7, 9, 39
    (2, 1, 1, "TGV", "UNCORR"), (3, 2, 1, "TGV", "FROB"), (3, 3, 1, "TGV", "FROB"), (2, 5, 1, "TV", "UNCORR"),
    (3, 2, 3, "TGV", "FROB"), (3, 1, 7, "TGV", "UNCORR"), (3, 9, 1, "TV", "FROB"), (3, 13, 3, "TGV", "UNCORR"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_padding_slices_reach_no_result(case):
    from graptor_gb300 import phantom
    from graptor_gb300.solver import Problem
    from oracle import oracle as O
    dim, Nz, C, reg, cpl = case
    N, nd, nang, ne = 23, 23, 14, 16.0
    rng = np.random.default_rng(zlib.crc32(repr(case).encode()))
    ang = phantom.angles_deg(nang)
    ofs = O.radon_struct(ang, N, nd)
    f = phantom.poisson(O.radon(np.abs(rng.standard_normal((C * Nz, N, N))).astype(np.float32), ofs, nd), 200.0, 1)
    mu = rng.uniform(0.1, 0.5, C)
    fields = ("u", "p", "v", "w", "lambda") if reg == "TGV" else ("u", "v", "lambda")
    with Problem(dim, N, Nz, C, nd, ang, (3.0, 1.5), mu, "KL", reg, cpl, 1.0, ne) as p:
        p.set_data(f).run(7).synchronize()
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


def test_padded_second_buffer_set_of_schedule_2():
    from graptor_gb300 import phantom
    from graptor_gb300.solver import Problem
    N, Nz, C, nang = 20, 10, 1, 11  # S = 10, padded to 12
    f = np.abs(np.random.default_rng(4).standard_normal((C * Nz, nang, N))).astype(np.float32)
    got = []
    with Problem(3, N, Nz, C, N, phantom.angles_deg(nang), (4, 1), [0.3] * C, normest=15.0) as p:
        for schedule in (0, 2):
            p.set_schedule(schedule)
            p.set_data(f).run(9).synchronize()
            p.snapshot()
            p.run(35).synchronize()
            got.append([p.get(k) for k in ("u", "ubar", "p", "v", "w", "lambda")] + [np.array(p.movement())])
    for x, y in zip(*got):
        np.testing.assert_array_equal(x, y)
