"""The two-resolution solver where its two series differ in angles and where a group has enough
slices for the pair kernels: buffers that no run has written stay zero, projections against the
CPU oracle's, and every channel against the same channel solved beside few others."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, MU = 24, 0.2


def _subs(C0, C1, Nz, nang0, nang1, coupling="UNCORR"):
    from graptor_gb300.radon_tgv_primal_dual_3dsubsample import Subsampling
    ang = [np.deg2rad(np.linspace(15, 165, n)) if n > 2 else np.deg2rad(np.array([33.0, 101.0])[:n]) for n in (nang0, nang1)]
    return ang, Subsampling(N, Nz, C0, C1, N // 2, Nz // 2, *ang, (4, 1), [MU] * (C0 + C1), 2.0,
                            [(N / 2 - 1) / 2, (Nz / 2 - 1) / 2], [(N - 1) / 2, (Nz - 1) / 2], "KL", "TGV", coupling, 1.0, 9.0)


def _data(C, Nz, nang, nd, seed):
    return np.abs(np.random.default_rng(seed).standard_normal((C, Nz, nang, nd))).astype(np.float32)


@pytest.mark.parametrize("C0,C1,nang0,nang1", [(7, 1, 71, 2), (1, 7, 2, 71), (1, 1, 2, 200)])
def test_fields_are_zero_until_a_run_writes_them(C0, C1, nang0, nang1):
    """(7, 1) and (1, 7) with 14 slices: the larger group's pair table; (1, 1): the coarse series has 100
    times the fine one's angles."""
    _, s = _subs(C0, C1, 14, nang0, nang1)
    with s:
        for k in ("u", "ku0", "ku1", "kulo"):
            assert not s.get(k).any(), k


@pytest.mark.parametrize("C0,C1,nang0,nang1", [(7, 1, 31, 2), (1, 7, 2, 31), (1, 1, 2, 200)])
def test_projections_of_both_series_match_oracle(C0, C1, nang0, nang1):
    from graptor_gb300 import _lib as L
    from oracle import oracle as O
    Nz = 14
    ang, s = _subs(C0, C1, Nz, nang0, nang1)
    x = np.random.default_rng(C0).random(((C0 + C1) * Nz, N, N)).astype(np.float32)
    with s:
        s.set_data(_data(C0, Nz, nang0, N, 1), _data(C1, Nz // 2, nang1, N // 2, 2))
        L.check(L.lib().gt_set_state(ctypes.c_void_p(L.lib().gt_subs_problem(s._h)), L.FIELDS["ubar"],
                                     ctypes.c_void_p(x.ctypes.data)))
        s.run(1)
        ku0, ku1 = s.get("ku0"), s.get("ku1")
    for ku, img, a in ((ku0, x[:C0 * Nz], ang[0]), (ku1, x[C0 * Nz:], ang[1])):
        want = O.radon(img, O.radon_struct(a, N, N), N)
        # sums of some 2 N products of weights and values of [0, 1], separately rounded there
        assert np.abs(ku - want).max() <= 2 * N * 2.0 ** -23 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("C0,C1,nang0,nang1", [(7, 1, 31, 2), (1, 7, 2, 31)])
def test_channels_of_a_large_group_equal_those_of_a_small_one(C0, C1, nang0, nang1):
    """Uncorrelated channels do not see each other: 98 slices (pair kernels) against 14 (flat kernels),
    bit for bit."""
    Nz = 14
    f0, f1 = _data(C0, Nz, nang0, N, 3), _data(C1, Nz // 2, nang1, N // 2, 4)
    _, s = _subs(C0, C1, Nz, nang0, nang1)
    with s:
        s.set_data(f0, f1).run(20)
        u, k0, k1 = s.get("u").reshape(C0 + C1, Nz, N, N), s.get("ku0").reshape(C0, Nz, -1), s.get("ku1").reshape(C1, Nz, -1)
    for c in (0, 3, 6):
        a, b = (c, 0) if C0 > 1 else (0, c)
        _, s = _subs(1, 1, Nz, nang0, nang1)
        with s:
            s.set_data(f0[a:a + 1], f1[b:b + 1]).run(20)
            v = s.get("u").reshape(2, Nz, N, N)
            np.testing.assert_array_equal(v[0], u[a])
            np.testing.assert_array_equal(v[1], u[C0 + b])
            np.testing.assert_array_equal(s.get("ku0").reshape(Nz, -1), k0[a])
            np.testing.assert_array_equal(s.get("ku1").reshape(Nz, -1), k1[b])
