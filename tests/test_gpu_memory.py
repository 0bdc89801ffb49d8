"""Problems that fit the device's memory only without the padding of their slice counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _fill_memory(leave):
    """A block that leaves `leave` bytes free."""
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def test_problem_without_room_for_its_padding():
    """5 slices of 1024^2: 19 fields of 8 slices take 638 MB, of 5 slices 398 MB; 545 MB are free."""
    from graptor_gb300.solver import Problem
    N, Nz = 1024, 5
    ang = np.deg2rad(np.array([30.0, 100.0]))
    f = np.abs(np.random.default_rng(1).standard_normal((Nz, 2, N))).astype(np.float32)
    got = []
    for full in (False, True):
        block = _fill_memory(520 << 20) if full else None
        try:
            with Problem(3, N, Nz, 1, N, ang, (4, 1), [0.2], normest=60.0) as p:
                p.set_data(f)
                if full:
                    with pytest.raises(ValueError):
                        p.set_tuning(1, 0)  # one projector shape: the slices are not padded
                p.run(6).synchronize()
                got.append([p.get(k) for k in ("u", "ku", "lambda", "v", "w")])
        finally:
            del block
            torch.cuda.empty_cache()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_two_resolution_problem_without_room_for_its_padding():
    """10 slices of 512^2 (5 of each channel): 239 + 34 MB of fields with 12 and 8 + 8 slices in memory, 199 + 21 MB
    with 10 and 5 + 5; 262 MB are free."""
    from graptor_gb300.radon_tgv_primal_dual_3dsubsample import Subsampling
    N, Nz = 512, 5
    ang = np.deg2rad(np.array([30.0, 100.0]))
    rng = np.random.default_rng(2)
    f0 = np.abs(rng.standard_normal((Nz, 2, N))).astype(np.float32)
    f1 = np.abs(rng.standard_normal((3, 2, N // 2))).astype(np.float32)
    got = []
    for full in (False, True):
        block = _fill_memory(250 << 20) if full else None
        try:
            with Subsampling(N, Nz, 1, 1, N // 2, 3, ang, ang, (4, 1), [0.2, 0.2], 2.0, [(N / 2 - 1) / 2, 1.0],
                             [(N - 1) / 2, 2.0], normest=60.0) as s:
                s.set_data(f0, f1).run(6)
                got.append([s.get(k) for k in ("u", "ku0", "ku1", "kulo")])
        finally:
            del block
            torch.cuda.empty_cache()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
