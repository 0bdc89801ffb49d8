"""The benchmark's count of the projectors' loads against a count pixel by pixel."""
import math
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _direct(kernel, shape, N, nd, angles):
    loads = 0
    for a in angles:
        X, Y = math.cos(a), math.sin(a)
        off = (nd - 1) / 2 - (X + Y) * (N - 1) / 2
        for y in range(N):
            bins = []
            for x in range(N):
                t = x * X + y * Y + off
                lo = math.floor(t)
                bins.append((lo, [b for b in (lo, lo + 1) if -1 < t < nd and 0 <= b < nd]))
            if kernel == "k_fwd" and shape in (8, 10, 11):
                loads += sum(len({b // 2 for b in bs}) for _, bs in bins)
            elif kernel == "k_bp" and shape in (9, 18, 19):
                for x0 in range(0, N, 4):
                    tile = [bins[min(x0 + r, N - 1)] for r in range(4)]
                    d = [tile[r + 1][0] - tile[r][0] for r in range(3)]
                    if all(len(bs) == 2 for _, bs in tile) and (set(d) <= {0, 1} or set(d) <= {0, -1}):
                        loads += len({b for _, bs in tile for b in bs})
                    else:
                        loads += sum(len(bs) for _, bs in tile)
            else:
                loads += sum(len(bs) for _, bs in bins)
    return loads


@pytest.mark.parametrize("kernel,shape", [("k_fwd", 0), ("k_fwd", 10), ("k_fwd", 8), ("k_bp", 10), ("k_bp", 18)])
@pytest.mark.parametrize("N,nd", [(9, 9), (16, 23), (10, 5)])
def test_loads_of_the_projectors(kernel, shape, N, nd):
    sys.path.insert(0, ROOT)
    import bench
    angles = [0.1, 0.8, 1.5, 2.2, 3.0]
    assert bench.gather_bytes(kernel, shape, N, nd, angles, 3) == 12 * _direct(kernel, shape, N, nd, angles)
