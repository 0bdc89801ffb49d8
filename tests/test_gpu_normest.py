"""The operator-norm estimate's projectors with each number of fraction bits of their fixed-point
geometry, and with FP64 geometry, against the power iteration with the exact FP64 matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _normest(N, nd, ang):
    from graptor_gb300.solver import Problem
    with Problem(2, N, 1, 1, nd, ang, (4, 1), [0.2], "L2", "TGV", "UNCORR", autotune=False) as p:
        p.set_data(np.ones((1, ang.size, nd), np.float32))
        return p.scalars["normest"]


@pytest.mark.parametrize("N,nd", [(7, 1009), (7, 1010), (6, 16371), (6, 16372), (5, 262133), (5, 262134), (600, 500)])
def test_fraction_bits(N, nd):
    """nd + 2 N on both sides of 2^10, 2^14 and 2^18: 52, 48, 44 fraction bits and FP64."""
    from oracle import fp64 as F
    ang = np.deg2rad(np.array([12.0, 47.0, 90.0, 133.0]))
    R = F.radon_matrix(ang, N, nd)
    x = np.ones(N * N)
    for _ in range(30):
        x = R.T @ (R @ (x / x.sum()))
    want = np.sqrt(x.sum())
    # it stops when two consecutive sums agree to 1e-8
    assert abs(_normest(N, nd, ang) - want) <= 1e-6 * want


def test_an_angle_that_is_not_a_number_takes_no_pixel():
    ang = np.deg2rad(np.array([12.0, 47.0, 90.0, 133.0]))
    assert _normest(24, 24, np.insert(ang, 2, np.nan)) == pytest.approx(_normest(24, 24, ang), rel=1e-12)
