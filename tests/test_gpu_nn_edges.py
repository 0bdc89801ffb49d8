"""Weight gradients where rows and columns of a volume end inside a tile: what is not finite
reaches the taps that use it and no others."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _wgrad(x, dy):
    """dW[co][ci][kd][kh][kw] in float64, each tap over the voxels whose neighbour is inside."""
    D, H, W = x.shape[2:]
    out = np.zeros((dy.shape[1], x.shape[1], 3, 3, 3))
    for t in np.ndindex(3, 3, 3):
        a = [slice(max(0, 1 - k), min(n, n + 1 - k)) for k, n in zip(t, (D, H, W))]  # voxels of dY
        b = [slice(s.start + k - 1, s.stop + k - 1) for s, k in zip(a, t)]           # their neighbours
        with np.errstate(invalid="ignore"):
            out[(slice(None), slice(None)) + t] = np.einsum("bodhw,bidhw->oi", dy[(slice(None), slice(None), *a)],
                                                            x[(slice(None), slice(None), *b)])
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 2, 9, 20), (1, 3, 6, 72), (2, 1, 5, 8), (1, 2, 8, 32)])
def test_infinite_activation_reaches_its_own_taps_only(shape, dtype):
    """Tiles of 8 x 16 and 4 x 32 voxels, ragged in rows, in columns, in both and in neither; infinite
    activations on the last row and column, dY positive (so that no tap sees infinity minus infinity)."""
    from graptor_gb300 import _lib as L
    B, D, H, W = shape
    ci, co = 3, 2
    g = torch.Generator().manual_seed(W)
    x = torch.randn((B, ci, D, H, W), generator=g).to(dtype)
    x[0, 0, 0, H - 1, W - 1] = float("inf")
    x[0, 1, D - 1, H - 1, W // 2] = float("inf")
    x[0, 2, 0, H // 2, W - 1] = float("inf")
    dy = torch.rand((B, co, D, H, W), generator=g) + 0.1
    want = _wgrad(x.double().numpy(), dy.double().numpy())
    assert np.isinf(want).any() and np.isfinite(want).any()
    xd, dyd = x.cuda(), dy.cuda()
    part, out = torch.empty(co * ci * 27, device="cuda"), torch.empty((co, ci, 3, 3, 3), device="cuda")
    L.check(L.lib().gt_nn_conv3d_wgrad(_p(dyd), co, co, 0, _p(xd), int(dtype == torch.bfloat16), ci, ci, 0, B, D, H, W, 3,
                                       B * D * H * W, _p(part), _p(out), 0, None))
    got = out.double().cpu().numpy()
    fin = np.isfinite(want)
    np.testing.assert_array_equal(np.isfinite(got), fin)
    np.testing.assert_array_equal(got[~fin], want[~fin])
    # float32 sums of n <= 1296 products of |x| dY: n 2^-24 times the sum of magnitudes, some 900
    assert np.abs(got[fin] - want[fin]).max() <= 0.07


@pytest.mark.parametrize("W", [32, 16])
def test_plane_of_more_than_2_31_voxels(W):
    """Voxel offsets inside a plane do not fit 32 bits: a pair of voxels and their products at both ends."""
    from graptor_gb300 import _lib as L
    H = (1 << 31) // W + 9
    x = torch.zeros((H, W), dtype=torch.bfloat16, device="cuda")
    dy = torch.zeros((H, W), device="cuda")
    x[0, 1], x[H - 2, 3], x[H - 1, W - 1] = 2.0, 3.0, 5.0
    dy[1, 2], dy[H - 1, 2], dy[H - 1, W - 1] = 0.5, 0.25, 4.0
    want = torch.zeros((3, 3))
    # dW[kh][kw] = sum of dY[h][w] X[h + kh - 1][w + kw - 1]
    want[0, 0] += 0.5 * 2.0
    want[0, 2] += 0.25 * 3.0
    want[1, 1] += 4.0 * 5.0
    kchunk = -(-H * W // 608)
    part, out = torch.empty(608 * 27, device="cuda"), torch.empty((3, 3, 3), device="cuda")
    L.check(L.lib().gt_nn_conv3d_wgrad(_p(dy), 1, 1, 0, _p(x), 1, 1, 1, 0, 1, 1, H, W, 3, kchunk, _p(part), _p(out), 0,
                                       None))
    got = out.cpu()
    assert torch.equal(got[1], want) and not got[0].any() and not got[2].any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W", [64, 40])
def test_1x1x1_convolution_large_tile(dtype, W):
    """8 channels x 4 voxels per thread; a partial channel tile, two input channels beyond a staged chunk."""
    from graptor_gb300 import _lib as L
    B, D, H, ci, co = 2, 16, 112, 18, 21
    g = torch.Generator().manual_seed(4)
    x = torch.randn((B, ci, D, H, W), generator=g).to(dtype)
    w = (torch.randn((co, ci, 1, 1, 1), generator=g) * 0.2).to(torch.bfloat16)
    bias = torch.randn(co, generator=g)
    y = torch.zeros((B, co, D, H, W), device="cuda")
    xd, wd, bd = x.cuda(), w.cuda(), bias.cuda()
    L.check(L.lib().gt_nn_conv3d(_p(xd), int(dtype == torch.bfloat16), ci, ci, 0, _p(wd), _p(bd), _p(y), 0, co, co, 0, B, D,
                                 H, W, 1, 0, 0, None))
    want = torch.nn.functional.conv3d(x.double(), w.double(), bias.double())
    assert float((y.double().cpu() - want).abs().max()) <= 19 * 2.0 ** -24 * 18 * 5  # 19 terms below 5


@pytest.mark.parametrize("B,vol", [(1, 1), (3, 5), (2, 1024), (1, 2048), (1, 2049), (2, 1028), (3, 683)])
def test_bias_gradient_on_both_sides_of_one_block(B, vol):
    from graptor_gb300 import _lib as L
    co = 5
    dy = torch.randn((B, co + 1, vol), generator=torch.Generator().manual_seed(vol))
    dyd, db = dy.cuda(), torch.full((co,), 2.0, device="cuda")
    for acc in (0, 1):
        L.check(L.lib().gt_nn_bias_grad(_p(dyd), co, co + 1, 1, B, vol, _p(db), acc, None))
        want = (1 + acc) * dy[:, 1:].double().sum((0, 2))
        scale = float(dy.double().abs().sum((0, 2)).max()) + 1
        assert float((db.double().cpu() - want).abs().max()) <= 40 * 2.0 ** -24 * scale  # some 9 + 5 + 8 additions deep
