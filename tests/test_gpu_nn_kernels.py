"""Kernels of the warm-start network's training at the edges of their tiles, against float64
PyTorch on the CPU: weight gradients (tiles of 4 x 32 and 8 x 16 voxels, 16 x 16 channels),
bias gradients (8 blocks per channel), the CUDA-core convolution's 8 x 8 tile and the pooling,
upsampling and ReLU kernels with whole and ragged runs of a row."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = torch.nn.functional


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _rel(a, b):
    return float((a.double().cpu() - b).norm() / b.norm())


def _lib():
    from graptor_gb300 import _lib as L
    return L


@pytest.mark.parametrize("k", [3, 1])
@pytest.mark.parametrize("shape", [(1, 1, 1, 4), (2, 3, 5, 32), (1, 2, 9, 20), (2, 2, 4, 64), (1, 3, 6, 72), (1, 1, 8, 16)])
@pytest.mark.parametrize("ci,co", [(1, 1), (17, 16), (16, 33)])
def test_weight_and_bias_gradient_tiles(k, shape, ci, co):
    L = _lib()
    B, D, H, W = shape
    g = torch.Generator().manual_seed(B * 100 + W + ci)
    x = torch.randn((B, ci + 1, D, H, W), generator=g).to(torch.bfloat16)
    dy = torch.randn((B, co + 2, D, H, W), generator=g)
    w = torch.zeros((co, ci, k, k, k), dtype=torch.float64, requires_grad=True)
    b = torch.zeros(co, dtype=torch.float64, requires_grad=True)
    gw, gb = torch.autograd.grad(F.conv3d(x[:, 1:].double(), w, b, padding=k // 2), (w, b), dy[:, 2:].double())
    nvox = B * D * H * W
    xd, dyd = x.cuda(), dy.cuda()
    for chunks in (1, 3):
        kchunk = -(-nvox // chunks)
        part = torch.empty(-(-nvox // kchunk) * co * ci * k ** 3, device="cuda")
        out = torch.empty((co, ci, k, k, k), device="cuda")
        L.check(L.lib().gt_nn_conv3d_wgrad(_p(dyd), co, co + 2, 2, _p(xd), 1, ci, ci + 1, 1, B, D, H, W, k, kchunk,
                                           _p(part), _p(out), 0, None))
        assert _rel(out, gw) < 1e-5  # float32 sums of at most 768 terms per weight
    db = torch.ones(co, device="cuda")
    L.check(L.lib().gt_nn_bias_grad(_p(dyd), co, co + 2, 2, B, D * H * W, _p(db), 1, None))
    assert _rel(db, gb + 1) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cuda_core_convolution_large_tile(dtype):
    L = _lib()
    B, D, H, W, ci, co = 2, 16, 64, 64, 3, 21  # 384 blocks of 8 channels x 8 voxels; a partial channel tile
    g = torch.Generator().manual_seed(3)
    x = torch.randn((B, ci, D, H, W), generator=g).to(dtype)
    w = (torch.randn((co, ci, 3, 3, 3), generator=g) * 0.2).to(torch.bfloat16)
    y = torch.zeros((B, co, D, H, W), device="cuda")
    xd, wd = x.cuda(), w.cuda()
    L.check(L.lib().gt_nn_conv3d(_p(xd), int(dtype == torch.bfloat16), ci, ci, 0, _p(wd), None, _p(y), 0, co, co, 0, B, D,
                                 H, W, 3, 0, 0, None))
    assert _rel(y, F.conv3d(x.double(), w.double(), padding=1)) < 1e-6


@pytest.mark.parametrize("W", [2, 4, 6, 8, 12, 16])
def test_pool_upsample_relu_runs(W):
    """W: row length of the coarse tensors."""
    L = _lib()
    lib = L.lib()
    B, C, D, H = 2, 3, 2, 3
    g = torch.Generator().manual_seed(W)
    fine = torch.randn((B, C + 2, 2 * D, 2 * H, 2 * W), generator=g).to(torch.bfloat16)
    coarse = torch.randn((B, C, D, H, W), generator=g).to(torch.bfloat16)
    fd, cd = fine.cuda(), coarse.cuda()
    out = torch.empty_like(cd)
    L.check(lib.gt_nn_pool2(_p(fd), C + 2, 1, _p(out), C, B, D, H, W, None))
    assert _rel(out, F.avg_pool3d(fine[:, 1:1 + C].double(), 2)) < 4e-3  # one bfloat16 rounding
    up = fd.clone()
    L.check(lib.gt_nn_up2(_p(cd), _p(up), C, C + 2, 1, B, 2 * D, 2 * H, 2 * W, None))
    want = fine.clone()
    want[:, 1:1 + C] = F.interpolate(coarse.float(), scale_factor=2, mode="nearest").to(torch.bfloat16)
    assert torch.equal(up.cpu(), want)
    gf = torch.randn((B, C + 2, 2 * D, 2 * H, 2 * W), generator=g)
    gc = torch.randn((B, C, D, H, W), generator=g)
    gfd, gcd = gf.cuda(), gc.cuda()
    dx = torch.empty_like(gcd)
    L.check(lib.gt_nn_up2_bwd(_p(gfd), C + 2, 1, _p(dx), C, B, D, H, W, None))
    assert _rel(dx, 8 * F.avg_pool3d(gf[:, 1:1 + C].double(), 2)) < 1e-6
    acc = gfd.clone()
    L.check(lib.gt_nn_pool2_bwd(_p(gcd), _p(acc), C, C + 2, 1, B, 2 * D, 2 * H, 2 * W, None))
    want = gf.double()
    want[:, 1:1 + C] += 0.125 * F.interpolate(gc.double(), scale_factor=2, mode="nearest")
    assert _rel(acc, want) < 1e-6
    acc = gfd.clone()
    L.check(lib.gt_nn_relu_bwd(_p(acc), _p(fd), 1, C, C + 2, 1, B, 8 * D * H * W, None))
    want = gf.clone()
    want[:, 1:1 + C] *= fine[:, 1:1 + C] > 0
    assert torch.equal(acc.cpu(), want)
