"""Kernels around the projections of a decoder block against plain PyTorch: gathers, norms, rotations and their gradients."""
import pytest
import torch

from polyrl_b200 import ops
from polyrl_b200.ops import functional as OF

pytestmark = pytest.mark.gpu


def _randn(*shape, seed=0, dtype=torch.bfloat16, scale=1.0, shift=0.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale + shift).to(dtype)


@pytest.mark.parametrize("t,nkv,page,d", [(1, 1, 1, 8), (7, 2, 16, 64), (300, 3, 16, 128), (1000, 8, 32, 80)])
def test_gather_cached(t, nkv, page, d):
    pages = 40
    kc, vc = _randn(pages, nkv, page, d, seed=1), _randn(pages, nkv, page, d, seed=2)
    g = torch.Generator().manual_seed(t)
    blk = torch.randint(-pages, pages, (t,), generator=g).cuda()          # indices below zero count from the end
    off = torch.randint(-page, page, (t,), generator=g).cuda()
    before = ops.LAUNCHES.get("gather_pages", 0)
    k, v = OF.gather_cached(kc, vc, blk, off)
    assert ops.LAUNCHES["gather_pages"] == before + 1
    assert torch.equal(k, kc[blk, :, off, :]) and torch.equal(v, vc[blk, :, off, :])
    # a strided cache takes the general path, with the same result
    wide = _randn(pages, nkv, page, 2 * d, seed=3)[..., :d]
    assert torch.equal(OF.gather_cached(wide, wide, blk, off)[0], wide[blk, :, off, :])


@pytest.mark.parametrize("t,h", [(1, 64), (3, 896), (301, 1024), (640, 2048), (1187, 4096), (299, 5120), (41, 8192)])
@pytest.mark.parametrize("res", [False, True])
def test_rmsnorm_residual(t, h, res):
    """Norm and residual stream together: one bf16 rounding per result, so 2^-9 of a value; the sums over rows and columns are fp32."""
    x, w = _randn(t, h, seed=1).requires_grad_(True), _randn(h, seed=2, scale=0.1, shift=1.0).requires_grad_(True)
    gy, gr = _randn(t, h, seed=3), _randn(t, h, seed=4)
    y, xr = ops.rmsnorm_residual(x, w, 1e-6)
    dx, dw = torch.autograd.grad([y, xr] if res else [y], [x, w], [gy, gr] if res else [gy])
    x64, w64 = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    y64 = x64 * torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-6) * w64
    wx, ww = torch.autograd.grad([y64, x64 * 1.0] if res else [y64], [x64, w64], [gy.double(), gr.double()] if res else [gy.double()])
    assert torch.equal(xr.detach(), x.detach())
    for got, want in ((y, y64), (dx, wx), (dw, ww)):
        err = (got.double() - want).abs()
        assert (err <= 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).all(), err.max()
    assert torch.equal(torch.autograd.grad(ops.rmsnorm(x, w, 1e-6), w, gy)[0], dw)          # the partial sums have a fixed order
