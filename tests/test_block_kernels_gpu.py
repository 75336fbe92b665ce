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
