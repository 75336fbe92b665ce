"""A dense decoder block (norm, attention, norm, SwiGLU) as ONE autograd function.

The same kernels run, in the same order and on the same operands, as in the chain of functions that ``models/transformer.py`` builds
from ``rmsnorm_residual``, ``linear``, ``rope_attention`` and ``linear_swiglu``.  Their seven graph nodes cost the host about 700 us a block,
forward and backward, which is more than the GPU needs below about a thousand tokens; this one costs about 200.
"""
from __future__ import annotations

import torch

from .attention import _heads, _own_ok, _rows
from .functional import _C, _cublas, _g2_operand, _sink_for, head_norm_ok

WEIGHTS = ("ln1", "wqkv", "bqkv", "q_norm", "k_norm", "wo", "ln2", "wgu", "wd")


class _DenseBlockFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, pos, cos, sin, cu, dims, *weights):
        ln1, wqkv, bqkv, q_norm, k_norm, wo, ln2, wgu, wd = weights
        nq, nkv, d, eps = dims
        C, t = _C(), x.shape[0]
        h1, rstd1 = C.rmsnorm_fwd(x, ln1, eps)
        qkv = C.gemm_bf16(h1, wqkv, None)
        if bqkv is not None:
            qkv.add_(bqkv)
        if q_norm is not None:
            rot = torch.empty(t, (nq + nkv) * d, device=x.device, dtype=x.dtype)
            C.qk_norm_rope_(qkv, pos, cos, sin, nq, nkv, d, q_norm, k_norm, eps, rot)
        else:
            C.rope_(qkv, pos, cos, sin, nq, nkv, d, 1.0, None, None, None, 16)
            rot = None
        o, lse = C.attn_fwd(*_heads(qkv if rot is None else rot, qkv, nq, nkv, d), cu, cu, d ** -0.5, True, True)
        x1 = C.gemm_bf16(o.view(t, nq * d), wo, x)
        h2, rstd2 = C.rmsnorm_fwd(x1, ln2, eps)
        a, gu = C.gemm_swiglu(h2, wgu, True)
        y = C.gemm_bf16(a, wd, x1)
        ctx.save_for_backward(x, rstd1, h1, qkv, rot, o, lse, x1, rstd2, h2, gu, a, pos, cos, sin, cu, *weights)
        ctx.dims = dims
        return y

    @staticmethod
    def backward(ctx, dy):
        x, rstd1, h1, qkv, rot, o, lse, x1, rstd2, h2, gu, a, pos, cos, sin, cu, ln1, wqkv, bqkv, q_norm, k_norm, wo, ln2, wgu, wd = ctx.saved_tensors
        # the names above are the last references, unless the graph is kept: activations are given up as soon as they are used, as the nodes
        # of a chain would (at 16 K tokens of an 8B block gu, a and h2 are 1.5 GB)
        ctx.maybe_clear_saved_tensors()
        nq, nkv, d, eps = ctx.dims
        C, t = _C(), x.shape[0]
        dy = _g2_operand(dy.contiguous())
        da, dwd = C.gemm2_grads(dy, wd, a, _sink_for(wd))
        del a
        dgu = C.swiglu_bwd(gu, da)
        del gu, da
        dh2, dwgu = C.gemm2_grads(dgu, wgu, h2, _sink_for(wgu))
        del dgu, h2
        dx1, dln2 = C.rmsnorm_bwd(x1, ln2, dh2, rstd2, dy, True)
        del x1, dh2, dy
        do, dwo = C.gemm2_grads(dx1, wo, o.view(t, nq * d), _sink_for(wo))
        g = torch.empty(qkv.shape, device=x.device, dtype=x.dtype)
        C.attn_bwd(*_heads(qkv if rot is None else rot, qkv, nq, nkv, d), o, do.view(t, nq, d), lse, cu, cu, d ** -0.5, True, g)
        del o, do, lse
        dqn = dkn = None
        if rot is not None:
            dqn, dkn = C.qk_norm_rope_bwd_(g, qkv, pos, cos, sin, nq, nkv, d, q_norm, k_norm, eps)
        else:
            C.rope_(g, pos, cos, sin, nq, nkv, d, -1.0, None, None, None, 16)
        del qkv, rot
        dh1, dwqkv = C.gemm2_grads(g, wqkv, h1, _sink_for(wqkv))
        dbqkv = None if bqkv is None else g.sum(0)
        del g, h1
        dx, dln1 = C.rmsnorm_bwd(x, ln1, dh1, rstd1, dx1, True)
        return (dx, None, None, None, None, None, dln1, dwqkv, dbqkv, dqn, dkn, dwo, dln2, dwgu, dwd)


def _plain(w: torch.Tensor) -> bool:
    return w.dtype == torch.bfloat16 and w.is_contiguous() and w.data_ptr() % 16 == 0


def dense_block(x: torch.Tensor, w: dict, pos: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, cu_seqlens: torch.Tensor, nq: int, nkv: int,
                d: int, eps: float) -> torch.Tensor | None:
    """Output of the block on packed rows x [T, H], or None where the chain of functions has to be built: something it multiplies is
    frozen, or operands that the kernels do not take as they are."""
    ws = [w.get(k) for k in WEIGHTS]
    if not (torch.is_grad_enabled() and x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.shape[0] > 0 and x.is_contiguous()
            and x.requires_grad and x.data_ptr() % 16 == 0 and not _cublas()):
        return None
    if any(t is None for t in (ws[0], ws[1], *ws[5:])) or (ws[3] is None) != (ws[4] is None) \
            or not all(t is None or (isinstance(t, torch.Tensor) and t.requires_grad and t.device == x.device and _plain(t)) for t in ws):
        return None
    h, qkv = x.shape[1], (nq + 2 * nkv) * d
    ln1, wqkv, bqkv, q_norm, k_norm, wo, ln2, wgu, wd = ws
    if not (h % 8 == 0 and h <= 8192 and wqkv.shape == (qkv, h) and wo.shape == (h, nq * d) and wgu.shape[1] == h and wgu.shape[0] % 256 == 0
            and wd.shape == (h, wgu.shape[0] // 2) and ln1.shape == ln2.shape == (h,) and (bqkv is None or bqkv.shape == (qkv,))
            and pos.is_cuda and pos.dtype == torch.int64 and pos.is_contiguous() and pos.dim() == 1 and pos.shape[0] == x.shape[0]
            and cu_seqlens.is_cuda and cu_seqlens.dtype == torch.int32 and cu_seqlens.is_contiguous() and not (cos.requires_grad or sin.requires_grad)):
        return None
    probe = wqkv.detach().view(nq + 2 * nkv, h, d)[:, :1].transpose(0, 1)        # [1, heads, d] of the rows' type and device
    if not _own_ok(probe[:, :nq], probe[:, nq:nq + nkv], probe[:, nq + nkv:]) or (q_norm is not None and not head_norm_ok(wqkv, cos, sin, d, q_norm, k_norm)):
        return None
    return _DenseBlockFn.apply(x, pos, cos, sin, cu_seqlens, (nq, nkv, d, eps), *ws)
