"""Packed (varlen) causal self-attention for training / prefill.

Backends, in order: the own tcgen05 / TMEM flash-attention kernels (csrc/attn_fwd.cu, csrc/attn_bwd.cu: head_dim 64 or 128, bf16,
GQA, bottom-right aligned causal mask for prefill behind a cached prefix) on CUDA; the flash-attn varlen library (what the
reference calls, 3rdparty/verl/verl/models/transformers/monkey_patch.py:108) for other head sizes / dtypes or when
``POLYRL_ATTN_BACKEND=flash``; PyTorch SDPA over a padded [B, S] view otherwise (CPU tests).  Decode-time attention is NOT
here: it is the hand-written paged kernel in csrc/decode_attn.cu.
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

import os

_FLASH = None


def _own_ok(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> bool:
    return (q.is_cuda and q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16 and v.dtype == torch.bfloat16
            and q.shape[-1] in (64, 128) and k.shape[-1] == v.shape[-1] == q.shape[-1] and q.shape[1] % k.shape[1] == 0
            and os.environ.get("POLYRL_ATTN_BACKEND", "own") == "own" and os.environ.get("POLYRL_GEMM_BACKEND", "tcgen05") != "cublas")


def _rows(t: torch.Tensor) -> torch.Tensor:
    """[T, heads, d] view whose heads are contiguous inside a token row (row pitch free): what the kernels' TMA maps need."""
    if t.stride(2) != 1 or t.stride(1) != t.shape[2] or t.stride(0) % 8 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


class _OwnAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, cu_q, cu_k, scale, causal):
        from . import ext

        q, k, v = _rows(q), _rows(k), _rows(v)
        need = q.requires_grad or k.requires_grad or v.requires_grad
        outs = ext().attn_fwd(q, k, v, cu_q, cu_k, float(scale), bool(causal), bool(need))
        if need:
            ctx.save_for_backward(q, k, v, outs[0], outs[1], cu_q, cu_k)
            ctx.scale, ctx.causal = float(scale), bool(causal)
        return outs[0]

    @staticmethod
    def backward(ctx, do):
        from . import ext

        q, k, v, o, lse, cu_q, cu_k = ctx.saved_tensors
        dq, dk, dv = ext().attn_bwd(q, k, v, o, _rows(do), lse, cu_q, cu_k, ctx.scale, ctx.causal)
        return dq, dk, dv, None, None, None, None


def _own_attention(q, k, v, cu_q, cu_k, scale, causal=True):
    cu_q = cu_q if cu_q.dtype == torch.int32 else cu_q.to(torch.int32)
    cu_k = cu_k if cu_k.dtype == torch.int32 else cu_k.to(torch.int32)
    if torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad):
        return _OwnAttnFn.apply(q, k, v, cu_q.contiguous(), cu_k.contiguous(), scale, causal)
    from . import ext

    return ext().attn_fwd(_rows(q), _rows(k), _rows(v), cu_q.contiguous(), cu_k.contiguous(), float(scale), bool(causal), False)[0]


class _RopeAttnFn(torch.autograd.Function):
    """Optional norm of the query and key heads, rotation and causal attention over packed rows of a fused projection.  One function,
    so that the backward kernels write query, key and value gradients side by side into the gradient of the projection: as separate
    functions, autograd filled, copied and added three tensors of the projection's size to put them together."""

    @staticmethod
    def forward(ctx, qkv, pos, cos, sin, q_norm, k_norm, eps, cu, nq, nkv, d, scale):
        from . import ext

        C, t = ext(), qkv.shape[0]
        if q_norm is not None:
            rot = torch.empty(t, (nq + nkv) * d, device=qkv.device, dtype=qkv.dtype)
            C.qk_norm_rope_(qkv, pos, cos, sin, nq, nkv, d, q_norm, k_norm, eps, rot)
        else:
            C.rope_(qkv, pos, cos, sin, nq, nkv, d, 1.0, None, None, None, 16)
            torch.autograd.graph.increment_version(qkv)          # (mark_dirty would make the rotated rows an output)
            rot = None
        q, k, v = _heads(qkv if rot is None else rot, qkv, nq, nkv, d)
        o, lse = C.attn_fwd(q, k, v, cu, cu, scale, True, True)
        ctx.save_for_backward(qkv, rot, o, lse, pos, cos, sin, q_norm, k_norm, cu)
        ctx.dims = (nq, nkv, d, scale, eps)
        return o

    @staticmethod
    def backward(ctx, do):
        from . import ext

        C = ext()
        qkv, rot, o, lse, pos, cos, sin, q_norm, k_norm, cu = ctx.saved_tensors
        nq, nkv, d, scale, eps = ctx.dims
        q, k, v = _heads(qkv if rot is None else rot, qkv, nq, nkv, d)
        g = torch.empty(qkv.shape, device=qkv.device, dtype=qkv.dtype)
        C.attn_bwd(q, k, v, o, _rows(do), lse, cu, cu, scale, True, g)
        dqn = dkn = None
        if rot is not None:
            dqn, dkn = C.qk_norm_rope_bwd_(g, qkv, pos, cos, sin, nq, nkv, d, q_norm, k_norm, eps)
        else:
            C.rope_(g, pos, cos, sin, nq, nkv, d, -1.0, None, None, None, 16)
        return g, None, None, None, dqn, dkn, None, None, None, None, None, None


def _heads(qk: torch.Tensor, qkv: torch.Tensor, nq: int, nkv: int, d: int):
    """Views [T, heads, d] of the query and key columns of ``qk`` and the value columns of ``qkv``."""
    t = qkv.shape[0]
    return (qk[:, : nq * d].view(t, nq, d), qk[:, nq * d:(nq + nkv) * d].view(t, nkv, d),
            qkv[:, (nq + nkv) * d:].view(t, nkv, d))


def rope_attention(qkv: torch.Tensor, pos: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, nq: int, nkv: int, d: int,
                   cu_seqlens: torch.Tensor, q_norm: torch.Tensor | None = None, k_norm: torch.Tensor | None = None,
                   eps: float = 1e-6) -> torch.Tensor | None:
    """Causal attention [T, nq, d] over packed rows ``qkv`` [T, (nq + 2 nkv) * d] of a projection, its query and key heads normed (if
    gains are given) and rotated first.  ``qkv`` is consumed: its contents afterwards are undefined, and autograd knows that they changed,
    so a node that saved them refuses its backward.  None: these operands need the general path (``apply_rope`` and
    ``attention_varlen``), as do a leaf and a view, whose change in place autograd has to see."""
    from .functional import head_norm_ok

    if not (qkv.dim() == 2 and qkv.is_contiguous() and qkv.shape[1] == (nq + 2 * nkv) * d and qkv.data_ptr() % 16 == 0 and cu_seqlens.is_cuda
            and pos.is_cuda and pos.dtype == torch.int64 and pos.is_contiguous() and pos.dim() == 1 and pos.shape[0] == qkv.shape[0]
            and not any(t.requires_grad for t in (cos, sin))):
        return None
    q, k, v = _heads(qkv.detach(), qkv.detach(), nq, nkv, d)
    if not _own_ok(q, k, v) or (q_norm is not None and not head_norm_ok(qkv, cos, sin, d, q_norm, k_norm)):
        return None
    if q_norm is None and torch.is_grad_enabled() and qkv.requires_grad and (qkv.is_leaf or qkv._is_view()):
        return None
    cu, scale = cu_seqlens.to(torch.int32).contiguous(), d ** -0.5
    if torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in (qkv, q_norm, k_norm)):
        return _RopeAttnFn.apply(qkv, pos, cos, sin, q_norm, k_norm, eps, cu, nq, nkv, d, scale)
    from . import ext

    if q_norm is not None:
        ext().qk_norm_rope_(qkv, pos, cos, sin, nq, nkv, d, q_norm, k_norm, eps)
    else:
        ext().rope_(qkv, pos, cos, sin, nq, nkv, d, 1.0, None, None, None, 16)
    if torch.is_grad_enabled():
        torch.autograd.graph.increment_version(qkv)
    return ext().attn_fwd(q, k, v, cu, cu, scale, True, False)[0]


def _flash():
    global _FLASH
    if _FLASH is None:
        try:
            from flash_attn import flash_attn_varlen_func

            _FLASH = flash_attn_varlen_func
        except Exception:  # pragma: no cover
            _FLASH = False
    return _FLASH


def _sdpa_varlen(q, k, v, cu_seqlens, max_seqlen, causal, scale):
    """q:[T,nq,d] k,v:[T,nkv,d] -> [T,nq,d] via a padded batch (supports autograd)."""
    t, nq, d = q.shape
    nkv = k.shape[1]
    b = cu_seqlens.numel() - 1
    lens = (cu_seqlens[1:] - cu_seqlens[:-1]).long()
    s = int(max_seqlen)
    seq_id = torch.repeat_interleave(torch.arange(b, device=q.device), lens, output_size=t)
    pos = torch.arange(t, device=q.device) - cu_seqlens[:-1].long()[seq_id]
    flat = seq_id * s + pos

    def pad(x):
        out = x.new_zeros(b * s, x.shape[1], x.shape[2])
        out = out.index_copy(0, flat, x)
        return out.view(b, s, x.shape[1], x.shape[2]).transpose(1, 2)      # [B, h, S, d]

    qp, kp, vp = pad(q), pad(k), pad(v)
    if nkv != nq:
        kp = kp.repeat_interleave(nq // nkv, dim=1)
        vp = vp.repeat_interleave(nq // nkv, dim=1)
    key_ok = torch.arange(s, device=q.device)[None, :] < lens[:, None]          # [B, S]
    mask = key_ok[:, None, None, :]
    if causal:
        mask = mask & torch.ones(s, s, dtype=torch.bool, device=q.device).tril()[None, None]
    o = F.scaled_dot_product_attention(qp, kp, vp, attn_mask=mask, scale=scale)
    return o.transpose(1, 2).reshape(b * s, nq, d).index_select(0, flat)


def attention_varlen(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens: torch.Tensor, max_seqlen: int,
                     causal: bool = True, scale: float | None = None) -> torch.Tensor:
    """q:[T,nq,d], k/v:[T,nkv,d] packed over sequences delimited by ``cu_seqlens`` (int32 [B+1])."""
    if scale is None:
        scale = q.shape[-1] ** -0.5
    if _own_ok(q, k, v):
        return _own_attention(q, k, v, cu_seqlens, cu_seqlens, scale, causal)
    fa = _flash() if q.is_cuda and q.dtype in (torch.bfloat16, torch.float16) else False
    if fa:
        return fa(q, k, v, cu_seqlens, cu_seqlens, int(max_seqlen), int(max_seqlen), 0.0, softmax_scale=scale,
                  causal=causal)
    return _sdpa_varlen(q, k, v, cu_seqlens, max_seqlen, causal, scale)


def attention_varlen_prefix(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_q: torch.Tensor, cu_k: torch.Tensor, max_q: int,
                            max_k: int, scale: float | None = None) -> torch.Tensor:
    """Prefill behind a cached prefix: sequence i has ``lq_i`` NEW query tokens and ``lk_i >= lq_i`` keys (cached prefix first,
    then the new tokens); causal mask aligned bottom-right.  q:[Tq,nq,d], k/v:[Tk,nkv,d]."""
    if scale is None:
        scale = q.shape[-1] ** -0.5
    if _own_ok(q, k, v):
        return _own_attention(q, k, v, cu_q, cu_k, scale, True)
    fa = _flash() if q.is_cuda and q.dtype in (torch.bfloat16, torch.float16) else False
    if fa:
        return fa(q, k, v, cu_q, cu_k, int(max_q), int(max_k), 0.0, softmax_scale=scale, causal=True)
    nq, nkv = q.shape[1], k.shape[1]
    out = torch.empty_like(q)
    cq, ck = cu_q.tolist(), cu_k.tolist()
    for i in range(len(cq) - 1):
        qs, ks, vs = q[cq[i]:cq[i + 1]], k[ck[i]:ck[i + 1]], v[ck[i]:ck[i + 1]]
        lq, lk = qs.shape[0], ks.shape[0]
        if nkv != nq:
            ks, vs = ks.repeat_interleave(nq // nkv, dim=1), vs.repeat_interleave(nq // nkv, dim=1)
        mask = torch.arange(lk, device=q.device)[None, :] <= (torch.arange(lq, device=q.device)[:, None] + (lk - lq))
        o = F.scaled_dot_product_attention(qs.transpose(0, 1), ks.transpose(0, 1), vs.transpose(0, 1), attn_mask=mask, scale=scale)
        out[cq[i]:cq[i + 1]] = o.transpose(0, 1)
    return out
