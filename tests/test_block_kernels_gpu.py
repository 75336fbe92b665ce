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


def _rope64(x, pos, cos, sin):
    c, s = cos[pos].double()[:, None], sin[pos].double()[:, None]
    lo, hi = x.chunk(2, -1)
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _heads64(qkv, pos, cos, sin, nq, nkv, d, qn, kn, eps):
    p = qkv.double().view(-1, nq + 2 * nkv, d)
    q, k, v = p[:, :nq], p[:, nq:nq + nkv], p[:, nq + nkv:]
    if qn is not None:
        q = q * torch.rsqrt(q.pow(2).mean(-1, keepdim=True) + eps) * qn.double()
        k = k * torch.rsqrt(k.pow(2).mean(-1, keepdim=True) + eps) * kn.double()
    return _rope64(q, pos, cos, sin), _rope64(k, pos, cos, sin), v


@pytest.mark.parametrize("d,nq,nkv", [(32, 3, 1), (64, 14, 2), (128, 8, 2), (256, 2, 2), (48, 2, 1)])
@pytest.mark.parametrize("norm", [False, True])
def test_norm_rope_and_cache(d, nq, nkv, norm):
    """One rounding to bf16 of a value computed in fp32; places without a slot leave the cache as it is.  Widths other than the kernel's
    (48 here) keep the general rotation."""
    if norm and d == 48:
        pytest.skip("the norm kernel is not built for this width")
    t, page, pages = 37, 16, 6
    qkv = _randn(t, (nq + 2 * nkv) * d, seed=1)
    cos, sin = (f.cuda() for f in OF.ref.rope_tables(64, d, 1e4))
    pos = (torch.arange(t) * 7 % 64).cuda()
    slots = torch.randperm(page * pages, generator=torch.Generator().manual_seed(0))[:t].cuda()
    slots[5] = -1
    kc, vc = _randn(pages, nkv, page, d, seed=2), _randn(pages, nkv, page, d, seed=3)
    qn, kn = (_randn(d, seed=4, scale=0.1, shift=1.0), _randn(d, seed=5, scale=0.1, shift=1.0)) if norm else (None, None)
    q, k, v = _heads64(qkv, pos, cos, sin, nq, nkv, d, qn, kn, 1e-6)
    wk, wv, ok = kc.double(), vc.double(), slots >= 0
    wk[slots[ok] // page, :, slots[ok] % page], wv[slots[ok] // page, :, slots[ok] % page] = k[ok], v[ok]
    if norm:
        OF.head_norm_rope_and_cache_(qkv, pos, cos, sin, nq, nkv, d, qn, kn, 1e-6, kc, vc, slots, page)
    else:
        OF.rope_and_cache_(qkv, pos, cos, sin, nq, nkv, d, kc, vc, slots, page)
    for got, want in ((qkv.view(t, -1, d), torch.cat([q, k, v], 1)), (kc, wk), (vc, wv)):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


@pytest.mark.parametrize("d,nq,nkv,lens", [(128, 4, 4, [1]), (128, 8, 2, [128, 1, 129]), (128, 6, 2, [77, 300, 5]), (64, 14, 2, [127, 600, 1, 256]),
                                           (128, 2, 1, [5] * 40)])
@pytest.mark.parametrize("norm", [False, True])
def test_rope_attention(d, nq, nkv, lens, norm):
    """Norm, rotation and attention as one function against autograd in 64 bits: probabilities and their gradients pass through bf16 on
    their way into the products, so 2e-2 of the norm.  A lone token has no gradient but the difference of two fp32 sums of 128 products,
    128 * 2^-24 * 128^-0.5 < 7e-7 an element of the 512 that a gain sums: 2e-5."""
    from polyrl_b200.ops.attention import rope_attention

    t = sum(lens)
    qkv = _randn(t, (nq + 2 * nkv) * d, seed=1)
    cos, sin = (f.cuda() for f in OF.ref.rope_tables(640, d, 1e4))
    pos = torch.cat([torch.arange(n) for n in lens]).cuda()
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    qn, kn = (_randn(d, seed=4, scale=0.1, shift=1.0), _randn(d, seed=5, scale=0.1, shift=1.0)) if norm else (None, None)
    go = _randn(t, nq, d, seed=6)
    leaves = [qkv.double().requires_grad_(True)] + ([g.double().requires_grad_(True) for g in (qn, kn)] if norm else [])
    q, k, v = _heads64(leaves[0], pos, cos, sin, nq, nkv, d, *(leaves[1:] if norm else (None, None)), 1e-6)
    outs = []
    for a, b, c in zip(q.split(lens), k.split(lens), v.split(lens)):
        b, c = b.repeat_interleave(nq // nkv, 1), c.repeat_interleave(nq // nkv, 1)
        z = torch.einsum("qhd,khd->hqk", a, b) * d ** -0.5
        z = z.masked_fill(torch.ones(z.shape[-2:], dtype=torch.bool, device="cuda").triu(1), float("-inf"))
        outs.append(torch.einsum("hqk,khd->qhd", z.softmax(-1), c))
    want = torch.cat(outs)
    wants = [want, *torch.autograd.grad(want, leaves, go.double())]
    with torch.no_grad():
        plain = rope_attention(qkv.clone(), pos, cos, sin, nq, nkv, d, cu, qn, kn)
    mine = [qkv.clone().requires_grad_(True)] + ([g.clone().requires_grad_(True) for g in (qn, kn)] if norm else [])
    got = rope_attention(mine[0] * 1.0, pos, cos, sin, nq, nkv, d, cu, *(mine[1:] if norm else (None, None)))
    assert torch.equal(plain, got)
    for a, b in zip([got, *torch.autograd.grad(got, mine, go)], wants):
        assert (a.double() - b).norm() <= 2e-2 * b.norm() + 2e-5
    assert rope_attention(qkv[:, : (nq + 2 * nkv) * d - 8], pos, cos, sin, nq, nkv, d, cu) is None        # not the rows it is made for


def test_rope_attention_changes_its_rows_in_the_open():
    """Without gains the rows are rotated in place: not a leaf's or a view's, and a node that saved them refuses its backward."""
    from polyrl_b200.ops.attention import rope_attention

    nq, nkv, d, t = 4, 2, 64, 70
    cos, sin = (f.cuda() for f in OF.ref.rope_tables(128, d, 1e4))
    pos, cu = torch.arange(t).cuda(), torch.tensor([0, t], dtype=torch.int32).cuda()
    leaf = _randn(t, (nq + 2 * nkv) * d, seed=1).requires_grad_(True)
    before = leaf.detach().clone()
    call = lambda x: rope_attention(x, pos, cos, sin, nq, nkv, d, cu)          # noqa: E731
    assert call(leaf) is None and call(leaf.view(t, -1)) is None and call((leaf * 1.0).view(t, -1)) is None
    assert torch.equal(leaf, before)
    rows = leaf * 1.0
    saved = rows.sin()
    out = call(rows)
    assert out is not None and torch.isfinite(torch.autograd.grad(out.sum(), leaf, retain_graph=True)[0]).all()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(saved.sum(), leaf)
    plain, w = before.clone(), _randn(1, seed=2).requires_grad_(True)
    saved = plain * w
    assert call(plain) is not None
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(saved.sum(), w)


@pytest.mark.parametrize("t,v,h", [(1, 264, 64), (128, 392, 64), (129, 392, 128), (300, 640, 64), (515, 5000, 896)])
@pytest.mark.parametrize("tau", [1.0, 0.7])
def test_linear_ce_edges(t, v, h, tau):
    """Labels at the edges of tiles and of the epilogue groups' halves, vocabularies that end in either half.  Statistics are fp32 sums over
    at most 5000 columns and products over 896 (1e-5); the gradient of the logits is rounded to bf16 on its way into the products (1e-2)."""
    x, w = _randn(t, h, seed=1).requires_grad_(True), _randn(v, h, seed=2, scale=0.1).requires_grad_(True)
    edges = [e for e in (0, 31, 32, 63, 64, 127, 128, 191, 255, 256, 383, 384, v - 1) if e < v]
    lab = torch.tensor([edges[i % len(edges)] for i in range(t)]).cuda()
    glp, gent = _randn(t, seed=3, dtype=torch.float32), _randn(t, seed=4, dtype=torch.float32)
    lp, ent = ops.linear_cross_entropy(x, w, lab, tau)
    got = [lp, ent, *torch.autograd.grad([lp, ent], [x, w], [glp, gent])]
    x64, w64 = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    logp = (x64 @ w64.t() / tau).log_softmax(-1)
    lp64, ent64 = logp.gather(1, lab[:, None])[:, 0], -(logp.exp() * logp).sum(-1)
    want = [lp64, ent64, *torch.autograd.grad([lp64, ent64], [x64, w64], [glp.double(), gent.double()])]
    for a, b, tol in zip(got, want, (1e-5, 1e-5, 1e-2, 1e-2)):
        assert (a.double() - b).norm() <= tol * b.norm()


@pytest.mark.parametrize("t,v,h,chunk", [(100, 1304, 128, 256), (515, 1304, 896, 256), (515, 1000, 896, 128), (150, 40008, 64, None), (6200, 17000, 64, None)])
@pytest.mark.parametrize("frozen", ["", "x", "w"])
def test_linear_ce_slices(t, v, h, chunk, frozen, monkeypatch):
    """Several slices of the vocabulary in the backward pass: labels at their edges, a ragged last one, gradients of both operands or of one,
    in one launch (515 rows) or two; the usual slices and, for short rows, shorter ones.  Bounds as above."""
    if chunk is not None:
        monkeypatch.setattr(OF, "_CE_CHUNK", chunk)
    step = OF._ce_slice(t)
    assert v > step
    x, w = _randn(t, h, seed=1), _randn(v, h, seed=2, scale=0.1)
    edges = [e for lo in range(0, v, step) for e in (lo, lo + 1, lo - 1) if 0 <= e < v] + [v - 1]
    lab = torch.tensor([edges[i % len(edges)] for i in range(t)]).cuda()
    glp, gent = _randn(t, seed=3, dtype=torch.float32), _randn(t, seed=4, dtype=torch.float32)

    def grads(leaves, f, g):
        keep = [p.requires_grad_(n != frozen) for p, n in zip(leaves, "xw")]
        out = f(*keep)
        return [*out, *torch.autograd.grad(out, [p for p in keep if p.requires_grad], g)]

    def plain(x64, w64):
        logp = (x64 @ w64.t() / 0.7).log_softmax(-1)
        return logp.gather(1, lab[:, None])[:, 0], -(logp.exp() * logp).sum(-1)

    want = grads([x.double(), w.double()], plain, [glp.double(), gent.double()])
    before = ops.LAUNCHES.get("gemm2_grads", 0)
    got = grads([x, w], lambda a, b: ops.linear_cross_entropy(a, b, lab, 0.7), [glp, gent])
    assert ops.LAUNCHES.get("gemm2_grads", 0) - before == (-(-v // step) if not frozen else 0)
    for a, b, tol in zip(got, want, (1e-5, 1e-5, 1e-2, 1e-2)):
        assert (a.double() - b).norm() <= tol * b.norm()


@pytest.mark.parametrize("m,n,k", [(300, 520, 8200), (257, 264, 4104), (2048, 2560, 16384), (129, 2816, 6000)])
def test_gemm_cut_along_the_reduction(m, n, k):
    """Products whose last round of tiles is cut: all layouts, residual, fp32 accumulation, gate / up.  One rounding to bf16; the fp32 sums
    are k / 16 additions, each at most 2^-23 off."""
    from polyrl_b200 import _C
    from polyrl_b200.ops import ext

    C = ext()
    a, b = _randn(m, k, seed=1), _randn(n, k, seed=2, scale=0.05)
    m8 = m // 8 * 8
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _C.gemm2_is_cut(m, n, k) and _C.gemm2_is_cut(m8, n, k) and _C.gemm2_is_cut(m, n // 256 * 256, k)
    want = a.double() @ b.double().t()

    def close(got, ref):
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * ref.abs().max()).all()

    close(C.gemm2_bf16(a, b, False, False, None, None, 0), want)
    close(C.gemm2_bf16(a, b.t().contiguous(), False, True, None, None, 0), want)
    at = a[:m8].t().contiguous()
    close(C.gemm2_bf16(at, b.t().contiguous(), True, True, None, None, 0), want[:m8])
    close(C.gemm2_bf16(at, b, True, False, None, None, 0), want[:m8])
    r = _randn(m, n, seed=3)
    close(C.gemm_bf16(a, b, r, None, 0), want + r.double())
    acc = _randn(m, n, seed=4, dtype=torch.float32)
    ref = want + 0.5 * acc.double()
    C.gemm2_accum_f32_(acc, a, b, False, False, 0.5)
    assert (acc.double() - ref).norm() <= k * 2.0 ** -27 * ref.norm()
    n2 = n // 256 * 256
    gu = want[:, :n2].view(m, -1, 2, 128)
    h, saved = C.gemm_swiglu(a, b[:n2], True)
    close(saved, want[:, :n2])
    close(h, (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).flatten(1))


def _attend64(q, k, v, lq, lk, causal):
    """Packed attention in 64 bits: (output, log-sum-exp [heads, T])."""
    outs, lses = [], []
    g, scale = q.shape[1] // k.shape[1], q.shape[2] ** -0.5
    for a, b, c in zip(q.split(lq), k.split(lk), v.split(lk)):
        z = torch.einsum("qhd,khd->hqk", a, b.repeat_interleave(g, 1)) * scale
        if causal:
            z = z.masked_fill(torch.ones(z.shape[-2:], dtype=torch.bool, device=q.device).triu(z.shape[2] - z.shape[1] + 1), float("-inf"))
        lses.append(z.logsumexp(-1))
        outs.append(torch.einsum("hqk,khd->qhd", z.softmax(-1), c.repeat_interleave(g, 1)))
    return torch.cat(outs), torch.cat(lses, 1)


def _packed(d, lq, lk, growth, nq=4, nkv=2):
    q, k, v = _randn(sum(lq), nq, d, seed=1), _randn(sum(lk), nkv, d, seed=2), _randn(sum(lk), nkv, d, seed=3)
    k = (k.float() * torch.cat([1 + growth * torch.arange(n, device="cuda") / 128 for n in lk])[:, None, None]).bfloat16()
    cu_q, cu_k = (torch.tensor([0] + x, dtype=torch.int32).cumsum(0).to(torch.int32).cuda() for x in (lq, lk))
    return q, k, v, cu_q, cu_k


_LENGTHS = [([1], [1], True), ([130], [130], True), ([3, 128, 257], [3, 128, 257], True), ([5, 200], [700, 333], True), ([64, 1], [640, 129], False),
            ([7] * 100, [7] * 100, True)]


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lq,lk,causal", _LENGTHS)
@pytest.mark.parametrize("growth", [0.0, 3.0])
def test_attention_forward_tiles(d, lq, lk, causal, growth):
    """Packed sequences, prompts behind a prefix among them.  ``growth`` makes later keys longer, so that row maxima rise by more than 2^8
    from tile to tile and the output is rescaled.  Probabilities and the output are bf16: each value within 2^-8, 1e-2 of the norm."""
    from polyrl_b200.ops import ext

    q, k, v, cu_q, cu_k = _packed(d, lq, lk, growth)
    o, lse = ext().attn_fwd(q, k, v, cu_q, cu_k, d ** -0.5, causal, True)
    want, lse64 = _attend64(q.double(), k.double(), v.double(), lq, lk, causal)
    assert (o.double() - want).norm() <= 1e-2 * want.norm()
    assert (lse.double() - lse64).abs().max() <= 1e-5 * (1 + lse64.abs().max()) + 1e-4


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lq,lk,causal", _LENGTHS + [([300], [100], True)])
def test_attention_backward_tiles(d, lq, lk, causal):
    """Gradients of packed sequences, of prompts behind a prefix, and of queries before the first key, which see none.  Probabilities and
    their gradients enter the products as bf16: 2e-2 of the norm; with one key the gradients of the scores are differences of equal sums."""
    from polyrl_b200.ops import ext

    q, k, v, cu_q, cu_k = _packed(d, lq, lk, 0.0)
    go = _randn(*q.shape, seed=4)
    o, lse = ext().attn_fwd(q, k, v, cu_q, cu_k, d ** -0.5, causal, True)
    got = ext().attn_bwd(q, k, v, o, go, lse, cu_q, cu_k, d ** -0.5, causal)
    blind = max(0, lq[0] - lk[0]) if causal else 0                        # queries of the first sequence that see no key
    leaves = [x.double().requires_grad_(True) for x in (q[blind:], k, v)]
    out, _ = _attend64(*leaves, [lq[0] - blind] + lq[1:], lk, causal)
    want = torch.autograd.grad(out, leaves, go[blind:].double())
    assert not got[0][:blind].any()
    for a, b in zip((got[0][blind:], got[1], got[2]), want):
        assert (a.double() - b).norm() <= 2e-2 * b.norm() + 1e-3


@pytest.mark.parametrize("d", [64, 128])
def test_attention_backward_outside_sequences(d):
    """Query rows that belong to no sequence, and queries without any key, have a zero gradient whatever lay in the memory before."""
    from polyrl_b200.ops import ext

    nq, nkv, t = 4, 2, 300
    q, k, v, go = (_randn(t, h, d, seed=i) for i, h in enumerate((nq, nkv, nkv, nq)))
    cu = torch.tensor([5, 150, 263], dtype=torch.int32).cuda()
    o, lse = ext().attn_fwd(q, k, v, cu, cu, d ** -0.5, True, True)
    for out in (None, torch.full((t, (nq + 2 * nkv) * d), float("nan"), device="cuda", dtype=torch.bfloat16)):
        junk = torch.full((t, nq, d), float("nan"), device="cuda", dtype=torch.bfloat16)
        del junk                                             # (its block is the one that the gradient takes)
        dq = ext().attn_bwd(q, k, v, o.nan_to_num(), go, lse, cu, cu, d ** -0.5, True, out)[0]
        assert not dq[:5].any() and not dq[263:].any() and torch.isfinite(dq).all() and dq[5:263].any()
    junk = torch.full((t, nq, d), float("nan"), device="cuda", dtype=torch.bfloat16)
    del junk
    none = torch.zeros(3, dtype=torch.int32, device="cuda")
    dq, dk, dv = ext().attn_bwd(q, k[:0], v[:0], o.nan_to_num(), go, lse, cu, none, d ** -0.5, True)
    assert not dq.any() and torch.isfinite(dq).all() and dk.shape == dv.shape == (0, nkv, d)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("lq,lk,causal", [([100, 77, 300], [100, 77, 300], True), ([1, 1, 1], [1, 1, 1], True), ([50, 3, 129], [400, 130, 257], True), ([64, 200, 65], [33, 129, 127], False),
                                          ([40, 9, 144], [144, 300, 40], True)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_attention_keeps_sequences_apart(d, lq, lk, causal, bad):
    """Values that are not finite, in the second of three packed sequences, leave outputs and gradients of the others as they are, bit for bit."""
    from polyrl_b200.ops import ext

    q, k, v, cu_q, cu_k = _packed(d, lq, lk, 0.0)
    go = _randn(*q.shape, seed=4)

    def run():
        o, lse = ext().attn_fwd(q, k, v, cu_q, cu_k, d ** -0.5, causal, True)
        grads = ext().attn_bwd(q, k, v, o, go, lse, cu_q, cu_k, d ** -0.5, causal)
        n = len(lq)
        split = [x.split(lq if x.shape[0] == sum(lq) else lk) for x in (o, *grads)] + [lse.split(lq, 1)]
        return [[p[i].clone() for p in split] for i in range(n)]

    want = run()
    for x, lens in ((q, lq), (k, lk), (v, lk), (go, lq)):
        x.split(lens)[1].fill_(bad)
    got = run()
    for i in (0, 2):
        assert all(torch.equal(a, b) and not torch.isnan(a).any() for a, b in zip(got[i], want[i])), i


@pytest.mark.parametrize("t,n,k,joint", [(8, 136, 136, True), (387, 1152, 896, True), (300, 4096, 520, False), (2503, 2048, 896, True), (520, 200, 2056, True),
                                         (1030, 6144, 1000, True), (515, 392, 896, True)])
def test_gemm2_grads(t, n, k, joint):
    """Input and weight gradient of a linear layer, in one launch where the plan says so (148 SMs): bf16 and accumulating fp32 input gradient,
    results of the separate products bit for bit where those sum whole tiles, ragged edges in every dimension."""
    from polyrl_b200 import _C
    from polyrl_b200.ops import ext

    C = ext()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _C.gemm2_grads_joint(t, n, k) == joint
    dy, w, x = _randn(t, n, seed=1), _randn(n, k, seed=2, scale=0.05), _randn(t, k, seed=3)
    dx, dw = C.gemm2_grads(dy, w, x)
    apart = C.gemm2_bf16(dy, w, False, True, None, None, 0), C.gemm2_bf16(dy, x, True, True, None, None, 0)
    for got, want, one, cut in ((dx, dy.double() @ w.double(), apart[0], _C.gemm2_is_cut(t, k, n)), (dw, dy.double().t() @ x.double(), apart[1], _C.gemm2_is_cut(n, k, t))):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).all()
        assert cut or torch.equal(got, one)
    acc = _randn(t, k, seed=4, dtype=torch.float32)
    ref = acc.double() + dy.double() @ w.double()
    out = torch.empty(n + 8, k + 8, device="cuda", dtype=torch.bfloat16)[8:, 8:]
    if out.data_ptr() % 16 == 0 and out.stride(0) % 8 == 0:
        C.gemm2_grads(dy, w, x, out, acc, 1.0)
        assert torch.equal(out, dw)
        assert (acc.double() - ref).norm() <= n * 2.0 ** -27 * ref.norm() + 1e-6 * ref.norm()


@pytest.mark.parametrize("model,lens", [("qwen2.5-0.5b", [3, 130]), ("qwen3-1.7b", [300, 1, 77]), ("llama3-8b", [40])])
def test_dense_block_is_the_chain(model, lens, monkeypatch):
    """The block as one function gives, bit for bit, what the chain of functions gives (its bias is added in the same place)."""
    from polyrl_b200.models import get_model_config
    from polyrl_b200.models import transformer as tf

    cfg, t = get_model_config(model), sum(lens)
    w = {n: _randn(*s, seed=i, scale=0.1 if len(s) == 1 else 0.02, shift=1.0 if n.startswith("ln") or n.endswith("norm") else 0.0).requires_grad_(True)
         for i, (n, s) in enumerate(tf.layer_param_specs(cfg, 0))}
    x, gy = _randn(t, cfg.hidden_size, seed=50).requires_grad_(True), _randn(t, cfg.hidden_size, seed=51)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32).cuda()
    inp = tf.PackedInput(torch.zeros(t, dtype=torch.long, device="cuda"), torch.cat([torch.arange(n) for n in lens]).cuda(), cu, max(lens))
    y = tf.layer_forward(cfg, w, x, inp)
    assert type(y.grad_fn).__name__.startswith("_DenseBlockFn")
    got = [y, *torch.autograd.grad(y, [x, *w.values()], gy)]
    monkeypatch.setattr(tf, "dense_block", lambda *a: None)
    y = tf.layer_forward(cfg, w, x, inp)
    for n, a, b in zip(["y", "x", *w], got, [y, *torch.autograd.grad(y, [x, *w.values()], gy)]):
        assert torch.equal(a, b), n
    w["wo"].requires_grad_(False)                        # a frozen weight: the chain, which leaves its gradient out
    monkeypatch.undo()
    assert not type(tf.layer_forward(cfg, w, x, inp).grad_fn).__name__.startswith("_DenseBlockFn")


@pytest.mark.parametrize("model", ["qwen3-1.7b", "llama3-8b"])
def test_dense_block_gives_up_its_activations(model, monkeypatch):
    """Memory at the peak of the backward pass is no more than with the chain of functions, whose nodes free theirs one by one; a graph that is
    kept can be gone through again."""
    from polyrl_b200.models import get_model_config
    from polyrl_b200.models import transformer as tf

    cfg, t = get_model_config(model), 4096
    w = {n: _randn(*s, seed=i, scale=0.02, shift=1.0 if len(s) == 1 else 0.0).requires_grad_(True) for i, (n, s) in enumerate(tf.layer_param_specs(cfg, 0))}
    x, gy = _randn(t, cfg.hidden_size, seed=50).requires_grad_(True), _randn(t, cfg.hidden_size, seed=51)
    cu = torch.tensor([0, t // 2, t], dtype=torch.int32).cuda()
    inp = tf.PackedInput(torch.zeros(t, dtype=torch.long, device="cuda"), torch.cat([torch.arange(t // 2)] * 2).cuda(), cu, t // 2)

    def peak():
        y = tf.layer_forward(cfg, w, x, inp)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        torch.autograd.grad(y, [x, *w.values()], gy)
        return torch.cuda.max_memory_allocated()

    block = [peak(), peak()][1]
    y = tf.layer_forward(cfg, w, x, inp)
    first, again = (torch.autograd.grad(y, [x, *w.values()], gy, retain_graph=k) for k in (True, False))
    assert all(torch.equal(a, b) for a, b in zip(first, again))
    del first, again, y
    monkeypatch.setattr(tf, "dense_block", lambda *a: None)
    chain = [peak(), peak()][1]
    assert block <= chain + (1 << 20), (block, chain)


@pytest.mark.parametrize("rows,impl,kernel", [(1, "stream", "stream_gemm"), (128, "stream", "stream_gemm"), (129, "stream", "gemm_swiglu"), (16, "skinny", "gemm_swiglu")])
def test_gate_up_of_a_decode_step(rows, impl, kernel, monkeypatch):
    """The stream kernel takes up to 128 rows where it is the chosen implementation, else the tile kernel; one rounding to bf16 of each
    factor's fp32 sum of 512 products."""
    monkeypatch.setenv("POLYRL_DECODE_GEMM_IMPL", impl)
    x, w = _randn(rows, 512, seed=1), _randn(1024, 512, seed=2, scale=0.05)
    before = ops.LAUNCHES.get(kernel, 0)
    with torch.no_grad():
        got = ops.linear_swiglu(x, w)
    assert ops.LAUNCHES.get(kernel, 0) == before + 1
    gu = (x.double() @ w.double().t()).view(rows, -1, 2, 128)
    want = (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).flatten(1)
    assert ((got.double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-3).all()


def test_decode_kernels_behind_each_other():
    """Kernels of a decode step may start while the one before still runs: a chain in which each reads what the last one wrote, its buffers
    freed and taken again on the way, gives the same values as with a wait after every kernel."""
    from polyrl_b200.ops import ext

    C, b, h, f = ext(), 45, 1024, 2048
    wq = [OF.quantize_weight_fp8(_randn(*s, seed=i, scale=0.03)) for i, s in enumerate([(2 * f, h), (h, f)])]
    norm = _randn(h, seed=5, scale=0.1, shift=1.0)

    def chain(wait):
        x = _randn(b, h, seed=9)
        sync = torch.cuda.synchronize if wait else (lambda: None)
        y = ops.rmsnorm(x, norm)
        for _ in range(30):
            sync()
            g = OF._linear_fp8(y, wq[0], swiglu=True)
            sync()
            d = OF._linear_fp8(g, wq[1])
            sync()
            y = C.add_rmsnorm_(x, d, norm, 1e-6)
        return x, y

    with torch.no_grad():
        want = chain(True)
        for _ in range(5):
            assert all(torch.equal(a, c) for a, c in zip(chain(False), want))
