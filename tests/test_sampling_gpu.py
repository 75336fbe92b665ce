"""The samplers against a restatement of their noise in torch: every alignment of a row, ends of granules, one element up to several
rounds of a cluster, masked logits, temperatures or their inverses."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from polyrl_b200 import ops

    return ops.ext()


def _hash(x):
    m = 0xFFFFFFFF
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & m
    x = ((x ^ (x >> 15)) * 0x846CA68B) & m
    return x ^ (x >> 16)


def _noise(seed, row, v):
    n = _hash(_hash((torch.arange(v, device="cuda") + 0x9E3779B9 * (row + 1)) & 0xFFFFFFFF) ^ (seed & 0xFFFFFFFF))
    u = ((_hash(n ^ (seed >> 32)) >> 8).clamp(max=0xFFFFFE).float() + 0.5) * (1.0 / 16777216.0)      # (the last number would give u = 1)
    return -torch.log(-torch.log(u))


def _rows(b, v, dtype, offset):
    """[b, v] logits whose rows start anywhere: pitch v + 3, first element ``offset``; a tenth of them masked."""
    base = torch.randn(b * (v + 3) + offset, device="cuda") * 2.5
    z = base.to(dtype)[offset:].as_strided((b, v), (v + 3, 1))
    z.masked_fill_(torch.rand(b, v, device="cuda") < 0.1, -math.inf)
    z[:, v // 2] = 3.0
    return z


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("b,v,offset", [(1, 1, 0), (3, 7, 1), (2, 255, 3), (5, 2049, 0), (3, 16385, 5), (2, 65543, 2), (2, 151936, 7), (33, 4096, 0)])
@pytest.mark.parametrize("top_k,top_p", [(-1, 1.0), (17, 1.0), (-1, 0.9), (40, 0.6)])
def test_choice_and_log_prob(C, dtype, b, v, offset, top_k, top_p):
    torch.manual_seed(b * 1000 + v)
    z = _rows(b, v, dtype, offset)
    t = torch.rand(b, device="cuda") + 0.4
    t[-1] = 0.0 if b > 2 else t[-1]                                    # one greedy row
    seeds = torch.randint(0, 2 ** 62, (b,), device="cuda")
    plain = top_k < 0 and top_p >= 1
    f = (lambda s, inv: C.sample(z, s, seeds, False, inv)) if plain else (lambda s, inv: C.sample_topk_topp(z, s, seeds, False, top_k, top_p, inv))
    tok, lp = f(t, False)
    inv_t = torch.where(t > 0, 1.0 / t.clamp_min(1e-6), torch.zeros_like(t))
    tok2, lp2 = f(inv_t, True)
    assert torch.equal(tok, tok2) and torch.equal(lp, lp2)
    for i in range(b):
        greedy = float(t[i]) == 0
        zi = z[i].double() / (1.0 if greedy else float(t[i]))
        order = zi.sort(descending=True).values
        if 0 < top_k < v:
            zi = zi.masked_fill(zi < order[top_k - 1], -math.inf)
        if top_p < 1 and not greedy:
            kept = zi.sort(descending=True).values
            p = kept.softmax(0)
            zi = zi.masked_fill(zi < kept[(p.cumsum(0) - p) < top_p][-1], -math.inf)
        want = zi.log_softmax(0)
        k = int(tok[i])
        assert 0 <= k < v and math.isfinite(float(want[k])), "a token outside the kept set"
        # fp32 sums of v positive terms in trees of at most 2^5 sequential additions a level: 1e-5 is over 50 of their units
        assert abs(float(lp[i]) - float(want[k])) < 1e-5 * max(1.0, abs(float(want[k])))
        key = zi if greedy else zi + _noise(int(seeds[i]), i, v).double()
        # the kernel's fast logarithm is 4e-7 off near one, where noise of up to log(2^24) comes from: 4e-7 e^11 relative for the
        # best of 65 K, so a choice may differ only where two keys are that close
        assert float(key.max() - key[k]) < 0.05


@pytest.mark.parametrize("b,v,offset", [(1, 2, 0), (2, 5, 1), (16, 17, 0), (18, 40, 3)])
@pytest.mark.parametrize("top_k,top_p", [(-1, 1.0), (3, 0.9)])
def test_rows_with_less_than_a_granule_a_block(C, b, v, offset, top_k, top_p):
    """Rows so short that most CTAs of a row's cluster have nothing to read and hand their part over at once."""
    for _ in range(20):
        test_choice_and_log_prob(C, torch.bfloat16, b, v, offset, top_k, top_p)


@pytest.mark.parametrize("top_k,top_p", [(-1, 1.0), (50, 0.9)])
def test_stretches_without_a_candidate(C, top_k, top_p):
    """Whole warps and whole turns of a CTA see masked logits only, others of the same row do not."""
    b, v = 5, 40000
    torch.manual_seed(v)
    for turn in range(20):
        z = torch.randn(b, v, device="cuda")
        z.masked_fill_((torch.rand(b, -(-v // 256), device="cuda") < (0.5, 0.97)[turn & 1]).repeat_interleave(256, 1)[:, :v], -math.inf)
        z[:, turn * 1999] = 1.0
        z = z.bfloat16()
        seeds = torch.randint(0, 2 ** 62, (b,), device="cuda")
        t = torch.full((b,), 0.8, device="cuda")
        tok, lp = C.sample(z, t, seeds, False, False) if top_k < 0 else C.sample_topk_topp(z, t, seeds, False, top_k, top_p, False)
        raw = z.gather(1, tok[:, None])[:, 0]
        assert torch.isfinite(raw).all() and torch.isfinite(lp).all()
        if top_k < 0:
            want = (z.double() / 0.8).log_softmax(-1).gather(1, tok[:, None])[:, 0]
            assert ((lp - want).abs() <= 1e-5 * want.abs().clamp_min(1)).all()       # fp32 sums, as above


def _unhash(h):
    """x with _hash(x) == h: every step of the mixer has an inverse."""
    m = 0xFFFFFFFF
    x = h ^ (h >> 16)
    x = (x * pow(0x846CA68B, -1, 1 << 32)) & m
    x = x ^ (x >> 15) ^ (x >> 30)
    x = (x * pow(0x7FEB352D, -1, 1 << 32)) & m
    return x ^ (x >> 16)


def _seed_for(bits, col, low):
    """A seed whose noise for element ``col`` of row 0 is made from the given 24 bits."""
    high = _unhash(bits << 8 | 0x5A) ^ _hash(_hash((col + 0x9E3779B9) & 0xFFFFFFFF) ^ low)
    s = high << 32 | low
    return s - (1 << 64) if s >> 63 else s


@pytest.mark.parametrize("bits", [0, 1, 12345678, 0xFFFFF0, 0xFFFFFD, 0xFFFFFE, 0xFFFFFF])
@pytest.mark.parametrize("top_k", [-1, 2])
def test_noise_at_its_ends(C, bits, top_k):
    """Two elements, the first with noise from given bits, against the noise in 64 bits: it wins with a logit that is 1 more than needed and
    loses with one that is 1 less.  Over all 2^24 values the noise is at most 0.84 from that, at the last three: there u is rounded to a
    multiple of 2^-23 and the fast logarithm of it is off by 0.4 of its value."""
    for low in (1, 77, 0xDEADBEEF):
        seed = _seed_for(bits, 0, low)
        other = _hash(_hash((1 + 0x9E3779B9) & 0xFFFFFFFF) ^ low)
        other = _hash(other ^ ((seed >> 32) & 0xFFFFFFFF)) >> 8
        assert _hash(_hash(_hash(0x9E3779B9) ^ low) ^ ((seed >> 32) & 0xFFFFFFFF)) >> 8 == bits
        first, second = (-math.log(-math.log((b + 0.5) / 2 ** 24)) for b in (bits, other))
        for more in (1.0, -1.0):
            z = torch.tensor([[second - first + more, 0.0, -math.inf]], device="cuda")
            s, t = torch.tensor([seed], device="cuda"), torch.ones(1, device="cuda")
            tok, lp = C.sample(z, t, s, False, False) if top_k < 0 else C.sample_topk_topp(z, t, s, False, top_k, 1.0, False)
            assert int(tok) == (0 if more > 0 else 1), (bits, low, more)
            assert abs(float(lp) - float(z.double().log_softmax(-1)[0, int(tok)])) < 1e-4


def _noise_of(seed, col):
    """Noise of one element of row 0, in 64 bits."""
    n = _hash(_hash((col + 0x9E3779B9) & 0xFFFFFFFF) ^ (seed & 0xFFFFFFFF))
    return -math.log(-math.log(((_hash(n ^ (seed >> 32 & 0xFFFFFFFF)) >> 8) + 0.5) / 2 ** 24))


def _seeds_for(col, most):
    """Seeds that give element ``col`` the largest noise (16.5) and element 0 at most ``most``."""
    return [s for s in (_seed_for(0xFFFFFE, col, low) for low in range(1, 4000)) if _noise_of(s, 0) < most][:8]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_nucleus_of_everything(C, dtype):
    """The largest top_p below one, and weights 1 and three of 0.7 * 2^-23: sums of 24 bits round each of the three up, and the mass asked for
    is then more than what the later digits of the keys find.  All of the row is kept, the elements at the low end of a digit among them."""
    z = torch.full((1, 4096), -math.inf, device="cuda")
    z[0, 0], z[0, 1:4] = 25.5, 2.0                          # 23.5 ln 2 = 16.29 apart
    z, scale = z.to(dtype), torch.full((1,), math.log(2.0), device="cuda")
    for seed in _seeds_for(1, 0.1):
        tok, _ = C.sample_topk_topp(z, scale, torch.tensor([seed], device="cuda"), False, -1, 1 - 2.0 ** -24, True)
        assert int(tok) == 1


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("small,kept", [(4, False), (5, True)])
def test_nucleus_mass_is_exact(C, dtype, small, kept):
    """Weights of powers of two: one of 1, 2048 of 2^-20 and a few of 2^-26 beside the first.  The largest top_p below one leaves out
    2^-24 (1 + 2^-9 + ...) at most: four of the smallest, not five.  A sum of 24 bits that starts from 1 loses every one of them."""
    z = torch.full((1, 4096), -math.inf, device="cuda")
    z[0, 0], z[0, 1:1 + small], z[0, 1024:3072] = 60.0, 34.0, 40.0            # 26 ln 2 = 18.02 apart
    z, scale, seeds = z.to(dtype), torch.full((1,), math.log(2.0), device="cuda"), _seeds_for(1, -1.7)
    assert len(seeds) == 8
    for seed in seeds:
        tok, _ = C.sample_topk_topp(z, scale, torch.tensor([seed], device="cuda"), False, -1, 1 - 2.0 ** -24, True)
        assert (int(tok) == 1) == kept


@pytest.mark.parametrize("top_k,top_p", [(-1, 1.0), (20, 0.9)])
def test_forms_of_temperatures(C, top_k, top_p):
    """Temperatures of any shape with an element a row, or one for all, give what a plain vector gives."""
    from polyrl_b200 import ops

    b, v = 6, 5000
    torch.manual_seed(0)
    z, seeds = torch.randn(b, v, device="cuda").mul_(3).bfloat16(), torch.randint(0, 2 ** 62, (b,), device="cuda")
    t = torch.tensor([0.7, 1.0, 0.0, 1.3, 0.5, 2.0], device="cuda")
    sample = lambda temp: ops.sample_tokens(z, temp, seeds, top_k=top_k, top_p=top_p)      # noqa: E731
    want = sample(t)
    for form in (t[:, None], t[None], t.double(), t.repeat(2), torch.stack([t, t], 1)[:, 0], t.view(2, 3)):
        assert all(torch.equal(a, c) for a, c in zip(sample(form), want))
    want = sample(torch.full((b,), 0.7, device="cuda"))
    for form in (0.7, torch.tensor(0.7, device="cuda"), torch.tensor([[0.7]], device="cuda")):
        assert all(torch.equal(a, c) for a, c in zip(sample(form), want))
    with pytest.raises(RuntimeError):
        sample(t[:4])
