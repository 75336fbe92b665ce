"""Performance cases: the work that RL post-training of a language model has this package do, through its public entry points.

A PPO / GRPO step is a rollout (prompts prefilled into the paged cache, decode steps, sampling) and an update (log-probs of the
sampled tokens, then forward and backward of the policy), so the cases are, with the sizes of the model presets:

  blocks   forward and backward of decoder blocks over packed sequences: the micro-batch of an update
  head     the fused LM head: log-prob and entropy of given tokens, alone (scoring) or with its backward (update)
  prefill  blocks over packed prompts that fill the paged cache, from scratch or behind a cached prefix
  decode   one decode step of blocks and LM head over the paged cache, bf16 or fp8 weights
  rollout  the rollout engine: prompts in, then decode steps over given tokens, logits at every step
  sample   tokens and log-probs from a step's logits: greedy, temperature, top-k, top-p

Blocks are stacked one to a few deep, which stands for a model's full depth: every block costs the same.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

from polyrl_b200 import ops
from polyrl_b200.models import ModelConfig, TransformerWeights, get_model_config
from polyrl_b200.models import transformer as tf
from polyrl_b200.rollout.engine import RolloutEngine

PAGE = 16
MODELS = ("qwen2.5-0.5b", "qwen3-1.7b", "qwen2-7b", "llama3-8b")
FP8 = ("wqkv", "wo", "wgu", "wd")


def listed():
    return [
        # the smallest update: a few short sequences through a small policy, where launches count
        dict(name="blocks 0.5b short", kind="blocks", model="qwen2.5-0.5b", layers=2, tokens=387, seqs=3),
        # an ordinary micro-batch of a small policy with query / key norms
        dict(name="blocks 1.7b", kind="blocks", model="qwen3-1.7b", layers=2, tokens=4099, seqs=9),
        # the full micro-batch of an 8B policy: prompt + response of GSM8K length, 16 K tokens at most
        dict(name="blocks 8b full", kind="blocks", model="llama3-8b", layers=1, tokens=12287, seqs=19),
        # update of a small policy: its vocabulary is as large as a big one's, so the head is most of its work
        dict(name="head 0.5b update", kind="head", model="qwen2.5-0.5b", rows=2503, temperature=1.0, grad=True),
        # old log-probs of a batch of responses, 8B
        dict(name="head 8b score", kind="head", model="llama3-8b", rows=6005, temperature=0.7, grad=False),
        # prompts of a GRPO batch
        dict(name="prefill 7b", kind="prefill", model="qwen2-7b", layers=2, tokens=2781, seqs=16, cached=0),
        # next turns of conversations whose earlier turns are in the cache
        dict(name="prefill 8b cached", kind="prefill", model="llama3-8b", layers=2, tokens=1165, seqs=5, cached=2432),
        # a small policy's rollout end to end through the engine
        dict(name="rollout 1.7b", kind="rollout", model="qwen3-1.7b", layers=6, seqs=16, prompt=203, steps=8),
        # the decode step of an 8B rollout at its full batch
        dict(name="decode 8b", kind="decode", model="llama3-8b", layers=2, seqs=128, context=769, fp8=False),
        # a partly drained batch of an fp8 rollout with long responses
        dict(name="decode 7b fp8", kind="decode", model="qwen2-7b", layers=2, seqs=45, context=1900, fp8=True),
        # temperature sampling, the setting of GRPO, at the full batch
        dict(name="sample", kind="sample", seqs=128, vocab=128256, temperature=1.0, top_k=-1, top_p=1.0),
        # nucleus sampling of validation runs
        dict(name="sample nucleus", kind="sample", seqs=47, vocab=151936, temperature=0.7, top_k=-1, top_p=0.95),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("blocks", "blocks", "head", "prefill", "decode", "decode", "rollout", "sample", "sample"))
    if kind == "sample":
        # plain temperature, top-k, nucleus or both; a tenth greedy
        top = rng.choice(((-1, 1.0), (-1, 1.0), (rng.randint(2, 200), 1.0), (-1, rng.uniform(0.5, 0.99)), (rng.randint(2, 200), rng.uniform(0.5, 0.99))))
        return dict(kind=kind, seqs=_log(rng, 1, 256), vocab=rng.choice((32768, 50257, 128256, 151936)),
                    temperature=rng.choice((0.0, 0.6, 0.8, 1.0, 1.0, 1.0, 1.2)), top_k=top[0], top_p=round(top[1], 3))
    if kind == "rollout":
        return dict(kind=kind, model=rng.choice(MODELS[:2]), layers=rng.randint(2, 6), seqs=_log(rng, 1, 64), prompt=_log(rng, 16, 500), steps=rng.randint(2, 12))
    model = rng.choice(MODELS)
    cfg = get_model_config(model)
    if kind == "head":
        grad = rng.random() < 0.5
        return dict(kind=kind, model=model, rows=_log(rng, 32, min(8192, 1.5e13 / (cfg.vocab_size * cfg.hidden_size * (8 if grad else 2)))),
                    temperature=rng.choice((0.7, 1.0, 1.0)), grad=grad)
    if kind == "decode":
        seqs = _log(rng, 1, 256)
        return dict(kind=kind, model=rng.choice(MODELS[2:]), layers=rng.randint(1, 2), seqs=seqs, context=_log(rng, 33, min(8000, 250000 // seqs)), fp8=rng.random() < 0.4)
    block = sum(math.prod(s) for _, s in tf.layer_param_specs(cfg, 0))
    layers = rng.randint(1, 2)
    tokens = _log(rng, 64, min(16384, 2.6e12 / (block * layers)))
    seqs = max(1 + tokens // 3000, _log(rng, 1, max(1, tokens // 40)))
    if kind == "blocks":
        return dict(kind=kind, model=model, layers=layers, tokens=tokens, seqs=seqs)
    cached = rng.choice((0, PAGE * _log(rng, 1, 250)))
    if cached:
        seqs = min(seqs, 8)
        tokens = min(tokens, 2500 * seqs)
    return dict(kind=kind, model=model, layers=layers, tokens=tokens, seqs=seqs, cached=cached)


# ---------------------------------------------------------------------------------------------------------------- inputs
def _config(case) -> ModelConfig:
    c = get_model_config(case["model"])
    return ModelConfig(**{**c.to_dict(), "num_layers": case.get("layers", 1), "eos_token_id": -1})


def _lengths(total: int, n: int, least: int = 1) -> list[int]:
    """``n`` uneven lengths with the given sum: a fixed function of the sizes, as a batch of responses is uneven."""
    r = random.Random(total * 1009 + n)
    share = [0.4 + r.random() for _ in range(n)]
    out = [max(least, int(total * s / sum(share))) for s in share]
    out[-1] += total - sum(out)
    while out[-1] < least:
        i = max(range(n), key=out.__getitem__)
        out[i] -= 1
        out[-1] += 1
    return out


def _gen(seed: int):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _normal(g, *shape, scale=1.0, shift=0.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).mul_(scale).add_(shift)).to(dtype)


def _layer(cfg, g, i) -> dict:
    """Weights at the scale of an initialised or lightly trained policy: projections about 0.02, gains about 1."""
    w = {}
    for name, shape in tf.layer_param_specs(cfg, i):
        if name.startswith("ln") or name.endswith("_norm"):
            w[name] = _normal(g, *shape, scale=0.1, shift=1.0)
        else:
            w[name] = _normal(g, *shape, scale=0.1 if name.startswith("b") else 0.02)
    return w


def _cu(lens):
    return torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(device="cuda", dtype=torch.int32)


def _positions(lens, start=0):
    return torch.cat([torch.arange(start, start + n) for n in lens]).cuda()


def _pages(g, lens):
    """Pages of sequences of the given lengths, scattered over the pool: (table [B, width] int32, number of pages; page 0 is idle)."""
    need = [-(-n // PAGE) for n in lens]
    perm = torch.randperm(sum(need), generator=g, device="cuda").cpu() + 1
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    lo = 0
    for i, n in enumerate(need):
        table[i, :n] = perm[lo:lo + n].int()
        lo += n
    return table.cuda(), sum(need) + 1


def _contexts(case):
    """Sequence lengths of a decode step, the new token included: uneven up to ``context``."""
    r = random.Random(case["context"] * 31 + case["seqs"])
    return [max(1, int(case["context"] * (1.0 if i == 0 else 0.25 + 0.75 * r.random()))) for i in range(case["seqs"])]


def _prompts(case, vocab, seed):
    r = random.Random(int(seed) * 104729 + 3)
    lens = _lengths(case["prompt"] * case["seqs"], case["seqs"], 2)
    return [[r.randrange(vocab) for _ in range(n + case["steps"])] for n in lens], lens


def _logits(case, seed):
    """Rows as a language model gives them: a broad background and a few dozen likely tokens."""
    g = _gen(seed)
    b, v = case["seqs"], case["vocab"]
    z = torch.randn(b, v, generator=g, device="cuda").mul_(1.8)
    likely = torch.randint(0, v, (b, 48), generator=g, device="cuda")
    z.scatter_add_(1, likely, torch.rand(b, 48, generator=g, device="cuda").mul_(14.0))
    seeds = torch.randint(0, 2 ** 62, (b,), generator=g, device="cuda", dtype=torch.int64)
    return z.to(torch.bfloat16), seeds


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        logits, seeds = _logits(case, seed)
        t = case["temperature"]
        return dict(case=case, logits=logits, seeds=seeds, temperature=torch.full((case["seqs"],), t if t > 0 else 1.0, device="cuda"))
    cfg, g = _config(case), _gen(seed)
    if kind == "rollout":
        w = TransformerWeights(cfg, device="cuda", dtype=torch.bfloat16, seed=int(seed))
        toks, lens = _prompts(case, cfg.vocab_size, seed)
        longest = max(map(len, toks))
        eng = RolloutEngine(cfg, torch.device("cuda"), max_num_seqs=case["seqs"], max_model_len=longest + 32,
                            kv_cache_tokens=case["seqs"] * (longest + 64))
        eng.set_weights(w.embed, w.layers, w.head)
        return dict(case=case, engine=eng, tokens=toks, lens=lens)
    if kind == "head":
        h, v, n = cfg.hidden_size, cfg.vocab_size, case["rows"]
        return dict(case=case, hidden=_normal(g, n, h).requires_grad_(case["grad"]), weight=_normal(g, v, h, scale=0.02).requires_grad_(case["grad"]),
                    labels=torch.randint(0, v, (n,), generator=g, device="cuda"), g_lp=_normal(g, n, dtype=torch.float32),
                    g_ent=_normal(g, n, scale=0.05, dtype=torch.float32))
    layers = [_layer(cfg, g, i) for i in range(cfg.num_layers)]
    nkv, d = cfg.num_kv_heads, cfg.head_dim
    if kind == "decode":
        lens = _contexts(case)
        table, pages = _pages(g, lens)
        caches = [(_normal(g, pages, nkv, PAGE, d), _normal(g, pages, nkv, PAGE, d)) for _ in layers]
        at = torch.tensor(lens, device="cuda") - 1
        slot = table.long().gather(1, (at // PAGE)[:, None])[:, 0] * PAGE + at % PAGE
        if case["fp8"]:
            layers = [{k: ops.quantize_weight_fp8(t) if k in FP8 else t for k, t in w.items()} for w in layers]
        v = cfg.vocab_size
        return dict(case=case, cfg=cfg, layers=layers, embed=_normal(g, v, cfg.hidden_size), caches=caches,
                    head={"norm_w": _normal(g, cfg.hidden_size, scale=0.1, shift=1.0), "lm_head": _normal(g, v, cfg.hidden_size, scale=0.02)},
                    inp=tf.DecodeInput(torch.randint(0, v, (len(lens),), generator=g, device="cuda"), at, slot, table,
                                       torch.tensor(lens, dtype=torch.int32, device="cuda"), table.shape[1] * PAGE))
    lens = _lengths(case["tokens"], case["seqs"])
    x = _normal(g, case["tokens"], cfg.hidden_size)
    if kind == "blocks":
        for w in layers:
            for t in w.values():
                t.requires_grad_(True)
        inp = tf.PackedInput(torch.zeros(case["tokens"], dtype=torch.long, device="cuda"), _positions(lens), _cu(lens), max(lens))
        return dict(case=case, cfg=cfg, layers=layers, x=x.requires_grad_(True), inp=inp, gy=_normal(g, *x.shape))
    cached = case["cached"]
    table, pages = _pages(g, [cached + n for n in lens])
    caches = [(_normal(g, pages, nkv, PAGE, d), _normal(g, pages, nkv, PAGE, d)) for _ in layers]
    pos = _positions(lens, cached)
    seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).cuda()
    slots = table.long()[seq, pos // PAGE] * PAGE + pos % PAGE
    gather = None
    if cached:
        full = [cached + n for n in lens]
        kpos, kseq = _positions(full), torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(full)).cuda()
        gather = (table.long()[kseq, kpos // PAGE], kpos % PAGE, _cu(full), max(full))
    inp = tf.PackedInput(torch.zeros(case["tokens"], dtype=torch.long, device="cuda"), pos, _cu(lens), max(lens), kv_gather=gather)
    return dict(case=case, cfg=cfg, layers=layers, x=x, inp=inp, caches=caches, slots=slots)


# ------------------------------------------------------------------------------------------------------------------ pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sample":
        return ops.sample_tokens(s["logits"], s["temperature"], s["seeds"], greedy=case["temperature"] == 0, top_k=case["top_k"], top_p=case["top_p"])
    if kind == "head":
        with torch.set_grad_enabled(case["grad"]):
            lp, ent = ops.linear_cross_entropy(s["hidden"], s["weight"], s["labels"], case["temperature"])
        if not case["grad"]:
            return lp, ent
        dh, dw = torch.autograd.grad((lp, ent), (s["hidden"], s["weight"]), (s["g_lp"], s["g_ent"]))
        return lp.detach(), ent.detach(), dh, dw
    if kind == "blocks":
        x = s["x"]
        for w in s["layers"]:
            x = tf.layer_forward(s["cfg"], w, x, s["inp"])
        leaves = [s["x"]] + [t for w in s["layers"] for t in w.values()]
        return [x.detach(), *torch.autograd.grad(x, leaves, s["gy"])]
    with torch.no_grad():
        if kind == "prefill":
            x = s["x"]
            for w, (k, v) in zip(s["layers"], s["caches"]):
                x = tf.layer_forward(s["cfg"], w, x, s["inp"], kv_sink=(k, v, s["slots"]))
            return [x, *(t for kv in s["caches"] for t in kv)]
        if kind == "decode":
            x, delta = F.embedding(s["inp"].input_ids, s["embed"]), None
            for w, (k, v) in zip(s["layers"], s["caches"]):
                x, delta = tf.layer_decode_fused(s["cfg"], w, x, delta, s["inp"], k, v)
            logits = tf.logits_forward(s["cfg"], s["head"], {}, tf.final_norm(s["cfg"], s["head"], x + delta))
            return [logits, *(t for kv in s["caches"] for t in kv)]
        eng, toks = s["engine"], s["tokens"]
        reqs = [eng.open() for _ in toks]
        out = [eng.extend([(r, t[:n], [n - 1]) for r, t, n in zip(reqs, toks, s["lens"])])]
        for i in range(case["steps"]):
            out.append(eng.extend([(r, t[n + i:n + i + 1], [0]) for r, t, n in zip(reqs, toks, s["lens"])]))
        for r in reqs:
            eng.close(r)
        return torch.stack(out)


# ------------------------------------------------------------------------------------------------------------------ work
def _pairs(lens, cached=0):
    return sum(n * (n + 1) // 2 + n * cached for n in lens)


def work(case):
    kind = case["kind"]
    if kind == "sample":
        n = case["seqs"] * case["vocab"]
        return {"bytes": 2 * n, "flops": 10 * n}
    cfg = _config(case)
    h, v, nq, d = cfg.hidden_size, cfg.vocab_size, cfg.num_heads, cfg.head_dim
    block = sum(math.prod(s) for _, s in tf.layer_param_specs(cfg, 0))
    kv = 2 * cfg.kv_size * 2                                     # bytes of a token's keys and values in one block
    if kind == "head":
        n = case["rows"]
        return {"bytes": (2 if case["grad"] else 1) * 2 * (n * h + v * h) + 16 * n, "flops": (8 if case["grad"] else 2) * n * v * h}
    if kind == "decode":
        lens = _contexts(case)
        return {"bytes": cfg.num_layers * (block * (1 if case["fp8"] else 2) + sum(lens) * kv) + 2 * v * h + 2 * len(lens) * v,
                "flops": 2 * len(lens) * (cfg.num_layers * block + v * h) + cfg.num_layers * sum(lens) * 4 * nq * d}
    if kind == "rollout":
        lens, steps, b = _lengths(case["prompt"] * case["seqs"], case["seqs"], 2), case["steps"], case["seqs"]
        seen = sum(lens) * steps + b * steps * (steps + 1) // 2
        return {"bytes": (steps + 1) * (cfg.num_layers * block * 2 + 2 * v * h) + cfg.num_layers * (seen + sum(lens)) * kv + 4 * (steps + 1) * b * v,
                "flops": 2 * cfg.num_layers * block * (sum(lens) + b * steps) + 2 * (steps + 1) * b * v * h + cfg.num_layers * 4 * nq * d * (_pairs(lens) + seen)}
    t, lens = case["tokens"], _lengths(case["tokens"], case["seqs"])
    pairs = _pairs(lens, case.get("cached", 0))
    if kind == "blocks":
        return {"bytes": cfg.num_layers * block * 4 + 8 * t * h, "flops": cfg.num_layers * (6 * block * t + 14 * nq * d * pairs)}
    return {"bytes": cfg.num_layers * (block * 2 + (t + case["seqs"] * case["cached"]) * kv) + 4 * t * h, "flops": cfg.num_layers * (2 * block * t + 4 * nq * d * pairs)}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}         # 32-bit sums; a tie of two noisy logits may go either way
    if kind == "head":
        return {"rel": 1e-2, "max": 0.3} if case["grad"] else {"rel": 1e-5, "max": 1e-3}
    if kind == "decode" and case["fp8"]:
        return {"rel": 3e-2, "max": 0.5}                          # activations in e4m3: a last-bit difference before it moves a value by 1/16
    if kind == "rollout":
        return {"rel": 3e-2, "max": 0.5}                          # a stack of blocks, each of them rounding its results to bf16
    return {"rel": 2e-2, "max": 0.3}


# ----------------------------------------------------------------------------------------------------------- in 64 bits
def _rms64(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _turn64(x, pos, theta):
    """Rotate-half of x [T, heads, d]."""
    d = x.shape[-1]
    a = pos.double()[:, None] * theta ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    c, s = a.cos()[:, None], a.sin()[:, None]
    lo, hi = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _qkv64(cfg, w, x, pos):
    nq, nkv, d = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
    p = _rms64(x, w["ln1"], cfg.rms_norm_eps) @ w["wqkv"].t()
    p = (p + w["bqkv"] if "bqkv" in w else p).view(-1, nq + 2 * nkv, d)
    q, k, v = p[:, :nq], p[:, nq:nq + nkv], p[:, nq + nkv:]
    if "q_norm" in w:
        q, k = _rms64(q, w["q_norm"], cfg.rms_norm_eps), _rms64(k, w["k_norm"], cfg.rms_norm_eps)
    return _turn64(q, pos, cfg.rope_theta), _turn64(k, pos, cfg.rope_theta), v


def _attend64(q, k, v):
    """q [n, nq, d] against k, v [m, nkv, d], the queries being the last n of m places."""
    n, m, r = q.shape[0], k.shape[0], q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(r, 1), v.repeat_interleave(r, 1)
    z = torch.einsum("qhd,khd->hqk", q, k) * q.shape[-1] ** -0.5
    hide = torch.ones(n, m, dtype=torch.bool, device=q.device).triu(m - n + 1)
    return torch.einsum("hqk,khd->qhd", z.masked_fill(hide, -math.inf).softmax(-1), v).flatten(1)


def _after64(cfg, w, x, a):
    x = x + a @ w["wo"].t()
    gu = (_rms64(x, w["ln2"], cfg.rms_norm_eps) @ w["wgu"].t()).view(x.shape[0], -1, 2, 128)
    return x + (F.silu(gu[:, :, 0]) * gu[:, :, 1]).flatten(1) @ w["wd"].t()


def _packed64(cfg, w, x, pos, lens):
    q, k, v = _qkv64(cfg, w, x, pos)
    a = torch.cat([_attend64(*t) for t in zip(q.split(lens), k.split(lens), v.split(lens))])
    return _after64(cfg, w, x, a)


def _wide(w):
    return {k: t.detach().double() for k, t in w.items()}


def _hash(x):
    """The 32-bit mixer of the sampler's noise, on int64 tensors."""
    m = 0xFFFFFFFF
    x = ((x ^ (x >> 16)) * 0x7FEB352D) & m
    x = ((x ^ (x >> 15)) * 0x846CA68B) & m
    return x ^ (x >> 16)


def _sample64(case, s):
    z, toks, lps = s["logits"].double(), [], []
    b, v = z.shape
    greedy, col = case["temperature"] == 0, torch.arange(v, device=z.device)
    for i in range(b):
        row = z[i] / (1.0 if greedy else case["temperature"])
        top, _ = row.sort(descending=True)
        cut = top[min(v, case["top_k"]) - 1] if case["top_k"] > 0 else top[-1]
        if case["top_p"] < 1 and not greedy:
            kept = top[top >= cut]
            p = kept.softmax(0)
            cut = kept[(p.cumsum(0) - p < case["top_p"])][-1]
        row = row.masked_fill(row < cut, -math.inf)
        seed = int(s["seeds"][i])
        n = _hash(_hash((col + 0x9E3779B9 * (i + 1)) & 0xFFFFFFFF) ^ (seed & 0xFFFFFFFF))
        u = ((_hash(n ^ (seed >> 32)) >> 8).double() + 0.5) / 16777216.0
        t = int((row if greedy else row - torch.log(-torch.log(u))).argmax())
        toks.append(t)
        lps.append(row.log_softmax(0)[t])
    return torch.tensor(toks), torch.stack(lps)


def _head64(case, s):
    w, lab, tau = s["weight"].detach().double(), s["labels"], case["temperature"]
    lps, ents, dhs = [], [], []
    dw = torch.zeros_like(w) if case["grad"] else None
    for lo in range(0, case["rows"], 512):
        c = slice(lo, lo + 512)
        h = s["hidden"].detach()[c].double()
        logp = (h @ w.t()).div_(tau).log_softmax(-1)
        p, at = logp.exp(), lab[c, None]
        lp, ent = logp.gather(1, at)[:, 0], -(p * logp).sum(-1)
        lps.append(lp)
        ents.append(ent)
        if case["grad"]:
            gl, ge = s["g_lp"][c, None].double(), s["g_ent"][c, None].double()
            dz = -gl * p - ge * p * (logp + ent[:, None])
            dz.scatter_add_(1, at, gl)
            dz /= tau
            dhs.append(dz @ w)
            dw += dz.t() @ h
    return (torch.cat(lps), torch.cat(ents)) + ((torch.cat(dhs), dw) if case["grad"] else ())


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample" and case["temperature"] > 0 and case["top_k"] < 0 and case["top_p"] >= 1:
        return None                         # over a whole vocabulary the last bits of the sampler's noise decide some rows
    s = prepare(case, seed)
    if kind == "sample":
        return _sample64(case, s)
    if kind == "head":
        return _head64(case, s)
    if kind == "rollout":
        cfg, eng, lens = s["engine"].cfg, s["engine"], s["lens"]
        full = [len(t) for t in s["tokens"]]
        pos = _positions(full)
        with torch.no_grad():
            x = eng.embed_w["embed"].double()[torch.tensor([i for t in s["tokens"] for i in t], device="cuda")]
            for w in eng.layer_w:
                x = _packed64(cfg, _wide(w), x, pos, full)
            start = torch.tensor([0] + full).cumsum(0)[:-1] + torch.tensor(lens) - 1
            rows = torch.stack([x[(start + i).cuda()] for i in range(case["steps"] + 1)])
            head = eng.embed_w["embed"] if cfg.tie_word_embeddings else eng.head_w["lm_head"]
            return _rms64(rows, eng.head_w["norm_w"].double(), cfg.rms_norm_eps) @ head.double().t()
    cfg = s["cfg"]
    if kind == "blocks":
        layers = [{k: t.requires_grad_(True) for k, t in _wide(w).items()} for w in s["layers"]]
        x0 = s["x"].detach().double().requires_grad_(True)
        x, lens = x0, _lengths(case["tokens"], case["seqs"])
        for w in layers:
            x = _packed64(cfg, w, x, s["inp"].position_ids, lens)
        return [x.detach(), *torch.autograd.grad(x, [x0] + [t for w in layers for t in w.values()], s["gy"].double())]
    with torch.no_grad():
        caches, pos = [[t.double() for t in kv] for kv in s["caches"]], s["inp"].position_ids
        if kind == "prefill":
            x, lens, slots, table = s["x"].double(), _lengths(case["tokens"], case["seqs"]), s["slots"], s["inp"].kv_gather
            full = [case["cached"] + n for n in lens]
        else:
            x, lens, slots, full = s["embed"].double()[s["inp"].input_ids], [1] * case["seqs"], s["inp"].slot_mapping, _contexts(case)
        for w, (ck, cv) in zip(s["layers"], caches):
            if case.get("fp8"):
                w = {k: (t.q.float() * t.scale[:, None]) if k in FP8 else t for k, t in w.items()}
            w = _wide(w)
            q, k, v = _qkv64(cfg, w, x, pos)
            ck[slots // PAGE, :, slots % PAGE], cv[slots // PAGE, :, slots % PAGE] = k, v
            if kind == "prefill" and table is None:
                keys, values = k.split(lens), v.split(lens)
            elif kind == "prefill":
                keys, values = (c[table[0], :, table[1]].split(full) for c in (ck, cv))
            else:
                keys, values = ([c[t.long()].transpose(1, 2).flatten(0, 1)[:n] for t, n in zip(s["inp"].block_table, full)] for c in (ck, cv))
            a = torch.cat([_attend64(*t) for t in zip(q.split(lens), keys, values)])
            x = _after64(cfg, w, x, a)
        if kind == "decode":
            x = _rms64(x, s["head"]["norm_w"].double(), cfg.rms_norm_eps) @ s["head"]["lm_head"].double().t()
        return [x, *(t for kv in caches for t in kv)]
