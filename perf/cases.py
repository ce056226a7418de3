"""The attention work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values.  Every kind goes through the entry point that such a program calls:

* ``train``     the ``FlashAttention`` cell, forward and backward through autograd;
* ``triangle``  the ``TriangleAttention`` cell, forward and backward;
* ``prefill``   the inference op ``flash_attention_tik`` on whole prompts (or on image tokens);
* ``decode``    one token per sequence over a key/value cache, contiguous or paged.

Sizes are those of the benchmark configurations and of the shapes that the tests use, and generic ones around them.
``work`` counts what the operation needs (scores that a mask, a band or a valid length excludes are not counted), each
input read once and each output written once.
"""
import math

import torch

from acctransformer_b200 import FlashAttention, TriangleAttention, flash_attention_decode, flash_attention_tik, ops
from acctransformer_b200.infer.flash_attention import DecodeWorkspace

DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}
BLOCK = 128        # the block that prev_block_num / next_block_num count
PAGE = 64          # rows of a page of the paged caches


def _case(name, kind, dtype, B, N, S_q, S_k, D, N_kv=None, **more):
    c = {"kind": kind, "dtype": dtype, "B": B, "N": N, "N_kv": N_kv or N, "S_q": S_q, "S_k": S_k, "D": D,
         "mask": "none", "docs": 0, "alibi": False, "prev": -1, "next": -1, "drop": 0.0, "block": 0,
         "lens": False, "fused": False, "paged": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a text encoder of an image generator: 77 tokens, causal; nothing but launch and call overhead
        _case("prefill-text", "prefill", "float16", 2, 12, 77, 77, 64, mask="causal"),
        # self-attention over the 64x64 latent of an image generator: narrow heads, every key visible
        _case("prefill-image", "prefill", "float16", 2, 8, 4096, 4096, 40),
        # long prompts of a serving batch
        _case("prefill-batch", "prefill", "float16", 8, 32, 4096, 4096, 128, mask="causal"),
        # one decoding step of a few interactive users: grouped heads, paged cache, short contexts
        _case("decode-step", "decode", "bfloat16", 4, 32, 1, 2048, 128, N_kv=8, lens=True, paged=True),
        # one decoding step of a full serving batch with long contexts of different lengths
        _case("decode-batch", "decode", "float16", 32, 32, 1, 16384, 128, lens=True),
        # a small model while it is being developed: short sequences, the causal mask given as the reference gives it
        _case("train-small", "train", "float16", 2, 8, 256, 256, 64, mask="causal"),
        # a mid-sized language model with alibi positions
        _case("train-alibi", "train", "float16", 4, 16, 2048, 2048, 128, mask="causal", alibi=True),
        # long-context causal training: the headline configuration
        _case("train-long", "train", "float16", 2, 32, 8192, 8192, 128, mask="causal"),
        # local attention with dropout
        _case("train-band", "train", "bfloat16", 2, 32, 8192, 8192, 128, prev=4, next=4, drop=0.1),
        # packed documents of a ragged length, grouped heads, q / k / v as views of one fused projection
        _case("train-documents", "train", "bfloat16", 2, 32, 3000, 3000, 128, N_kv=8, mask="docs", docs=4, fused=True),
        # the innermost level of an image generator: wide heads, few tokens
        _case("train-wide", "train", "float16", 8, 8, 1024, 1024, 160),
        # TriangleAttention over a causal mask
        _case("train-triangle", "triangle", "float16", 8, 32, 4096, 4096, 128, mask="causal", block=512),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_batch(rng, cost_of_one, most, cap=16):
    """A batch size whose cost stays below ``most``."""
    fit = int(most / cost_of_one)
    return _log_int(rng, 1, max(1, min(cap, fit)))


def draw(rng):
    kind = rng.choice(["train"] * 5 + ["triangle"] + ["prefill"] * 3 + ["decode"] * 3)
    dtype = rng.choice(["float16", "bfloat16"])
    if kind == "decode":
        N_kv, group = rng.choice([4, 8, 16, 32]), rng.choice([1, 1, 4, 8])
        D = rng.choice([64, 128, 128])
        S = _log_int(rng, 128, 16384)
        paged = rng.random() < 0.4
        if paged:
            S = -(-S // PAGE) * PAGE
        B = _draw_batch(rng, 4.0 * N_kv * S * D, 6e9, 64)
        return _case(None, "decode", dtype, B, N_kv * group, 1, S, D, N_kv=N_kv, lens=True, paged=paged)
    D = rng.choice([64, 64, 128, 128, 128, 40, 80, 160])
    N = rng.choice([4, 8, 12, 16, 32])
    S = _log_int(rng, 64, 8192)
    if rng.random() < 0.4:
        S = -(-S // BLOCK) * BLOCK
    c = _case(None, kind, dtype, 1, N, S, S, D)
    if kind == "prefill":
        if rng.random() < 0.6:
            c.update(mask="causal", lens=rng.random() < 0.5)
        elif rng.random() < 0.3:
            c.update(S_k=77)                                     # cross-attention to a text
    elif kind == "triangle":
        c.update(mask="causal", block=rng.choice([256, 512]))
    else:
        form = rng.choice(["causal", "causal", "alibi", "band", "docs", "none"])
        c.update(drop=0.1 if rng.random() < 0.3 else 0.0, fused=rng.random() < 0.5)
        if D <= 128 and rng.random() < 0.3:
            c.update(N_kv=N // 4)
        if form == "alibi":
            c.update(mask="causal", alibi=True)
        elif form == "band":
            c.update(prev=rng.choice([1, 2, 4, 8]), next=rng.choice([0, 1, 4]))
        elif form == "docs":
            c.update(mask="docs", docs=rng.choice([2, 4, 8]), S_q=min(S, 4096), S_k=min(S, 4096))
        else:
            c.update(mask=form)
    dense = 4.0 * c["N"] * c["S_q"] * c["S_k"] * c["D"] * (1.0 if kind == "prefill" else 3.5)
    c["B"] = _draw_batch(rng, dense, 1.5e12 if D > 128 else 4e12)
    return c


def _pairs(c):
    """Score positions of one (batch, head) slice that take part (the expected number where lengths are drawn)."""
    S_q, S_k = c["S_q"], c["S_k"]
    if c["mask"] == "docs":
        return S_q * S_k / (c["docs"] + 1.0)                     # uniform boundaries; causal inside each document
    if c["prev"] >= 0:
        total = 0
        for i in range(-(-S_q // BLOCK)):
            lo, hi = max(0, i - c["prev"]) * BLOCK, min(S_k, (i + c["next"] + 1) * BLOCK)
            total += min(BLOCK, S_q - i * BLOCK) * max(0, hi - lo)
        return total
    if c["mask"] == "causal":
        full = S_q * (S_q + 1) / 2.0                             # S_q = S_k
        return full * 0.8125 if c["lens"] else full              # valid lengths uniform in [S/4, S]
    return S_q * S_k * (0.625 if c["lens"] else 1.0)


def work(case):
    c = case
    q = c["B"] * c["N"] * c["S_q"] * c["D"] * 2.0
    kv = 2.0 * c["B"] * c["N_kv"] * c["S_k"] * c["D"] * 2.0      # keys and values
    pairs = c["B"] * c["N"] * _pairs(c)
    if c["kind"] == "decode":
        return {"bytes": 2 * q + 0.625 * kv, "flops": 4.0 * pairs * c["D"]}
    if c["kind"] == "prefill":
        return {"bytes": 2 * q + kv, "flops": 4.0 * pairs * c["D"]}
    extra = 2.0 * c["B"] * c["S_q"] * c["S_k"] if c["mask"] == "docs" else 0.0
    # forward: q, k, v -> o; backward: q, k, v, o, dO -> dq, dk, dv (five products for the forward's two)
    return {"bytes": 2 * q + kv + 4 * q + 2 * kv + extra, "flops": 3.5 * 4.0 * pairs * c["D"]}


def tolerance(case):
    # half-precision probabilities, score gradients and results: a handful of roundings of 2^-9 (bf16) or 2^-12 (fp16)
    # of the values' size each, on top of fp32 sums
    return {"rel": 1e-2} if case["dtype"] == "bfloat16" else {"rel": 2e-3}


def _lengths(c, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(max(1, c["S_k"] // 4), c["S_k"] + 1, (c["B"],), generator=g, dtype=torch.int32)


def _mask(c, dt, seed):
    """The mask tensor as the reference's users build it: 1 where a key must not be seen, in the inputs' type."""
    S_q, S_k = c["S_q"], c["S_k"]
    if c["mask"] == "causal":
        return torch.triu(torch.ones(1, S_q, S_k, device="cuda", dtype=dt), diagonal=1)
    if c["mask"] != "docs":
        return None
    g = torch.Generator().manual_seed(seed)
    pos = torch.arange(S_q, device="cuda")
    rows = []
    for _ in range(c["B"]):
        cuts = torch.randint(1, S_q, (c["docs"] - 1,), generator=g).sort().values.cuda()
        doc = torch.bucketize(pos, cuts, right=True)
        rows.append(((doc[:, None] != doc[None, :]) | (pos[None, :] > pos[:, None])).to(dt))
    return torch.stack(rows)


def prepare(case, seed):
    c = case
    dt, dev = DTYPES[c["dtype"]], "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    B, N, N_kv, S_q, S_k, D = (c[k] for k in ("B", "N", "N_kv", "S_q", "S_k", "D"))

    def normal(*shape, std=1.0):
        return torch.empty(shape, device=dev, dtype=dt).normal_(0.0, std, generator=g)

    s = {"case": c}
    if c["kind"] == "decode":
        s["q"] = normal(B, N, 1, D)
        lens = _lengths(c, seed)
        s["lens"] = lens.to(dev)
        if c["paged"]:
            pages = S_k // PAGE
            s["k"], s["v"] = normal(B * pages, N_kv, PAGE, D), normal(B * pages, N_kv, PAGE, D)
            order = torch.randperm(B * pages, generator=torch.Generator().manual_seed(seed))
            s["table"] = order.to(torch.int32).view(B, pages).to(dev)
        else:
            s["k"], s["v"] = normal(B, N_kv, S_k, D), normal(B, N_kv, S_k, D)
        s["workspace"] = DecodeWorkspace(B, N, D, dev)           # kept by the serving loop
        return s
    std = 0.5 if c["prev"] >= 0 else 1.0
    if c["fused"]:
        x = normal(B, S_q, (N + 2 * N_kv) * D, std=std)          # one projection's output; S_q = S_k
        q, k, v = x.split([N * D, N_kv * D, N_kv * D], dim=2)
        q, k, v = (t.view(B, S_q, -1, D).transpose(1, 2) for t in (q, k, v))
    else:
        q, k, v = normal(B, N, S_q, D, std=std), normal(B, N_kv, S_k, D, std=std), normal(B, N_kv, S_k, D, std=std)
    if c["kind"] == "prefill":
        s.update(q=q, k=k, v=v, lens=_lengths(c, seed).to(dev) if c["lens"] else None)
        return s
    if c["kind"] == "triangle":
        q.mul_(D ** -0.5)                                        # the caller of this cell scales q itself
        s["layer"] = TriangleAttention(block_size=c["block"], dropout_rate=c["drop"])
    else:
        band = dict(prev_block_num=c["prev"], next_block_num=c["next"]) if c["prev"] >= 0 else {}
        s["layer"] = FlashAttention(D, dropout_rate=c["drop"], alibi=c["alibi"], **band)
        s["layer"].allow_grouped_kv = N_kv != N
    s["layer"].train()
    s["layer"].generator = torch.Generator().manual_seed(seed)
    s["mask"] = _mask(c, dt, seed)
    s["alibi"] = None
    if c["alibi"]:
        slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / N) for h in range(N)], device=dev)
        s["alibi"] = (slopes.view(1, N, 1, 1) * torch.arange(S_k, device=dev).view(1, 1, 1, S_k)).expand(B, N, 1, S_k) \
            .to(dt).contiguous()
    s.update(q=q.detach().requires_grad_(), k=k.detach().requires_grad_(), v=v.detach().requires_grad_())
    s["d_out"] = normal(B, S_q, N, D) if c["fused"] else normal(B, N, S_q, D)
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "decode":
        if c["paged"]:
            return ops.infer_decode(s["q"], s["k"], s["v"], s["lens"], workspace=s["workspace"], block_table=s["table"])
        return flash_attention_decode(s["q"], s["k"], s["v"], s["lens"], workspace=s["workspace"])
    if c["kind"] == "prefill":
        return flash_attention_tik(s["q"], s["k"], s["v"], scale=c["D"] ** -0.5, causal=c["mask"] == "causal",
                                   seq_lens=s["lens"])
    if c["kind"] == "triangle":
        out = s["layer"](s["q"], s["k"], s["v"], s["mask"])
    else:
        out = s["layer"](s["q"], s["k"], s["v"], s["mask"], s["alibi"])
    if c["fused"]:
        out = out.transpose(1, 2)                                # [B, S, N, D]: what the output projection reads
    return (out,) + torch.autograd.grad(out, (s["q"], s["k"], s["v"]), s["d_out"])
