"""Backward at head_dim in (64, 128] on pairs of thread blocks: two K/V tiles per work item, products over both.

Checked against the one-block kernel, which the deterministic flag selects: the two share the formulas, round P and dS to 16
bits and sum in fp32, so a gradient differs by the rounding of its 16 bits and by fp32 sums in another order.
"""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# (B, N, N_kv, S_q, S_k, D, options): the fewest tiles that take this path (16, and 24 at head_dim up to 96), pairs with an absent second tile (17), a last
# Q tile of one row, of one block's rows (64) and of one more, fewer and more items than pairs of SMs, query heads in a group
CASES = [
    (1, 1, 1, 2945, 1921, 72, {}),
    (1, 2, 2, 1984, 2100, 128, {"causal": True}),
    (2, 2, 1, 2049, 2048, 104, {"causal": True}),
    (1, 12, 12, 1985, 2177, 128, {}),
    (2, 20, 5, 2048, 2048, 120, {"causal": True}),
    (2, 8, 8, 2000, 2300, 128, {"lens": [1, 1333]}),
    (1, 4, 2, 2048, 2048, 128, {"causal": True, "alibi": True}),
    (1, 2, 2, 2304, 2304, 128, {"tri_block": 384}),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c[:6])) + "-" + "+".join(c[6]))
@pytest.mark.parametrize("f32", [False, True])
def test_against_the_one_block_kernel(case, dtype, f32):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    B, N, N_kv, S_q, S_k, D, opt = case
    g = torch.Generator().manual_seed(S_q + S_k + D)

    def rnd(*shape):
        return torch.randn(*shape, generator=g).to(dtype).cuda()
    q, d_o, k, v = rnd(B, N, S_q, D), rnd(B, N, S_q, D), rnd(B, N_kv, S_k, D), rnd(B, N_kv, S_k, D)
    kw = {x: opt[x] for x in ("causal", "tri_block") if x in opt}
    if "lens" in opt:
        kw["seq_lens"] = torch.tensor(opt["lens"], dtype=torch.int32).cuda()
    if "alibi" in opt:
        kw["alibi"] = (-0.1 * torch.arange(S_k).float()).expand(B, N, 1, S_k).to(dtype).cuda()
    scale = 1.0 / math.sqrt(D)
    o, lse = ops.fa_forward(q, k, v, scale=scale, **kw)
    want = ops.fa_backward(q, k, v, o, lse, d_o, scale=scale, grads_fp32=f32, deterministic=True, **kw)
    # a P or dS that rounds to its other 16-bit neighbour moves a gradient by 2^-11 (fp16) / 2^-8 (bf16) of one term;
    # the terms are of the size of the largest gradient at most
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for _ in range(3):                # (the blocks of a pair meet in another order each time)
        got = ops.fa_backward(q, k, v, o, lse, d_o, scale=scale, grads_fp32=f32, **kw)
        torch.cuda.synchronize()
        _lib.device_status()
        for a, b in zip(got, want):
            assert torch.isfinite(a).all()
            err = (a.float() - b.float()).abs().max().item()
            assert err <= 2 * unit * max(b.float().abs().max().item(), 1e-3)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
def test_keys_past_the_valid_length_do_not_exist(causal, f32, fill):
    """What a padded buffer holds behind the valid keys reaches no gradient, wherever in a pair of tiles the length ends."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import ops
    lens = [0, 128, 384, 2176]
    g = torch.Generator().manual_seed(5)
    q, k, v, d_o = (torch.randn(4, 2, 2304, 128, generator=g).half().cuda() for _ in range(4))
    kw = {"scale": 128 ** -0.5, "causal": causal, "seq_lens": torch.tensor(lens, dtype=torch.int32).cuda()}
    o, lse = ops.fa_forward(q, k, v, **kw)
    want = ops.fa_backward(q, k, v, o, lse, d_o, grads_fp32=f32, deterministic=True, **kw)
    for b, n in enumerate(lens):
        k[b, :, n:] = v[b, :, n:] = fill
    got = ops.fa_backward(q, k, v, o, lse, d_o, grads_fp32=f32, **kw)
    for a, b in zip(got[1:], want[1:]):      # (the sums behind dK and dV have a fixed order)
        assert torch.equal(a, b)
        for i, n in enumerate(lens):
            assert not a[i, :, n:].any()
    # dQ: fp32 sums of up to 17 tiles in another order, rounded to 16 bits unless f32
    bound = (2.0 ** -18 if f32 else 2.0 ** -10) * want[0].float().abs().amax()
    assert (got[0].float() - want[0].float()).abs().amax() <= bound


@pytest.mark.parametrize("S_q, S_k, opt", [
    (2304, 2304, {"causal": True}),                         # the first Q tile of a pair needs its first K/V tile alone
    (2176, 2304, {"causal": True}),                         # and no Q tile needs the last K/V tile
    (2176, 2176, {}),                                       # a pair without a second tile
    (2304, 2304, {"tri_block": 384}),                       # a pair across the end of a row group
    (2304, 2304, {"tri_block": 384, "causal": True}),
    (2100, 2300, {"tri_block": 128, "causal": True}),
])
@pytest.mark.parametrize("where", ["q", "k", "v", "d_o"])
@pytest.mark.parametrize("f32", [False, True])
def test_what_is_not_finite_stays_with_the_tiles_that_see_it(S_q, S_k, opt, where, f32):
    """NaN and infinity reach the gradients that they reach on the one-block kernel, and no others."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import ops
    g = torch.Generator().manual_seed(S_q + S_k)
    t = {n: torch.randn(1, h, s, 128, generator=g).half().cuda() for n, h, s in
         (("q", 2, S_q), ("k", 1, S_k), ("v", 1, S_k), ("d_o", 2, S_q))}
    kw = {"scale": 128 ** -0.5, **opt}
    for row, value in ((5, float("nan")), (200, float("inf")), (450, float("nan")), (S_q - 3, float("inf"))):
        x = {n: u.clone() for n, u in t.items()}
        x[where][0, 0, row] = value
        o, lse = ops.fa_forward(x["q"], x["k"], x["v"], **kw)
        want = ops.fa_backward(x["q"], x["k"], x["v"], o, lse, x["d_o"], grads_fp32=f32, deterministic=True, **kw)
        got = ops.fa_backward(x["q"], x["k"], x["v"], o, lse, x["d_o"], grads_fp32=f32, **kw)
        for a, b in zip(got, want):
            ok = torch.isfinite(b)
            assert torch.equal(torch.isfinite(a), ok)
            # sums of the same fp32 terms in another order, rounded to 16 bits unless f32
            a, b = a.float()[ok], b.float()[ok]
            assert a.numel() == 0 or (a - b).abs().amax() <= (2.0 ** -17 if f32 else 2.0 ** -9) * b.abs().amax()
