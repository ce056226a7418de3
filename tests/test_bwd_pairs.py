"""Backward at head_dim in (64, 128] on pairs of thread blocks: two K/V tiles per work item, products over both.

Checked against the one-block kernel, which the deterministic flag selects, and against float64.  The two kernels share the
formulas, the roundings of P and dS to 16 bits and the products behind them, so their gradients differ by fp32 sums in another
order and the last rounding.
"""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# (B, N, N_kv, S_q, S_k, D, options): the fewest tiles that take this path (16, and 24 at head_dim up to 96), pairs with an
# absent second tile, a last Q tile of one row, of one block's rows (64) and of one more, fewer and more items than pairs of SMs,
# query heads in a group, pairs of which no Q tile needs the second K/V tile or either of them
CASES = [
    (1, 1, 1, 2945, 1921, 72, {}),
    (1, 2, 2, 1984, 2100, 128, {"causal": True}),
    (2, 2, 1, 2049, 2048, 104, {"causal": True}),
    (1, 12, 12, 1985, 2177, 128, {}),
    (2, 20, 5, 2048, 2048, 120, {"causal": True}),
    (1, 2, 2, 2304, 2304, 128, {"tri_block": 384}),
    (1, 4, 1, 2176, 4200, 128, {"causal": True}),
    (1, 2, 1, 8191, 2100, 96, {"causal": True}),
]


def kernel_of(q, k, causal=False, tri_block=0):
    from acctransformer_b200 import _lib
    a = _lib.FaArgs()
    a.B, a.N, a.S_q, a.D = q.shape
    a.N_kv, a.S_k = k.shape[1:3]
    a.causal, a.tri_block = int(causal), tri_block
    a.prev_block_num = a.next_block_num = _lib.BAND_UNBOUNDED
    return _lib.load().acct_fa_bwd_kernel(C.byref(a))


def assert_same_sums(got, want, steps):
    """Gradients of the two kernels, tile by tile: a late tile under a causal mask is small beside the early ones."""
    for a, b in zip(got, want):
        # 16 bits: values next to one another at most, beside what the sums differ by
        ulp = {torch.float32: 0.0, torch.float16: 2.0 ** -10, torch.bfloat16: 2.0 ** -7}[b.dtype]
        tiny = {torch.float32: 0.0, torch.float16: 2.0 ** -24, torch.bfloat16: 2.0 ** -133}[b.dtype]
        a, b = a.float(), b.float()
        assert torch.isfinite(a).all()
        for i in range(0, b.shape[2], 128):
            x, y = a[:, :, i:i + 128], b[:, :, i:i + 128]
            # 8 additions per 128 positions, each off by 2^-23 (a truncated sum) of a partial sum, which is no larger than the
            # largest results of its tile; on both sides
            size = y.abs().amax(dim=(2, 3), keepdim=True)
            assert ((x - y).abs() <= 2 * 8 * steps * 2.0 ** -23 * size + ulp * y.abs() + tiny).all()
            assert not x[(y == 0).all(-1)].any()      # no query sees the key, or the other way round


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
    assert kernel_of(q, k, **opt) == _lib.BWD_PAIR
    scale = 1.0 / math.sqrt(D)
    o, lse = ops.fa_forward(q, k, v, scale=scale, **opt)
    want = ops.fa_backward(q, k, v, o, lse, d_o, scale=scale, grads_fp32=f32, deterministic=True, **opt)
    for _ in range(3):                # (the blocks of a pair meet in another order each time)
        got = ops.fa_backward(q, k, v, o, lse, d_o, scale=scale, grads_fp32=f32, **opt)
        torch.cuda.synchronize()
        _lib.device_status()
        assert_same_sums(got, want, -(-max(S_q * N // N_kv, S_k) // 128))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S, N, N_kv, opt", [(2048, 2, 2, {}), (2100, 4, 1, {"causal": True}), (2200, 2, 1, {"tri_block": 640}),
                                             (2304, 2, 2, {"tri_block": 384, "causal": True})])
def test_views_of_a_projection_against_float64(S, N, N_kv, opt, dtype):
    """q, k, v as views of one fused projection, o and its gradient in the layout of the output projection."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    B, D = 2, 128
    g = torch.Generator().manual_seed(S)
    x = torch.randn(B, S, (N + 2 * N_kv) * D, generator=g).to(dtype).cuda()
    q, k, v = (t.view(B, S, -1, D).transpose(1, 2) for t in x.split([N * D, N_kv * D, N_kv * D], dim=2))
    d_o = torch.randn(B, S, N, D, generator=g).to(dtype).cuda().transpose(1, 2)
    assert kernel_of(q, k, **opt) == _lib.BWD_PAIR
    out = torch.empty(B, S, N, D, dtype=dtype, device="cuda").transpose(1, 2)
    o, lse = ops.fa_forward(q, k, v, scale=D ** -0.5, **opt)
    out.copy_(o)
    got = (out,) + tuple(ops.fa_backward(q, k, v, out, lse, d_o, scale=D ** -0.5, **opt))
    _lib.device_status()
    qd, kd, vd = (t.double().detach().requires_grad_() for t in (q, k, v))
    s = qd @ kd.repeat_interleave(N // N_kv, 1).transpose(-1, -2) * D ** -0.5
    row, col = torch.arange(S, device="cuda")[:, None], torch.arange(S, device="cuda")[None]
    if opt.get("causal"):
        s = s.masked_fill(col > row, -math.inf)
    if "tri_block" in opt:
        s = s.masked_fill(col >= (row // opt["tri_block"] + 1) * opt["tri_block"], -math.inf)
    ref = torch.softmax(s, -1) @ vd.repeat_interleave(N // N_kv, 1)
    want = (ref,) + torch.autograd.grad(ref, (qd, kd, vd), d_o.double())
    for a, b in zip(got, want):
        # a handful of roundings to 16 bits (2^-9, 2^-12 of the values' size each), tile by tile
        for i in range(0, S, 128):
            y = b[:, :, i:i + 128]
            assert (a[:, :, i:i + 128].double() - y).norm() <= (1e-2 if dtype == torch.bfloat16 else 2e-3) * y.norm()


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
    from acctransformer_b200 import _lib, ops
    g = torch.Generator().manual_seed(S_q + S_k)
    t = {n: torch.randn(1, h, s, 128, generator=g).half().cuda() for n, h, s in
         (("q", 2, S_q), ("k", 1, S_k), ("v", 1, S_k), ("d_o", 2, S_q))}
    kw = {"scale": 128 ** -0.5, **opt}
    assert kernel_of(t["q"], t["k"], **opt) == _lib.BWD_PAIR
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
