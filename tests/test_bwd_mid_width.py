"""Backward at head_dim in (128, 160]: one thread block holds dK and dV of a K/V tile whole, in steps of 64 queries.

Checked against the split-width kernel, which the deterministic flag selects: two kernels that share the formulas and the
keep bits of in-kernel dropout (those are checked against the oracle below, that kernel elsewhere).  Both round P and dS to
16 bits and sum in fp32, so a gradient differs by the rounding of its 16 bits and by fp32 sums in another order.
"""
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref as ref

pytestmark = pytest.mark.gpu

# (B, N, N_kv, S_q, S_k, D, options): one partial tile; a Q tile whose second half is empty (64 rows) or holds one row
# (65); tile edges; one K/V tile without any Q tile; every MODE of the kernel
CASES = [
    (1, 1, 1, 1, 1, 136, {}),
    (1, 2, 2, 64, 129, 160, {}),
    (2, 2, 1, 65, 128, 144, {"causal": True}),
    (1, 4, 2, 321, 257, 160, {"causal": True}),
    (1, 2, 2, 700, 300, 152, {"prev_block_num": 1, "next_block_num": 0}),
    (2, 2, 2, 200, 500, 160, {"lens": [1, 333]}),
    (1, 2, 2, 256, 384, 160, {"philox": True}),
    (1, 2, 1, 300, 300, 160, {"philox": True, "causal": True, "alibi": True}),
    (1, 2, 2, 260, 330, 160, {"mask": True}),
    (1, 2, 2, 193, 190, 136, {"drop": True, "mask": True}),
    (1, 2, 2, 384, 384, 160, {"tri_block": 256}),
    (1, 2, 2, 384, 384, 160, {"tri_block": 96}),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c[:6])) + "-" + "+".join(c[6]))
@pytest.mark.parametrize("f32", [False, True])
def test_against_the_split_width_kernel(case, dtype, f32):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    B, N, N_kv, S_q, S_k, D, opt = case
    g = torch.Generator().manual_seed(S_q + S_k + D)

    def rnd(*shape):
        return torch.randn(*shape, generator=g).to(dtype).cuda()
    q, d_o, k, v = rnd(B, N, S_q, D), rnd(B, N, S_q, D), rnd(B, N_kv, S_k, D), rnd(B, N_kv, S_k, D)
    kw = {x: opt[x] for x in ("causal", "prev_block_num", "next_block_num", "tri_block") if x in opt}
    mask = None
    if "mask" in opt:
        mask = (torch.rand(1, S_q, S_k, generator=g) < 0.3).to(dtype).cuda()
    if "lens" in opt:
        kw["seq_lens"] = torch.tensor(opt["lens"], dtype=torch.int32).cuda()
    if "alibi" in opt:
        kw["alibi"] = (-0.1 * torch.arange(S_k).float()).expand(B, N, 1, S_k).to(dtype).cuda()
    if "philox" in opt:
        kw.update(keep_prob=0.75, dropout_seed=11, dropout_offset=3)
    if "drop" in opt:
        kw.update(keep_prob=0.75, dropout_mask=(torch.rand(B, N, S_q, S_k, generator=g) < 0.75).to(torch.uint8).cuda())
    scale = 1.0 / math.sqrt(D)
    o, lse = ops.fa_forward(q, k, v, mask, scale=scale, **kw)
    got = ops.fa_backward(q, k, v, o, lse, d_o, mask, scale=scale, grads_fp32=f32, **kw)
    want = ops.fa_backward(q, k, v, o, lse, d_o, mask, scale=scale, grads_fp32=f32, deterministic=True, **kw)
    torch.cuda.synchronize()
    _lib.device_status()
    # a P or dS that rounds to its other 16-bit neighbour moves a gradient by 2^-11 (fp16) / 2^-8 (bf16) of one term;
    # the terms are of the size of the largest gradient at most
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(got, want):
        assert torch.isfinite(a).all()
        err = (a.float() - b.float()).abs().max().item()
        assert err <= 2 * unit * max(b.float().abs().max().item(), 1e-3)


@pytest.mark.parametrize("causal", [False, True])
def test_in_kernel_dropout_against_the_oracle(causal):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    S, D = 200, 160
    g = torch.Generator().manual_seed(D)
    q, k, v, d_o = (torch.randn(1, 2, S, D, generator=g).half() for _ in range(4))
    scale, kw = 1.0 / math.sqrt(D), dict(causal=causal, keep_prob=0.75, dropout_seed=11, dropout_offset=3)
    o, lse = ops.fa_forward(q.cuda(), k.cuda(), v.cuda(), scale=scale, **kw)
    got = ops.fa_backward(q.cuda(), k.cuda(), v.cuda(), o, lse, d_o.cuda(), scale=scale, grads_fp32=True, **kw)
    torch.cuda.synchronize()
    _lib.device_status()
    drop = ops.dropout_mask(1, 2, S, S, 0.75, 11, 3).cpu().numpy()
    want = ref.sa_grad(*(t.float().numpy() for t in (q, k, v, d_o)), drop_mask=drop, keep_prob=ref.dropout_threshold(0.75) / 256.0,
                       causal=causal, scale=scale)
    for a, b in zip(got, want):      # P, dS and the forward's O to 2^-11, sums of 200 terms of both signs: 1e-2 of the largest
        assert float(np.max(np.abs(a.cpu().numpy() - b))) <= 1e-2 * float(np.max(np.abs(b)))
