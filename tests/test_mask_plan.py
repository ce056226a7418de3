"""What a mask tensor leaves out is not computed (acct_mask_plan); results are those of computing every tile.

The cells make the plan; ops.fa_forward / fa_backward compute every tile.  What is left out would have added exact zeros;
in mixed tiles the scores of unmasked keys skip one rounding on their way to the exponential.
"""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref as ref

pytestmark = pytest.mark.gpu


def _documents(S, cuts, B=1):
    pos = torch.arange(S)
    rows = []
    for b in range(B):
        doc = torch.bucketize(pos, torch.tensor(cuts[b % len(cuts)]), right=True)
        rows.append((doc[:, None] != doc[None, :]) | (pos[None, :] > pos[:, None]))
    return torch.stack(rows).float()


def _case(name):
    B, N, N_kv, S, D, dt = 2, 32, 8, 1500, 64, torch.float16
    mask = _documents(S, [[400, 900, 1400]])
    if name == "documents per sequence":
        D, dt = 128, torch.bfloat16
        mask = _documents(S, [[128, 256, 1024], [1, 700]], B)
    elif name == "padding":
        mask = torch.zeros(B, S, S)
        mask[0, :, 300:], mask[1, :, 1281:] = 1.0, 1.0
    elif name == "a row that sees nothing":          # its Q tile must be computed whole
        mask[0, 1000, :] = 1.0
    elif name == "block sparse":                     # a Q tile that only sees a far tile; key tiles that nobody sees
        mask = torch.ones(1, S, S)
        mask[0, :, 1280:1400] = 0.0
        mask[0, 256:384, :128] = 0.0
    elif name == "values that are no mask":          # tiles with them are read
        mask[0, 130, 5], mask[0, 700, 650] = 0.5, 0.25
    elif name == "wide heads":
        N, N_kv, S, D = 64, 64, 1030, 160
        mask = _documents(S, [[300, 600]])
    return B, N, N_kv, S, D, dt, mask


def _run(B, N, N_kv, S, D, dt, mask, change=None):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import FlashAttention, _lib, ops
    g = torch.Generator().manual_seed(S + D)
    q, d_o = (torch.randn(B, N, S, D, generator=g) for _ in range(2))
    k, v = (torch.randn(B, N_kv, S, D, generator=g) for _ in range(2))
    if change is not None:
        change(q, k, v, d_o)
    q, k, v, d_o, m = (t.to(dt).cuda() for t in (q, k, v, d_o, mask))
    scale = 1.0 / math.sqrt(D)
    tiles = ops.mask_tile_classes(m)
    a, keep = ops._fill_fa_args(q, k, v, q, None, m, False, False, None, 1.0, None, None, 65536, 65536, scale, None,
                                mask_tiles=tiles)
    _lib.load().acct_mask_plan_bytes.restype = C.c_size_t
    assert _lib.load().acct_mask_plan_bytes(C.byref(a)) > 0      # the cell's call takes the planned route
    o0, lse0 = ops.fa_forward(q, k, v, m, scale=scale, mask_tiles=tiles)
    g0 = ops.fa_backward(q, k, v, o0, lse0, d_o, m, scale=scale, mask_tiles=tiles)
    layer = FlashAttention(D)
    layer.allow_grouped_kv = True
    qq, kk, vv = (t.clone().requires_grad_() for t in (q, k, v))
    o1 = layer(qq, kk, vv, m)
    g1 = torch.autograd.grad(o1, (qq, kk, vv), d_o)
    torch.cuda.synchronize()
    _lib.device_status()
    # a probability or dS that rounds to its other 16-bit neighbour moves a result by one unit (2^-11 / 2^-8) of a term,
    # and the terms are of the size of the largest result at most; then the result's own rounding
    unit = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    for a_, b_ in ((o1, o0), *zip(g1, g0)):
        assert torch.equal(torch.isnan(a_), torch.isnan(b_)) and torch.equal(torch.isinf(a_), torch.isinf(b_))
        a_, b_ = (torch.nan_to_num(t.detach().float(), 0.0, 0.0, 0.0) for t in (a_, b_))
        assert (a_ - b_).abs().max().item() <= 2 * unit * b_.abs().max().item()
    return q, k, v, d_o, o1, g1


@pytest.mark.parametrize("name", ["documents", "documents per sequence", "padding", "a row that sees nothing", "block sparse",
                                  "values that are no mask", "wide heads"])
def test_same_results_as_every_tile(name):
    B, N, N_kv, S, D, dt, mask = _case(name)
    q, k, v, d_o, o, grads = _run(B, N, N_kv, S, D, dt, mask)
    m = mask.numpy() if mask.shape[0] == 1 else mask[1:2].numpy()
    one = [t[1:2, :1].float().cpu().numpy() for t in (q, k, v)]      # one slice against the oracle
    o_ref, _ = ref.sa_fwd(*one, attn_mask=m, scale=1.0 / math.sqrt(D))
    assert float(np.max(np.abs(o[1:2, :1].detach().float().cpu().numpy() - o_ref))) <= (2e-3 if dt == torch.float16 else 2e-2)


# operands for which a tile that is all 1 does count: they must not be left out
@pytest.mark.parametrize("what", ["scores beyond the mask's -10000", "NaN key", "infinite value", "infinite output gradient"])
def test_operands_that_reach_past_the_mask(what):
    def change(q, k, v, d_o):
        if what.startswith("scores"):
            q.mul_(300.0), k.mul_(300.0)
        elif what == "NaN key":
            k[1, 3, 1450, 5] = float("nan")
        elif what == "infinite value":
            v[0, 2, 10, 0] = float("inf")
        else:
            d_o[1, 5, 1499, 7] = float("-inf")
    _run(*_case("documents"), change)


# what a call keeps for its backward besides the tensors that it has to: at most a sixteenth of those, nothing where the
# backward uses no plan (deterministic, wide heads); (8 heads, 4 096 tokens): drawn up again, (64, 2 048): kept
@pytest.mark.parametrize("N,S,D,deterministic", [(8, 4096, 64, False), (64, 2048, 64, False), (64, 2048, 64, True),
                                                 (64, 2048, 160, False)])
def test_memory_held_until_the_backward(N, S, D, deterministic):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    from acctransformer_b200.flash_attention.ops.flash_attention.flash_attention_impl import get_flash_attention
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, d_o = (torch.randn(1, N, S, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(4))
    mask = _documents(S, [[500, 1100]]).half().cuda()
    tiles = ops.mask_tile_classes(mask)
    fa = get_flash_attention(scale=1.0 / math.sqrt(D), deterministic=deterministic)
    xs = [t.requires_grad_() for t in (q, k, v)]
    before = torch.cuda.memory_allocated()
    o, lse = fa(*xs, mask)
    held = torch.cuda.memory_allocated() - before - o.numel() * 2 - lse.numel() * 4
    kept = N == 64 and D == 64 and not deterministic
    assert held <= (4 * q.numel() * 2 // 16 if kept else 4096)
    for retain in (True, False):     # the second backward finds what the first did
        got = torch.autograd.grad(o, xs, d_o, retain_graph=retain)
        with torch.no_grad():
            want = ops.fa_backward(q, k, v, o, lse, d_o, mask, scale=1.0 / math.sqrt(D), mask_tiles=tiles, deterministic=deterministic)
        for a, b in zip(got, want):      # one unit of a 16-bit P or dS, then the result's own rounding
            assert (a.float() - b.float()).abs().max().item() <= 2 * 2.0 ** -11 * b.float().abs().max().item()
    del got, want, a, b
    assert torch.cuda.memory_allocated() - before - o.numel() * 2 - lse.numel() * 4 <= 4096      # given back, although the output still lives
    torch.cuda.synchronize()
    _lib.device_status()


# what else goes with a plan: in-kernel dropout, masks of other types, of two dimensions, that are views, that are not square
@pytest.mark.parametrize("form", ["dropout", "uint8", "bool, two dimensions", "view", "fewer queries than keys"])
def test_with_a_plan_as_without(form):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    from acctransformer_b200.flash_attention.ops.flash_attention.flash_attention_impl import get_flash_attention
    N, S_q, S_k, D = 64, 1500, 1500, 64
    if form == "fewer queries than keys":
        S_q, S_k = 1100, 1800
    g = torch.Generator(device="cuda").manual_seed(S_k)
    q, d_o = (torch.randn(1, N, S_q, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(2))
    k, v = (torch.randn(1, N, S_k, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(2))
    mask = _documents(S_k, [[400, 900, 1400]])[:, :S_q].half().cuda()
    given = mask
    if form == "uint8":
        given = mask.to(torch.uint8)
    elif form.startswith("bool"):
        given = mask[0].bool()
    elif form == "view":
        given = torch.nn.functional.pad(mask, (3, 5, 2, 1))[:, 2:-1, 3:-5]
        assert not given.is_contiguous()
    kw = dict(keep_prob=0.75, dropout_seed=11, dropout_offset=5) if form == "dropout" else {}
    scale = 1.0 / math.sqrt(D)
    xs = [t.clone().requires_grad_() for t in (q, k, v)]
    o1, lse1 = get_flash_attention(scale=scale)(*xs, given, **kw)
    g1 = torch.autograd.grad(o1, xs, d_o)
    o0, lse0 = ops.fa_forward(q, k, v, mask, scale=scale, **kw)
    g0 = ops.fa_backward(q, k, v, o0, lse0, d_o, mask, scale=scale, **kw)
    torch.cuda.synchronize()
    _lib.device_status()
    for a, b in ((o1, o0), *zip(g1, g0)):      # the bound of _run
        assert (a.float() - b.float()).abs().max().item() <= 2 * 2.0 ** -11 * b.float().abs().max().item()
    # and one slice against the oracle
    h = 5
    drop, keep = None, 1.0
    if kw:
        drop = ops.dropout_mask(1, N, S_q, S_k, 0.75, 11, 5)[:, h:h + 1].cpu().numpy()
        keep = ref.dropout_threshold(0.75) / 256.0
    ins = [t[:, h:h + 1].float().cpu().numpy() for t in (q, k, v, d_o)]
    m = mask.float().cpu().numpy()
    o_ref, _ = ref.sa_fwd(*ins[:3], attn_mask=m, drop_mask=drop, keep_prob=keep, scale=scale)
    assert float(np.max(np.abs(o1[:, h:h + 1].detach().float().cpu().numpy() - o_ref))) <= 4e-3     # P and O to 2^-11 of up to 4 / keep
    for a, b in zip(g1, ref.sa_grad(*ins, attn_mask=m, drop_mask=drop, keep_prob=keep, scale=scale)):
        # dS and P to 2^-11 per term, sums of up to 1 500 terms of both signs, the result to 2^-11: 1e-2 of the largest
        assert float(np.max(np.abs(a[:, h:h + 1].float().cpu().numpy() - b))) <= 1e-2 * float(np.max(np.abs(b)))
