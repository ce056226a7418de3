"""Forward kernels whose scores run ahead of P V: head_dim up to 64 (two Q tiles, three S buffers taken in turn) and above 128
(one Q tile, two S buffers).  Which buffer a tile gets depends on how many tiles either Q tile has had: lengths and limits
that give the two Q tiles of a thread block different numbers of K/V tiles, against the oracle."""
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref as ref

pytestmark = pytest.mark.gpu


# one K/V tile; a second Q tile that is absent, or of one row; 1, 2, 3, 4 and 7 K/V tiles; causal (Q tile 1 has one more),
# bands (the Q tiles' ranges begin and end apart), valid lengths that cut or empty the ranges
@pytest.mark.parametrize("D", [64, 40, 160, 256])
@pytest.mark.parametrize("S_q,S_k,kw", [
    (1, 1, {}), (128, 129, {}), (129, 384, {}), (256, 500, {}), (300, 896, {}),
    (129, 129, {"causal": True}), (640, 640, {"causal": True}), (900, 900, {"causal": True}),
    (900, 900, {"prev_block_num": 0, "next_block_num": 0}), (1024, 1024, {"prev_block_num": 2, "next_block_num": 1}),
    (513, 700, {"prev_block_num": 1, "next_block_num": 65536}), (640, 640, {"lens": [1, 130, 640]}),
    (300, 600, {"lens": [600, 0, 257]}),
])
def test_against_the_oracle(D, S_q, S_k, kw):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    kw = dict(kw)
    lens = kw.pop("lens", None)
    B, N = (3 if lens else 1), 2
    g = torch.Generator().manual_seed(S_q + S_k + D)
    # growing keys: the running maximum, and with it O, is rescaled again and again
    q = torch.randn(B, N, S_q, D, generator=g).half()
    k = (torch.randn(B, N, S_k, D, generator=g) * torch.linspace(0.2, 4.0, S_k)[:, None]).half()
    v = torch.randn(B, N, S_k, D, generator=g).half()
    scale = 1.0 / math.sqrt(D)
    sl = torch.tensor(lens, dtype=torch.int32).cuda() if lens else None
    o, lse = ops.fa_forward(q.cuda(), k.cuda(), v.cuda(), scale=scale, seq_lens=sl, **kw)
    torch.cuda.synchronize()
    _lib.device_status()
    o, lse = o.float().cpu().numpy(), lse.cpu().numpy()
    for b in range(B):
        n = lens[b] if lens else S_k
        if n == 0:
            assert not o[b].any()
            continue
        want, l_want = ref.sa_fwd(q[b:b + 1].numpy(), k[b:b + 1, :, :n].numpy(), v[b:b + 1, :, :n].numpy(), scale=scale, **kw)
        seen = np.isfinite(l_want[0])               # (a row whose band lies past the last key sees nothing)
        # P rounded to 16 bits (2^-11 of the largest |v|, about 4) and O rounded to 16 bits (2^-11 of up to 4)
        assert float(np.max(np.abs(np.where(seen[..., None], o[b] - want[0], 0.0)))) <= 4e-3
        assert float(np.max(np.abs(np.where(seen, lse[b] - l_want[0], 0.0)))) <= 4e-3


def _check(D, S_q, S_k, lse_too=True, tri=None, **kw):
    """One call against the oracle; `kw` in the oracle's names, scale 1/8."""
    from acctransformer_b200 import _lib, ops
    g = torch.Generator().manual_seed(S_q + S_k + D)
    q, k, v = (torch.randn(1, 2, S, D, generator=g).half() for S in (S_q, S_k, S_k))
    k *= 8.0 / math.sqrt(D)
    gpu = {}
    if "attn_mask" in kw:
        gpu["attn_mask"] = torch.tensor(kw["attn_mask"]).half().cuda()
    if "alibi" in kw:
        gpu["alibi"] = torch.tensor(kw["alibi"]).half().cuda()
    if "philox" in kw:
        gpu.update(keep_prob=0.75, dropout_seed=9, dropout_offset=2)
        kw["drop_mask"] = ops.dropout_mask(1, 2, S_q, S_k, 0.75, 9, 2).cpu().numpy()
        kw["keep_prob"] = ref.dropout_threshold(kw.pop("philox")) / 256.0
    elif "drop_mask" in kw:
        gpu.update(keep_prob=kw["keep_prob"], dropout_mask=torch.tensor(kw["drop_mask"]).cuda())
    o, lse = ops.fa_forward(q.cuda(), k.cuda(), v.cuda(), scale=0.125, tri_block=tri or 0, causal=kw.get("causal", False), **gpu)
    torch.cuda.synchronize()
    _lib.device_status()
    if tri:
        want = ref.triangle_fwd(q.numpy() * np.float16(0.125), k.numpy(), v.numpy(), np.zeros((1, S_q, S_k), np.float32), tri)
    else:
        want, l_want = ref.sa_fwd(q.numpy(), k.numpy(), v.numpy(), scale=0.125, **kw)
        if lse_too:
            assert float(np.max(np.abs(lse.cpu().numpy() - l_want))) <= 4e-3
    # P rounded to 16 bits (2^-11 of the largest |v|, about 4, over keep_prob) and O rounded to 16 bits
    assert float(np.max(np.abs(o.float().cpu().numpy() - want))) <= 4e-3 / kw.get("keep_prob", 1.0)


# the same kernels with row groups that end inside a tile, on its edge and past the last row, and with dropout decided in the
# kernel, by a uint8 tensor with aligned rows and by one without (each an instantiation of its own)
@pytest.mark.parametrize("D", [64, 40, 160, 256])
@pytest.mark.parametrize("what", ["groups 96", "groups 256", "groups 1000", "philox", "philox causal", "uint8", "uint8 unaligned"])
def test_row_groups_and_dropout_against_the_oracle(D, what):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if what.startswith("groups"):
        _check(D, 640, 640, tri=int(what.split()[1]))
        return
    S_k = 500 if "unaligned" in what else 640
    kw = {"causal": True} if "causal" in what else {}
    if what.startswith("philox"):
        kw["philox"] = 0.75
    else:
        keep = np.random.RandomState(D).random_sample((1, 2, 640, S_k)) < 0.75
        kw.update(drop_mask=keep.astype(np.uint8), keep_prob=0.75)
    _check(D, 640, S_k, **kw)


# masks and alibi above head_dim 128: one Q tile, two S buffers, the general path of the softmax stage
@pytest.mark.parametrize("D", [160, 256])
@pytest.mark.parametrize("what", ["mask", "alibi", "both"])
def test_mask_and_alibi_of_wide_heads_against_the_oracle(D, what):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rs = np.random.RandomState(D)
    kw = {}
    if what != "alibi":
        kw["attn_mask"] = (rs.random_sample((1, 400, 500)) < 0.4).astype(np.float32)
    if what != "mask":
        kw["alibi"] = np.float32(np.float16(-0.05 * np.arange(500))).reshape(1, 1, 1, 500).repeat(2, axis=1)
    _check(D, 400, 500, **kw)
