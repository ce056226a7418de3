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
# bands (the Q tiles' ranges begin and end apart), row groups, valid lengths that cut or empty the ranges
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
