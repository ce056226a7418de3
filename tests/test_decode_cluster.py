"""Decoding over few and short contexts, where the parts of a slice form one thread-block cluster that merges them."""
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref as ref

pytestmark = pytest.mark.gpu


# one part (<= 128 keys), two (129 keys: the second part is all but empty), eight, and more slices than leave room for
# eight parts; head groups on CUDA cores, on MMA rows 0-7 and 0-15; sequences of one key, so that most parts are empty
@pytest.mark.parametrize("B,n_kv,group,S,D,dtype", [
    (1, 1, 1, 1, 64, "float16"), (2, 3, 1, 128, 128, "bfloat16"), (2, 2, 1, 129, 40, "float16"),
    (1, 2, 1, 1100, 256, "float16"), (3, 2, 4, 4096, 128, "bfloat16"), (2, 1, 16, 700, 64, "float16"),
    (4, 16, 4, 1000, 128, "float16"), (8, 32, 1, 515, 80, "bfloat16"), (2, 2, 8, 257, 160, "float16"),
])
def test_clustered_parts_against_the_oracle(B, n_kv, group, S, D, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    dt = getattr(torch, dtype)
    g = torch.Generator().manual_seed(S + D)
    q = torch.randn(B, n_kv * group, 1, D, generator=g).to(dt)
    k, v = (torch.randn(B, n_kv, S, D, generator=g).to(dt) for _ in range(2))
    lens = torch.randint(1, S + 1, (B,), generator=g, dtype=torch.int32)
    lens[0], lens[-1] = 1, S
    scale = 1.0 / math.sqrt(D)
    y = ops.infer_decode(q.cuda(), k.cuda(), v.cuda(), lens.cuda(), scale=scale)
    torch.cuda.synchronize()
    _lib.device_status()
    want = ref.decode_ref(q.float().numpy(), k.float().numpy().repeat(group, axis=1), v.float().numpy().repeat(group, axis=1),
                          lens.numpy(), scale)
    # results up to about 4 in size, rounded to 16 bits (half a unit: 2^-10 fp16, 2^-7 bf16); with head groups the
    # probabilities are rounded to 16 bits too (at most 2^-11 / 2^-8 of the largest |v|, about 4)
    tol = 4e-3 if dtype == "float16" else 3e-2
    assert float(np.max(np.abs(y.float().cpu().numpy() - want))) <= tol


# around the lines of the rule: more slices than clusters of 8 (4, 2) parts fit at once, parts of 512 keys and one more (1 024
# where a block carries a group), a workspace that holds fewer parts
@pytest.mark.parametrize("B,n_kv,group,S,fit", [
    (70, 1, 1, 600, 64), (71, 1, 1, 2048, 64), (72, 1, 1, 2049, 64), (142, 1, 1, 600, 64), (149, 1, 1, 1024, 64),
    (149, 1, 1, 1025, 64), (297, 1, 1, 256, 64), (33, 1, 4, 1024, 64), (35, 1, 4, 4096, 64), (72, 1, 4, 2048, 64),
    (74, 1, 4, 2049, 64), (149, 1, 4, 300, 64), (2, 2, 1, 1000, 3), (2, 2, 4, 1000, 1),
])
def test_around_the_lines_of_the_rule(B, n_kv, group, S, fit):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    D = 64
    g = torch.Generator(device="cuda").manual_seed(S + B)
    q = torch.randn(B, n_kv * group, 1, D, device="cuda", generator=g).half()
    k, v = (torch.randn(B, n_kv, S, D, device="cuda", generator=g).half() for _ in range(2))
    lens = torch.randint(1, S + 1, (B,), generator=torch.Generator().manual_seed(S), dtype=torch.int32).cuda()
    ws = ops.DecodeWorkspace(B, n_kv * group, D, "cuda", fit)
    y = ops.infer_decode(q, k, v, lens, workspace=ws)
    one = ops.infer_decode(q, k, v, lens, num_splits=1)          # the whole slice in one part
    torch.cuda.synchronize()
    _lib.device_status()
    # one rounding of a result of up to 4, and with groups probabilities rounded against another running maximum
    assert (y.float() - one.float()).abs().max().item() <= 4e-3


# the second kernel, which merges the parts where they are no cluster: batches of 16 parts, two halves of 32; empty parts
@pytest.mark.parametrize("splits", [1, 2, 15, 16, 17, 32, 33, 49, 64])
@pytest.mark.parametrize("group,D,dtype", [(1, 40, "float16"), (4, 128, "bfloat16"), (1, 256, "float16")])
def test_merge_of_any_number_of_parts(splits, group, D, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    dt = getattr(torch, dtype)
    B, n_kv, S = 3, 2, 4200
    g = torch.Generator().manual_seed(splits + D)
    q = torch.randn(B, n_kv * group, 1, D, generator=g).to(dt)
    k, v = (torch.randn(B, n_kv, S, D, generator=g).to(dt) for _ in range(2))
    lens = torch.tensor([1, 2000, S], dtype=torch.int32)
    scale = 1.0 / math.sqrt(D)
    y = ops.infer_decode(q.cuda(), k.cuda(), v.cuda(), lens.cuda(), scale=scale, num_splits=splits)
    torch.cuda.synchronize()
    _lib.device_status()
    want = ref.decode_ref(q.float().numpy(), k.float().numpy().repeat(group, axis=1), v.float().numpy().repeat(group, axis=1),
                          lens.numpy(), scale)
    tol = 4e-3 if dtype == "float16" else 3e-2      # as above
    assert float(np.max(np.abs(y.float().cpu().numpy() - want))) <= tol
