"""The C entry points behind the cells, as a caller without the Python layers uses them: an output gradient in a layout of its
own, and a mask plan made, used and drawn up again from its norms."""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(B, N, S, D, mask=None, tiles=None):
    """(library, args, io, tensors) of a backward whose forward has run."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from acctransformer_b200 import _lib, ops
    lib = _lib.load()
    lib.acct_mask_plan_bytes.restype = C.c_size_t
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v, d_o = (torch.randn(B, N, S, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(4))
    o, lse = ops.fa_forward(q, k, v, mask, scale=1.0 / math.sqrt(D), mask_tiles=tiles)
    a, keep = ops._fill_fa_args(q, k, v, o, lse, mask, False, False, None, 1.0, None, None, 65536, 65536, 1.0 / math.sqrt(D), None,
                                mask_tiles=tiles)
    grads = [torch.empty_like(t) for t in (q, k, v)]
    ws = torch.empty(lib.acct_fa_bwd_workspace_bytes(C.byref(a)), dtype=torch.uint8, device="cuda")
    io = _lib.FaBwdIO()
    io.dq, io.dk, io.dv = (t.data_ptr() for t in grads)
    io.workspace, io.workspace_bytes = ws.data_ptr(), ws.numel()
    return lib, a, io, (q, k, v, o, lse, d_o, grads, ws, keep)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("D", [64, 160])
@pytest.mark.parametrize("form", ["null", "zeros", "transposed", "padded"])
def test_output_gradient_with_strides(D, form):
    from acctransformer_b200 import _lib, ops
    lib, a, io, (q, k, v, o, lse, d_o, grads, *_rest) = _call(2, 3, 130, D)
    want = ops.fa_backward(q, k, v, o, lse, d_o, scale=1.0 / math.sqrt(D))
    given = d_o
    if form == "transposed":
        given = d_o.transpose(1, 2).contiguous().transpose(1, 2)
    elif form == "padded":
        given = torch.cat([d_o, d_o], -1)[..., :D]
    strides = {"null": None, "zeros": (C.c_int64 * 3)(0, 0, 0)}.get(form, (C.c_int64 * 3)(*given.stride()[:3]))
    io.d_o = given.data_ptr()
    _lib.check(lib.acct_fa_bwd_strided(C.byref(a), C.byref(io), strides, _stream()))
    torch.cuda.synchronize()
    _lib.device_status()
    for x, y in zip(grads, want):       # (dq: two K/V tiles, a sum of two has no order)
        assert torch.equal(x, y)
    bad = (C.c_int64 * 3)(given.stride(0), given.stride(1), given.stride(2) + 4)
    assert lib.acct_fa_bwd_strided(C.byref(a), C.byref(io), bad, _stream()) != 0       # refused: rows off the 16-byte grid


def test_plan_made_used_and_drawn_up_again():
    from acctransformer_b200 import _lib, ops
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    S, D = 1500, 64
    pos = torch.arange(S, device="cuda")
    mask = ((pos[:, None] // 400 != pos[None, :] // 400) | (pos[None, :] > pos[:, None])).half()[None]
    tiles = ops.mask_tile_classes(mask)
    lib, a, io, (q, k, v, o, lse, d_o, grads, *_rest) = _call(1, 64, S, D, mask, tiles)
    n = lib.acct_mask_plan_bytes(C.byref(a))
    assert n > 0
    scratch, norms = (torch.empty(16, dtype=torch.uint8, device="cuda") for _ in range(2))
    io.d_o = d_o.data_ptr()

    def bwd(plan):
        _lib.check(lib.acct_fa_bwd_planned(C.byref(a), C.byref(io), None, C.c_void_p(plan.data_ptr()), C.c_void_p(scratch.data_ptr()),
                                           _stream()))
        return [t.clone() for t in grads[1:]]
    first, second, third = (torch.empty(n, dtype=torch.uint8, device="cuda") for _ in range(3))
    _lib.check(lib.acct_mask_plan(C.byref(a), C.c_void_p(first.data_ptr()), _stream()))
    _lib.check(lib.acct_fa_fwd_planned(C.byref(a), C.c_void_p(first.data_ptr()), _stream()))
    want = bwd(first)
    for plan, known in ((second, 0), (third, 1)):
        _lib.check(lib.acct_mask_plan_norms(C.byref(a), C.c_void_p(plan.data_ptr()), C.c_void_p(norms.data_ptr()), known, _stream()))
        assert torch.equal(plan[:16], first[:16]) and torch.equal(norms[:12], first[:12])
        for x, y in zip(bwd(plan), want):
            assert torch.equal(x, y)
    torch.cuda.synchronize()
    _lib.device_status()
    q2 = q.float().square().sum(-1).max().item()
    assert abs(norms.view(torch.float32)[0].item() / q2 - 1) < 1e-5
    assert lib.acct_mask_plan_norms(C.byref(a), C.c_void_p(third.data_ptr()), None, 1, _stream()) != 0     # known, but not given
