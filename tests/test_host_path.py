"""The native host path of the cells takes and refuses what a Python autograd Function around the operator does."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B, N, S, D, seed=0):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(B, N, S, D, device="cuda", dtype=torch.float16, generator=g) for _ in range(4)]


def _layer(D, **kw):
    from acctransformer_b200 import FlashAttention
    return FlashAttention(D, **kw)


# an output gradient whose head dimension has size 1 and a stride that means nothing (1), one whose rows are not
# 16-byte aligned, one expanded from a scalar
@pytest.mark.parametrize("form", ["size-one stride", "misaligned", "expanded"])
def test_output_gradient_in_any_layout(form):
    q, k, v, d_o = _inputs(2, 1, 130, 64)
    if form == "size-one stride":
        odd = d_o.view(2, 130, 64).clone().unsqueeze(3).permute(0, 3, 1, 2)
        assert odd.stride(1) == 1
    elif form == "misaligned":
        odd = d_o.new_empty(2, 1, 130, 65)[..., 1:]
        odd.copy_(d_o)
    else:
        d_o = torch.full_like(d_o, 0.5)
        odd = torch.full((), 0.5, device="cuda", dtype=d_o.dtype).expand(2, 1, 130, 64)
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    out = _layer(64)(q, k, v)
    want = torch.autograd.grad(out, (q, k, v), d_o, retain_graph=True)
    got = torch.autograd.grad(out, (q, k, v), odd)
    # dk and dv are reproducible; dq is summed over two K/V tiles, and a sum of two does not depend on the order
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_optional_input_that_requires_a_gradient_is_part_of_the_graph():
    q, k, v, d_o = _inputs(1, 2, 128, 64)
    alibi = torch.zeros(1, 2, 1, 128, device="cuda", dtype=torch.float16, requires_grad=True)
    out = _layer(64, alibi=True)(q, k, v, None, alibi)
    assert out.requires_grad
    out.backward(d_o)
    assert alibi.grad is None


def test_forward_mode_is_refused():
    import torch.autograd.forward_ad as fwad
    q, k, v, t = _inputs(1, 2, 128, 64)
    with fwad.dual_level():
        with pytest.raises(NotImplementedError):
            _layer(64)(fwad.make_dual(q, t), k, v)


def _documents(S, dtype=torch.float16):
    """Two documents, causal inside each: [1, S, S], 1 where a key must not be seen."""
    pos = torch.arange(S, device="cuda")
    doc = pos >= S // 3
    return ((doc[:, None] != doc[None, :]) | (pos[None, :] > pos[:, None])).to(dtype)[None]


def _grads(layer, qkv, d_o, *rest):
    xs = [t.detach().requires_grad_() for t in qkv]
    return torch.autograd.grad(layer(*xs, *rest), xs, d_o)


def test_mask_first_seen_under_inference_mode_can_be_trained_with():
    q, k, v, d_o = _inputs(1, 2, 200, 64)
    mask = _documents(200)
    with torch.inference_mode():
        _layer(64)(q, k, v, mask)
    got = _grads(_layer(64), (q, k, v), d_o, mask)
    want = _grads(_layer(64), (q, k, v), d_o, mask.clone())
    # (dq is a sum over two K/V tiles: no order to depend on)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


# operands that a kernel would read or write out of range, or not at all from where they are: errors on the host, no launch
@pytest.mark.parametrize("what", ["lengths on the host", "too few lengths", "key dtype", "out dtype", "out too small",
                                  "strided out", "workspace on the host", "table on the host"])
def test_decode_refuses_what_the_kernels_cannot_reach(what):
    from acctransformer_b200 import ops
    q, _, _, _ = _inputs(2, 4, 1, 64)
    k, v, _, _ = _inputs(2, 4, 64, 64)
    kw = {"seq_lens": torch.tensor([3, 64], dtype=torch.int32, device="cuda")}
    if what == "lengths on the host":
        kw["seq_lens"] = kw["seq_lens"].cpu()
    elif what == "too few lengths":
        kw["seq_lens"] = kw["seq_lens"][:1]
    elif what == "key dtype":
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
    elif what == "out dtype":
        kw["out"] = torch.empty_like(q, dtype=torch.uint8)
    elif what == "out too small":
        kw["out"] = torch.empty_like(q[:1])
    elif what == "strided out":
        kw["out"] = torch.empty(2, 4, 1, 128, device="cuda", dtype=q.dtype)[..., :64]
    elif what == "workspace on the host":
        kw["workspace"] = ops.DecodeWorkspace(2, 4, 64, "cpu")
    else:
        kw["block_table"] = torch.zeros(2, 1, dtype=torch.int32)
    with pytest.raises(ValueError):
        ops.infer_decode(q, k, v, **kw)


def test_decode_takes_lengths_and_out_in_any_shape():
    from acctransformer_b200 import ops
    q, _, _, _ = _inputs(2, 4, 1, 64)
    k, v, _, _ = _inputs(2, 4, 64, 64)
    want = ops.infer_decode(q, k, v, torch.tensor([3, 64], dtype=torch.int32, device="cuda"))
    out = torch.empty(2, 4, 64, device="cuda", dtype=q.dtype)
    got = ops.infer_decode(q, k, v, torch.tensor([[3], [64], [5]], device="cuda"), out=out)
    assert got is out or got.data_ptr() == out.data_ptr()
    assert torch.equal(out.view_as(want), want)


@pytest.mark.parametrize("what", ["lengths on the host", "too few lengths", "key dtype", "value on the host"])
def test_prefill_refuses_what_the_kernels_cannot_reach(what):
    from acctransformer_b200 import ops
    q, k, v, _ = _inputs(2, 2, 130, 64)
    lens = torch.tensor([130, 7], dtype=torch.int32, device="cuda")
    if what == "lengths on the host":
        lens = lens.cpu()
    elif what == "too few lengths":
        lens = lens[:1]
    elif what == "key dtype":
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
    else:
        v = v.cpu()
    with pytest.raises(ValueError):
        ops.infer_prefill(q, k, v, seq_lens=lens)


@pytest.mark.parametrize("what", ["key", "mask", "alibi", "dropout mask"])
def test_training_refuses_what_the_kernels_cannot_reach(what):
    from acctransformer_b200.flash_attention.ops.flash_attention.flash_attention_impl import get_flash_attention
    q, k, v, _ = _inputs(1, 2, 130, 64)
    kw = {}
    if what == "key":
        k = k.cpu()
    elif what == "mask":
        kw["attn_mask"] = torch.zeros(1, 130, 130, dtype=q.dtype)
    elif what == "alibi":
        kw["alibi_mask"] = torch.zeros(1, 2, 1, 130, dtype=q.dtype)
    else:
        kw["dropout_mask"] = torch.ones(1, 2, 130, 130, dtype=torch.uint8)
    with pytest.raises(ValueError):
        get_flash_attention()(q, k, v, **kw)


def test_numbers_in_any_form_that_int_and_float_take():
    from acctransformer_b200 import TriangleAttention
    from acctransformer_b200.flash_attention.ops.flash_attention.flash_attention_impl import get_flash_attention
    q, k, v, _ = _inputs(1, 2, 300, 64)
    assert torch.equal(_layer(64, prev_block_num=1.0, next_block_num=0.0)(q, k, v), _layer(64, prev_block_num=1, next_block_num=0)(q, k, v))
    assert torch.equal(_layer(64, prev_block_num=10 ** 30)(q, k, v), _layer(64)(q, k, v))
    with pytest.raises(Exception, match="prev/next_block_num must be >= 0"):
        _layer(64, prev_block_num=-1)(q, k, v)
    mask = _documents(300)
    assert torch.equal(TriangleAttention(block_size=128.0)(q, k, v, mask), TriangleAttention(block_size=128)(q, k, v, mask))
    fa = get_flash_attention(scale="0.125")
    want = get_flash_attention(scale=0.125)(q, k, v, keep_prob=0.75, dropout_seed=7, dropout_offset=2)[0]
    assert torch.equal(fa(q, k, v, keep_prob="0.75", dropout_seed=7.0, dropout_offset=torch.tensor(2.0))[0], want)
    assert torch.equal(fa(q, k, v, keep_prob=0.75, dropout_seed=7 + 2 ** 64, dropout_offset=2)[0], want)


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return None


def test_output_gradient_that_is_not_there_counts_as_zero():
    q, k, v, d_o = _inputs(1, 2, 130, 64)
    xs = [t.requires_grad_() for t in (q, k, v)]
    for g in torch.autograd.grad(_NoGradient.apply(_layer(64)(*xs)), xs, d_o):
        assert g.shape == q.shape and not g.any()


# saved-tensor hooks that hand back the same values in another layout: rows of 128 elements of which 64 count, every second
# element of a score-shaped tensor, an output that is aligned to nothing, and tensors that were on the host meanwhile
@pytest.mark.parametrize("form", ["padded rows", "every second element", "misaligned output", "offloaded"])
def test_saved_tensors_in_any_layout(form):
    q, k, v, d_o = _inputs(2, 2, 200, 64)
    mask = _documents(200)
    want = _grads(_layer(64), (q, k, v), d_o, mask)
    o_shape = q.shape

    def unpack_misaligned(t):
        if t.dim() != 4 or t.requires_grad or t.shape != o_shape:
            return t
        r = t.new_empty(t.shape[:3] + (t.shape[3] + 1,))[..., 1:]
        return r.copy_(t)
    pack, unpack = {
        "padded rows": (lambda t: torch.cat([t, torch.zeros_like(t)], -1) if t.dim() == 4 else t,
                        lambda t: t[..., :64] if t.dim() == 4 else t),
        "every second element": (lambda t: torch.stack([t, torch.zeros_like(t)], -1) if t.dim() == 3 else t,
                                 lambda t: t[..., 0] if t.shape[-1] == 2 else t),
        "misaligned output": (lambda t: t, unpack_misaligned),
        "offloaded": (lambda t: t.cpu(), lambda t: t.cuda()),
    }[form]
    xs = [t.detach().requires_grad_() for t in (q, k, v)]
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        out = _layer(64)(*xs, mask)
    for a, b in zip(torch.autograd.grad(out, xs, d_o), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("which", ["q", "o", "lse", "mask"])
def test_saved_tensors_left_on_the_host_are_refused(which):
    q, k, v, d_o = _inputs(1, 2, 130, 64)
    shape = {"q": (1, 2, 130, 64), "o": (1, 2, 130, 64), "lse": (1, 2, 130), "mask": (1, 130, 130)}[which]
    xs = [t.detach().requires_grad_() for t in (q, k, v)]
    mine = (lambda t: t.requires_grad and t.is_leaf) if which == "q" else (lambda t: not (t.requires_grad and t.is_leaf))
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (t.shape == shape and mine(t), t), lambda p: p[1].cpu() if p[0] else p[1]):
        out = _layer(64)(*xs, _documents(130))
    with pytest.raises((ValueError, RuntimeError), match="CUDA tensor|device"):
        torch.autograd.grad(out, xs, d_o)


# a mask that is a view is saved itself, not as the packed copy that the kernels read: it counts as memory of its owner,
# and a change between forward and backward is noticed
@pytest.mark.parametrize("packed", [True, False])
def test_mask_changed_before_the_backward_is_refused(packed):
    q, k, v, d_o = _inputs(1, 2, 200, 64)
    owner = _documents(256)
    mask = owner[:, :200, :200]
    if packed:
        mask = mask.contiguous()
    xs = [t.detach().requires_grad_() for t in (q, k, v)]
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t.data_ptr()) or t, lambda t: t):
        _layer(64)(*xs, mask)
    assert mask.data_ptr() in saved
    out = _layer(64)(*xs, mask)
    mask.zero_()
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, xs, d_o)


def test_backward_under_compiled_autograd():
    from torch._dynamo import compiled_autograd
    q, k, v, d_o = _inputs(1, 2, 200, 64)
    mask = _documents(200)
    xs = [t.requires_grad_() for t in (q, k, v)]
    layer = _layer(64, dropout_rate=0.25)
    for seed in (1, 2):      # the second backward is the same graph with another dropout key
        def forward():
            layer.generator = torch.Generator().manual_seed(seed)
            return layer(*xs, mask)
        want = torch.autograd.grad(forward(), xs, d_o)
        out = forward()
        with compiled_autograd._enable(lambda graph: graph):
            out.backward(d_o)
        for t, b in zip(xs, want):
            assert torch.equal(t.grad, b)
            t.grad = None


@pytest.mark.parametrize("masked", [False, True])
def test_traced_cell_runs_on_new_inputs(masked):
    layer = _layer(64)
    ins = _inputs(1, 2, 200, 64)[:3] + ([_documents(200)] if masked else [])
    traced = torch.jit.trace(lambda *x: layer(*x), tuple(ins), check_trace=False)
    q, k, v, d_o = _inputs(1, 2, 200, 64, seed=1)
    rest = [_documents(200).roll(7, dims=2)] if masked else []
    with torch.no_grad():
        assert torch.equal(traced(q, k, v, *rest), layer(q, k, v, *rest))
    for a, b in zip(_grads(traced, (q, k, v), d_o, *rest), _grads(layer, (q, k, v), d_o, *rest)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("reentrant", [False, True])
def test_checkpointed_cell(reentrant):
    from torch.utils.checkpoint import checkpoint
    q, k, v, d_o = _inputs(1, 2, 200, 64)
    mask, layer = _documents(200), _layer(64, dropout_rate=0.25)
    torch.manual_seed(3)
    want = _grads(layer, (q, k, v), d_o, mask)
    xs = [t.detach().requires_grad_() for t in (q, k, v)]
    torch.manual_seed(3)
    checkpoint(layer, *xs, mask, use_reentrant=reentrant).backward(d_o)
    for t, b in zip(xs, want):
        assert torch.equal(t.grad, b)


def test_threads_and_streams():
    """Four threads, each with a stream and inputs of its own, run the cell forward and backward at the same time."""
    import threading
    layer, mask = _layer(64), _documents(200)
    ins = [_inputs(1, 2, 200, 64, seed=s) for s in range(4)]
    want = [_grads(layer, x[:3], x[3], mask) for x in ins]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(20):
                got = _grads(layer, ins[i][:3], ins[i][3], mask)
                stream.synchronize()
                if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                    wrong.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
