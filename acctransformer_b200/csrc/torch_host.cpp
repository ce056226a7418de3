// The host path of the Python layers in native code: takes torch tensors, checks them, fills the C ABI's argument
// blocks and launches, without a Python frame, a ctypes structure or a context manager per call, and carries the
// custom function of the training operator.
//
// Built as the CPython module `_torch_host` next to libacct_b200.so, whose entry points it looks up at load time
// (`init`), so it adds no second copy of any kernel.  What bounds the small calls is this path: one forward + backward
// of B=2 N=8 S=256 D=64 took 204 us of which the GPU worked about 40; per call the interpreter spent 15 to 40 us in
// attribute look-ups, ctypes fields and torch.cuda.device.
//
// Error conditions and texts are those of the Python front end (ops.py); a non-zero status of the library becomes its
// AcctError.  The reference registers its operators with the framework in Python
// (train/acctransformer/flash_attention/ops/flash_attention/flash_attention_impl.py:96-154); its custom
// function stands for the `bprop` there.
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include "../../include/acct_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Library {
  decltype(&acct_fa_fwd_planned) fa_fwd;
  decltype(&acct_fa_bwd_planned) fa_bwd;
  decltype(&acct_mask_plan_bytes) mask_plan_bytes;
  decltype(&acct_mask_plan_norms) mask_plan;
  decltype(&acct_fa_bwd_workspace_bytes) fa_bwd_workspace_bytes;
  decltype(&acct_infer_prefill) infer_prefill;
  decltype(&acct_infer_decode) infer_decode;
} g_lib;

#define HOST_CHECK TORCH_CHECK_VALUE

// A non-zero status of the library, raised as the AcctError that _lib.check() builds from it (the message is the
// calling thread's).  Also used from the autograd engine's threads, which do not hold the GIL.
void check(int rc) {
  if (rc == 0) return;
  PyGILState_STATE gil = PyGILState_Ensure();
  PyObject* mod = PyImport_ImportModule("acctransformer_b200._lib");
  if (mod != nullptr) {
    PyObject* r = PyObject_CallMethod(mod, "check", "i", rc);
    Py_XDECREF(r);
    Py_DECREF(mod);
  }
  python_error err;
  err.persist();
  PyGILState_Release(gil);
  throw err;
}

int dtype_code(at::ScalarType t, const char* what) {
  switch (t) {
    case at::kHalf: return ACCT_F16;
    case at::kBFloat16: return ACCT_BF16;
    case at::kByte: case at::kBool: return ACCT_U8;
    default: HOST_CHECK(false, what, ": unsupported dtype ", t);
  }
  return -1;
}

void require_cuda(const char* name, const Tensor& t) {
  HOST_CHECK(t.defined() && t.is_cuda(), name, " must be a CUDA tensor (this library has no CPU path)");
}

// Every pointer that a kernel gets is checked here: a host address or one of another GPU would fault on the device.
void require_on(const char* name, const Tensor& t, const Tensor& q) {
  require_cuda(name, t);
  HOST_CHECK(t.device() == q.device(), name, " must be on the device of q, ", q.device(), ", not on ", t.device());
}

// valid lengths as the kernels read them: at least one int32 per sequence
Tensor lengths(const Tensor& lens, int64_t B, const Tensor& q) {
  require_on("seq_lens", lens, q);
  HOST_CHECK(lens.numel() >= B, "seq_lens must hold a length for each of ", B, " sequences, got ", lens.numel());
  return lens.to(at::kInt).contiguous();
}

void strides3(const Tensor& t, int64_t (&out)[3]) {
  HOST_CHECK(t.stride(-1) == 1, "head_dim must be contiguous");
  for (int i = 0; i < 3; ++i) out[i] = t.stride(i);
}

Tensor empty_like_shape(at::IntArrayRef size, at::ScalarType dtype, const Tensor& like) {
  return at::detail::empty_cuda(size, dtype, like.device(), std::nullopt);
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// What a call carries besides tensors.
struct FaConfig {
  int64_t mask_tile128 = 0, causal = 0, deterministic = 0, has_seed = 0;      // (flags; no padding, see pack())
  double keep_prob = 1.0, scale = 1.0;
  int64_t prev = ACCT_BAND_UNBOUNDED, next = ACCT_BAND_UNBOUNDED, tri_block = 0;
  uint64_t seed = 0, offset = 0;

  // in the form that a custom function may keep
  std::vector<int64_t> pack() const {
    std::vector<int64_t> out(sizeof(FaConfig) / 8);
    memcpy(out.data(), this, sizeof(FaConfig));
    return out;
  }
  static FaConfig unpack(const std::vector<int64_t>& from) {
    FaConfig c;
    memcpy(&c, from.data(), sizeof(FaConfig));
    return c;
  }
};
static_assert(std::is_trivially_copyable_v<FaConfig> && sizeof(FaConfig) == 11 * 8);

// Fills `a` from the tensors (check_fa_inputs has seen to their shapes, and to contiguity where the ABI wants it).
void fill_args(acct_fa_args& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse,
               const Tensor& mask, const Tensor& drop, const Tensor& alibi, const Tensor& tiles, const FaConfig& c) {
  memset(&a, 0, sizeof(a));
  const int64_t B = q.size(0), N = q.size(1), S_q = q.size(2), D = q.size(3), N_kv = k.size(1), S_k = k.size(2);
  a.dtype = q.scalar_type() == at::kBFloat16 ? ACCT_BF16 : ACCT_F16;
  a.B = B; a.N = N; a.S_q = S_q; a.S_k = S_k; a.D = D; a.N_kv = N_kv;
  a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr(); a.o = const_cast<void*>(o.const_data_ptr());
  a.lse = lse.defined() ? const_cast<float*>(static_cast<const float*>(lse.const_data_ptr())) : nullptr;
  strides3(q, a.q_stride); strides3(k, a.k_stride); strides3(v, a.v_stride); strides3(o, a.o_stride);
  a.mask_kind = ACCT_MASK_NONE;
  if (mask.defined()) {
    a.mask_dtype = dtype_code(mask.scalar_type(), "attn_mask");
    if (c.mask_tile128) {
      a.mask_kind = ACCT_MASK_TILE128;
      a.mask_batch = 1;
    } else {
      a.mask_kind = ACCT_MASK_FULL;
      a.mask_batch = mask.dim() == 2 ? 1 : mask.size(0);
    }
    a.attn_mask = mask.const_data_ptr();
  }
  if (tiles.defined()) a.mask_tiles = static_cast<const uint8_t*>(tiles.const_data_ptr());
  a.causal = c.causal ? 1 : 0;
  a.keep_prob = static_cast<float>(c.keep_prob);
  if (drop.defined()) {
    a.dropout_mask = drop.const_data_ptr();
    a.dropout_dtype = dtype_code(drop.scalar_type(), "dropout_mask");
  }
  if (alibi.defined()) a.alibi = alibi.const_data_ptr();
  a.prev_block_num = static_cast<int32_t>(c.prev);
  a.next_block_num = static_cast<int32_t>(c.next);
  a.scale = static_cast<float>(c.scale);
  if (c.has_seed) {
    a.flags |= ACCT_FLAG_DROPOUT_PHILOX;
    a.dropout_seed = c.seed;
    a.dropout_offset = c.offset;
  }
  a.tri_block = static_cast<int32_t>(c.tri_block);
}

void check_fa_inputs(const Tensor& q, const Tensor& k, const Tensor& v, Tensor& mask, Tensor& drop, Tensor& alibi,
                     const Tensor& tiles, const FaConfig& c) {
  const Tensor* qkv[3] = {&q, &k, &v};
  const char* names[3] = {"q", "k", "v"};
  for (int i = 0; i < 3; ++i) {
    require_on(names[i], *qkv[i], q);
    HOST_CHECK(qkv[i]->dim() == 4, names[i], " must be [B, N, S, D]");
  }
  const auto dt = q.scalar_type();
  HOST_CHECK((dt == at::kHalf || dt == at::kBFloat16) && k.scalar_type() == dt && v.scalar_type() == dt,
             "q, k, v must share dtype float16 or bfloat16");
  const int64_t B = q.size(0), N = q.size(1), S_q = q.size(2), D = q.size(3), N_kv = k.size(1), S_k = k.size(2);
  HOST_CHECK(k.size(0) == B && k.size(3) == D && v.sizes() == k.sizes() && N_kv >= 1 && N % N_kv == 0, "shape mismatch: q ",
             q.sizes(), ", k ", k.sizes(), ", v ", v.sizes(), " (k and v may have fewer heads than q if their head count divides q's)");
  if (mask.defined()) {
    require_on("attn_mask", mask, q);
    mask = mask.contiguous();
    if (c.mask_tile128) {
      HOST_CHECK(mask.numel() == 128 * 128, "the tile form of attn_mask must hold 128x128 elements");
    } else {
      HOST_CHECK((mask.dim() == 2 || (mask.dim() == 3 && (mask.size(0) == 1 || mask.size(0) == B))) && mask.size(-2) == S_q &&
                     mask.size(-1) == S_k,
                 "attn_mask must be [1 or B, S_q, S_k], got ", mask.sizes());
    }
  }
  if (tiles.defined()) {
    HOST_CHECK(mask.defined() && !c.mask_tile128, "mask_tiles goes with a full attn_mask tensor");
    require_on("mask_tiles", tiles, q);
    const int64_t mb = mask.dim() == 2 ? 1 : mask.size(0);
    HOST_CHECK(tiles.scalar_type() == at::kByte && tiles.is_contiguous() && tiles.dim() == 3 && tiles.size(0) == mb &&
                   tiles.size(1) == (S_q + 127) / 128 && tiles.size(2) == (S_k + 127) / 128,
               "mask_tiles must be a contiguous uint8 tensor as mask_tile_classes() returns it");
  }
  if (drop.defined()) {
    require_on("dropout_mask", drop, q);
    HOST_CHECK(drop.dim() == 4 && drop.size(0) == B && drop.size(1) == N && drop.size(2) == S_q && drop.size(3) == S_k,
               "dropout_mask must be [B, N, S_q, S_k]");
    HOST_CHECK(!c.has_seed, "give either dropout_mask (tensor form) or dropout_seed (in-kernel form), not both");
    drop = drop.contiguous();
  }
  if (alibi.defined()) {
    require_on("alibi", alibi, q);
    HOST_CHECK(alibi.dim() == 4 && alibi.size(0) == B && alibi.size(1) == N && alibi.size(2) == 1 && alibi.size(3) == S_k &&
                   alibi.scalar_type() == dt,
               "alibi must be [B, N, 1, S_k] in the dtype of q");
    alibi = alibi.contiguous();
  }
}

// A [B, N, S, D] operand that the kernels read in its own layout where they can (head_dim contiguous, address and the other
// strides multiples of 16 bytes), else a packed copy; `strides` = those of B, N, S.  (The stride of a dimension of size 1
// may be anything, also in a tensor that counts as contiguous: those of the packed form are computed.)
Tensor readable(const Tensor& t, int64_t (&strides)[3]) {
  bool as_is = t.stride(3) == 1 && reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0 && t.stride(2) >= t.size(3);
  for (int i = 0; i < 3; ++i) {
    strides[i] = t.stride(i);
    as_is = as_is && strides[i] > 0 && strides[i] % 8 == 0;
  }
  if (as_is) return t;
  for (int i = 2; i >= 0; --i) strides[i] = i == 2 ? t.size(3) : strides[i + 1] * t.size(i + 1);
  return t.contiguous();
}

// The gradient of the training operator: dq, dk, dv in the inputs' type (what the reference's bprop hands back after
// its cast, flash_attention_impl.py:117-124).  The output gradient is read in the layout it arrives in: behind a transpose
// back to [B, S, N*D] it is a strided view, and copying it would be one more pass over memory.
//
// The forward and this are one custom function of torch's C++ interface, so that what autograd offers around a function --
// saved-tensor hooks, compiled autograd, gradients that are not there -- works as around a Python one.
struct FaCall {
  FaConfig cfg;
  Tensor tiles;          // of the mask: this library's own, no user sees or changes it
  Tensor* lse;           // (not an output of the function: it has no gradient, and its saved form is not an output's)
};

struct FaFunction : public torch::autograd::Function<FaFunction> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& mask_in,
                        const std::optional<Tensor>& drop_in, const std::optional<Tensor>& alibi_in, const FaCall& call) {
    const FaConfig& c = call.cfg;
    Tensor mask = mask_in.value_or(Tensor()), drop = drop_in.value_or(Tensor()), alibi = alibi_in.value_or(Tensor());
    Tensor o, lse, plan, norms;
    at::AutoDispatchBelowADInplaceOrView below;
    check_fa_inputs(q, k, v, mask, drop, alibi, call.tiles, c);     // (packs the last three)
    c10::cuda::OptionalCUDAGuard guard(q.device());
    o = empty_like_shape(q.sizes(), q.scalar_type(), q);
    lse = empty_like_shape(q.sizes().slice(0, 3), at::kFloat, q);
    acct_fa_args a;
    fill_args(a, q, k, v, o, lse, mask, drop, alibi, call.tiles, c);
    const size_t plan_bytes = g_lib.mask_plan_bytes(&a);
    bool keep_plan = false;
    if (plan_bytes > 0) {
      // The backward uses a plan up to head_dim 128 and where dQ is summed in any order.  The plan is kept for it where that
      // adds at most a sixteenth to what is saved anyway; a larger one (up to 64 MB, in every layer) is drawn up again from
      // the mask and its 16 bytes of norms, which takes about 25 us (3 000 tokens of four documents, 2 x 32 heads of 128:
      // 4.7 MB next to 123 MB, forward and backward 471 us kept, 496 us drawn up again).
      const bool wanted = q.size(3) <= 128 && !c.deterministic;
      keep_plan = wanted && plan_bytes * 16 <= 2 * (q.nbytes() + k.nbytes());
      plan = empty_like_shape({static_cast<int64_t>(plan_bytes)}, at::kByte, q);
      if (wanted && !keep_plan) norms = empty_like_shape({16}, at::kByte, q);
      check(g_lib.mask_plan(&a, plan.data_ptr(), norms.defined() ? norms.data_ptr() : nullptr, 0, stream_of(q)));
    }
    check(g_lib.fa_fwd(&a, plan.defined() ? plan.const_data_ptr() : nullptr, stream_of(q)));
    *call.lse = lse;
    // (the optional inputs as given, not their packed copies)
    ctx->save_for_backward({q, k, v, o, lse, mask_in.value_or(Tensor()), drop_in.value_or(Tensor()), alibi_in.value_or(Tensor()),
                            keep_plan ? plan : Tensor()});
    ctx->saved_data["config"] = c.pack();
    if (call.tiles.defined()) ctx->saved_data["tiles"] = call.tiles;
    if (norms.defined()) ctx->saved_data["norms"] = norms;
    return o;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    Tensor o = saved[3], lse = saved[4], mask = saved[5], drop = saved[6], alibi = saved[7], d_o = grads[0];
    const auto tensor_of = [ctx](const char* key) {
      const auto it = ctx->saved_data.find(key);
      return it == ctx->saved_data.end() ? Tensor() : it->second.toTensor();
    };
    const Tensor tiles = tensor_of("tiles"), norms = tensor_of("norms");
    const FaConfig cfg = FaConfig::unpack(ctx->saved_data.at("config").toIntVector());

    at::AutoDispatchBelowADInplaceOrView below;
    // saved-tensor hooks may have handed back tensors of another layout, or of another device: checked like the inputs
    check_fa_inputs(q, k, v, mask, drop, alibi, tiles, cfg);
    require_on("o", o, q);
    require_on("lse", lse, q);
    HOST_CHECK(o.sizes() == q.sizes() && o.scalar_type() == q.scalar_type(), "o must have the shape and dtype of q");
    HOST_CHECK(lse.sizes() == q.sizes().slice(0, 3) && lse.scalar_type() == at::kFloat, "lse must be float32 [B, N, S_q]");
    lse = lse.contiguous();
    c10::cuda::OptionalCUDAGuard guard(q.device());
    int64_t o_strides[3], d_o_strides[3];
    o = readable(o, o_strides);
    d_o = readable(d_o, d_o_strides);
    acct_fa_args a;
    fill_args(a, q, k, v, o, lse, mask, drop, alibi, tiles, cfg);
    std::copy(o_strides, o_strides + 3, a.o_stride);
    if (cfg.deterministic) a.flags |= ACCT_FLAG_DETERMINISTIC;
    const auto dt = q.scalar_type();
    Tensor dq = empty_like_shape(q.sizes(), dt, q), dk = empty_like_shape(k.sizes(), dt, q), dv = empty_like_shape(v.sizes(), dt, q);
    const size_t nbytes = g_lib.fa_bwd_workspace_bytes(&a);
    const int64_t own = (nbytes + 15) / 16 * 16;      // behind it 16 bytes for the statistics that go with a mask plan
    Tensor ws = empty_like_shape({own + 16}, at::kByte, q);
    acct_fa_bwd_io g;
    memset(&g, 0, sizeof(g));
    g.d_o = d_o.const_data_ptr();
    g.dq = dq.data_ptr(); g.dk = dk.data_ptr(); g.dv = dv.data_ptr();
    g.workspace = ws.data_ptr(); g.workspace_bytes = nbytes;
    Tensor plan = saved[8];
    if (plan.defined()) {
      require_on("plan", plan, q);
      HOST_CHECK(plan.scalar_type() == at::kByte && static_cast<size_t>(plan.numel()) == g_lib.mask_plan_bytes(&a), "not the plan that was saved");
      plan = plan.contiguous();
    } else if (norms.defined()) {
      plan = empty_like_shape({static_cast<int64_t>(g_lib.mask_plan_bytes(&a))}, at::kByte, q);
      check(g_lib.mask_plan(&a, plan.data_ptr(), norms.data_ptr(), 1, stream_of(q)));
    }
    check(g_lib.fa_bwd(&a, &g, d_o_strides, plan.defined() ? plan.const_data_ptr() : nullptr,
                       static_cast<uint8_t*>(ws.data_ptr()) + own, stream_of(q)));
    return {dq, dk, dv, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ---------------------------------------------------------------------------------------------
// CPython entry points (positional arguments only; ops.py and the operator modules are the callers)
// ---------------------------------------------------------------------------------------------
Tensor tensor_or_undefined(PyObject* p) {
  if (p == Py_None) return Tensor();
  HOST_CHECK(THPVariable_Check(p), "expected a tensor or None");
  return THPVariable_Unpack(p);
}
Tensor tensor_arg(PyObject* p, const char* name) {
  HOST_CHECK(THPVariable_Check(p), name, " must be a CUDA tensor (this library has no CPU path)");
  return THPVariable_Unpack(p);
}
int64_t int_arg(PyObject* p) {
  const long long v = PyLong_AsLongLong(p);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
// what int() and float() take, for the arguments that the Python front end passes through them
THPObjectPtr as_int(PyObject* p) {
  THPObjectPtr v(PyNumber_Long(p));
  if (!v) throw python_error();
  return v;
}
uint64_t low_bits_arg(PyObject* p) {
  const uint64_t v = PyLong_AsUnsignedLongLongMask(as_int(p).get());
  if (PyErr_Occurred()) throw python_error();
  return v;
}
int64_t block_count_arg(PyObject* p) {      // anything below 0 is refused by the library, anything large means unbounded
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(as_int(p).get(), &overflow);
  if (v == -1 && overflow == 0 && PyErr_Occurred()) throw python_error();
  if (overflow != 0) return overflow > 0 ? ACCT_BAND_UNBOUNDED : -1;
  return std::max<long long>(-1, std::min<long long>(v, ACCT_BAND_UNBOUNDED));
}
double float_arg(PyObject* p) {
  THPObjectPtr v(PyNumber_Float(p));
  if (!v) throw python_error();
  return PyFloat_AS_DOUBLE(v.get());
}
bool bool_arg(PyObject* p) {
  const int v = PyObject_IsTrue(p);
  if (v < 0) throw python_error();
  return v != 0;
}
PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }

PyObject* py_init(PyObject*, PyObject* path) {
  HANDLE_TH_ERRORS
  const char* p = PyUnicode_AsUTF8(path);
  if (p == nullptr) throw python_error();
  void* h = dlopen(p, RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h != nullptr, "cannot load ", p, ": ", dlerror());
  auto sym = [&](const char* name) {
    void* f = dlsym(h, name);
    TORCH_CHECK(f != nullptr, p, " has no ", name);
    return f;
  };
  g_lib.fa_fwd = reinterpret_cast<decltype(g_lib.fa_fwd)>(sym("acct_fa_fwd_planned"));
  g_lib.fa_bwd = reinterpret_cast<decltype(g_lib.fa_bwd)>(sym("acct_fa_bwd_planned"));
  g_lib.mask_plan_bytes = reinterpret_cast<decltype(g_lib.mask_plan_bytes)>(sym("acct_mask_plan_bytes"));
  g_lib.mask_plan = reinterpret_cast<decltype(g_lib.mask_plan)>(sym("acct_mask_plan_norms"));
  g_lib.fa_bwd_workspace_bytes = reinterpret_cast<decltype(g_lib.fa_bwd_workspace_bytes)>(sym("acct_fa_bwd_workspace_bytes"));
  g_lib.infer_prefill = reinterpret_cast<decltype(g_lib.infer_prefill)>(sym("acct_infer_prefill"));
  g_lib.infer_decode = reinterpret_cast<decltype(g_lib.infer_decode)>(sym("acct_infer_decode"));
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// fa_apply(q, k, v, attn_mask, dropout_mask, alibi, mask_tiles, mask_tile128, causal, keep_prob, prev, next, scale,
//          tri_block, deterministic, seed | None, offset) -> (output, rowsum), differentiable in q, k, v
PyObject* py_fa_apply(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  HOST_CHECK(n == 17, "fa_apply takes 17 arguments, got ", n);
  const Tensor q = tensor_arg(args[0], "q"), k = tensor_arg(args[1], "k"), v = tensor_arg(args[2], "v");
  const Tensor mask = tensor_or_undefined(args[3]), drop = tensor_or_undefined(args[4]), alibi = tensor_or_undefined(args[5]);
  const Tensor tiles = tensor_or_undefined(args[6]);
  FaConfig c;
  c.mask_tile128 = bool_arg(args[7]);
  c.causal = bool_arg(args[8]);
  c.keep_prob = float_arg(args[9]);
  c.prev = block_count_arg(args[10]);
  c.next = block_count_arg(args[11]);
  c.scale = float_arg(args[12]);
  c.tri_block = static_cast<int32_t>(low_bits_arg(args[13]));
  c.deterministic = bool_arg(args[14]);
  if (args[15] != Py_None) {
    c.has_seed = 1;
    c.seed = low_bits_arg(args[15]);
    c.offset = low_bits_arg(args[16]);
  }
  // as a Python autograd Function without a `jvp` does; a tangent would be dropped silently otherwise
  for (const Tensor* t : {&q, &k, &v, &mask, &drop, &alibi})
    TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(/*level=*/0).defined(),
                                "the flash attention operator does not support forward mode AD");
  // (an optional input may require a gradient too: it gets none, but the output is part of the graph)
  const auto given = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
  Tensor o, lse;
  {
    pybind11::gil_scoped_release no_gil;
    o = FaFunction::apply(q, k, v, given(mask), given(drop), given(alibi), FaCall{c, tiles, &lse});
  }
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, wrap(o));
  PyTuple_SET_ITEM(r, 1, wrap(lse));
  return r;
  END_HANDLE_TH_ERRORS
}

// infer_prefill(q, k, v, causal, scale, seq_lens | None) -> y
PyObject* py_infer_prefill(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  HOST_CHECK(n == 6, "infer_prefill takes 6 arguments, got ", n);
  Tensor q = tensor_arg(args[0], "q"), k = tensor_arg(args[1], "k"), v = tensor_arg(args[2], "v");
  const bool causal = bool_arg(args[3]);
  const double scale = float_arg(args[4]);
  Tensor lens = tensor_or_undefined(args[5]), y;
  {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    require_cuda("q", q); require_on("k", k, q); require_on("v", v, q);
    HOST_CHECK(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), "q, k, v must share one dtype");
    const int64_t rank = q.dim();
    HOST_CHECK(rank == 3 || rank == 4, "q must have rank 3 or 4");
    HOST_CHECK(k.dim() == rank && v.dim() == rank && k.sizes() == v.sizes(), "k and v must have q's rank and one shape");
    q = q.contiguous(); k = k.contiguous(); v = v.contiguous();
    const int64_t hd = rank - 3;       // position of the head dimension
    HOST_CHECK((rank == 3 || q.size(0) == k.size(0)) && q.size(-1) == k.size(-1) && k.size(hd) > 0 && q.size(hd) % k.size(hd) == 0,
               "q and k must agree on batch and head_dim, and k's head count must divide q's");
    c10::cuda::OptionalCUDAGuard guard(q.device());
    y = empty_like_shape(q.sizes(), q.scalar_type(), q);
    acct_infer_args a;
    memset(&a, 0, sizeof(a));
    a.dtype = q.scalar_type() == at::kHalf ? ACCT_F16 : q.scalar_type() == at::kBFloat16 ? ACCT_BF16 : -1;
    a.rank = rank;
    a.B = rank == 4 ? q.size(0) : 1; a.N = q.size(hd); a.S_q = q.size(hd + 1); a.D = q.size(hd + 2);
    a.N_kv = k.size(hd); a.S_k = k.size(hd + 1);
    a.q = q.const_data_ptr(); a.k = k.const_data_ptr(); a.v = v.const_data_ptr(); a.y = y.data_ptr();
    a.causal = causal ? 1 : 0;
    a.scale = static_cast<float>(scale);
    if (lens.defined()) {
      lens = lengths(lens, a.B, q);
      a.seq_lens = static_cast<const int32_t*>(lens.const_data_ptr());
    }
    check(g_lib.infer_prefill(&a, stream_of(q)));
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// infer_decode(q, k_cache, v_cache, seq_lens | None, scale, num_splits, workspace, out | None, block_table | None) -> y
PyObject* py_infer_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  HOST_CHECK(n == 9, "infer_decode takes 9 arguments, got ", n);
  Tensor q = tensor_arg(args[0], "q"), k = tensor_arg(args[1], "k_cache"), v = tensor_arg(args[2], "v_cache");
  Tensor lens = tensor_or_undefined(args[3]);
  const double scale = float_arg(args[4]);
  const int64_t splits = int_arg(args[5]);
  const Tensor ws = tensor_arg(args[6], "workspace");
  Tensor y = tensor_or_undefined(args[7]), table = tensor_or_undefined(args[8]);
  {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    require_cuda("q", q); require_on("k_cache", k, q); require_on("v_cache", v, q); require_on("workspace", ws, q);
    HOST_CHECK(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
               "q, k_cache, v_cache must share one dtype");
    HOST_CHECK(q.dim() == 4 && q.size(2) == 1, "decode takes one query token: q must be [B, N, 1, D]");
    const int64_t B = q.size(0), N = q.size(1), D = q.size(3);
    const bool paged = table.defined();
    HOST_CHECK(k.dim() == 4 && k.sizes() == v.sizes() && (paged || k.size(0) == B) && k.size(3) == D && k.size(1) >= 1 &&
                   N % k.size(1) == 0,
               "k_cache and v_cache must be [B, N_kv, S_max, D] (or page pools [pages, N_kv, page_size, D]) with N_kv dividing q's head count");
    HOST_CHECK(k.strides() == v.strides(), "k_cache and v_cache must share strides");
    c10::cuda::OptionalCUDAGuard guard(q.device());
    q = q.contiguous();
    if (y.defined()) {
      require_on("out", y, q);
      HOST_CHECK(y.scalar_type() == q.scalar_type() && y.is_contiguous() && y.numel() == q.numel(),
                 "out must be a contiguous tensor with the dtype and the number of elements of q");
    } else {
      y = empty_like_shape(q.sizes(), q.scalar_type(), q);
    }
    acct_decode_args a;
    memset(&a, 0, sizeof(a));
    a.dtype = q.scalar_type() == at::kHalf ? ACCT_F16 : q.scalar_type() == at::kBFloat16 ? ACCT_BF16 : -1;
    a.B = B; a.N = N; a.D = D; a.N_kv = k.size(1);
    if (paged) {
      require_on("block_table", table, q);
      table = table.to(at::kInt).contiguous();
      HOST_CHECK(table.dim() == 2 && table.size(0) == B, "block_table must be [B, max_pages]");
      a.block_table = static_cast<const int32_t*>(table.const_data_ptr());
      a.page_size = k.size(2);
      a.max_pages = table.size(1);
      a.S_max = a.page_size * a.max_pages;
    } else {
      a.S_max = k.size(2);
    }
    a.q = q.const_data_ptr(); a.k_cache = k.const_data_ptr(); a.v_cache = v.const_data_ptr(); a.y = y.data_ptr();
    strides3(k, a.kv_stride);
    if (lens.defined()) {
      lens = lengths(lens, a.B, q);
      a.seq_lens = static_cast<const int32_t*>(lens.const_data_ptr());
    }
    a.scale = static_cast<float>(scale);
    a.num_splits = splits;
    a.workspace = ws.data_ptr();
    a.workspace_bytes = ws.nbytes();
    check(g_lib.infer_decode(&a, stream_of(q)));
  }
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(F)); }

PyMethodDef kMethods[] = {
    {"init", py_init, METH_O, "look the entry points up in the library at this path"},
    {"fa_apply", fast<py_fa_apply>(), METH_FASTCALL, "training operator, differentiable"},
    {"infer_prefill", fast<py_infer_prefill>(), METH_FASTCALL, "inference op"},
    {"infer_decode", fast<py_infer_decode>(), METH_FASTCALL, "one decoding step"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_host", "native host path of acctransformer_b200", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

// (the loader compares `built_for` with the running torch and interpreter before it calls anything: build.py)
PyMODINIT_FUNC PyInit__torch_host(void) {
  PyObject* m = PyModule_Create(&kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", ACCT_BUILT_FOR) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
