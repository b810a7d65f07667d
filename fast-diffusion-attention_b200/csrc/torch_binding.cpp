// Host path of the Python functions, in C++: argument checks, output and workspace allocation, the launch through the
// C ABI (include/fda.h) and the autograd node. It replaces the reference's torch operators and autograd Functions
// (csrc/fda/flash_api.cpp:92-139, :322-682 and fast_diffusion_attention/interface.py:40-207 there).
//
// Why native: a training step on a small problem is a handful of kernels of 5 to 20 us each, and the same work done
// in Python (custom-operator wrappers, argument structs filled field by field, a Python autograd node) took 290 us of
// host time a step, more than the GPU needs for two samples of 1K tokens and 32 heads. Here a call costs the tensor
// allocations and the launches.
//
// The module is a plain CPython extension. `attention` and `attention_packed` serve ordinary eager calls and answer
// None for everything else (tensor subclasses, fake or meta tensors, dispatch modes, functorch, tracing): the Python
// layer then takes its operators, whose bodies come back here through `forward` and `backward`.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <dlfcn.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <optional>
#include <string>

#include "../../include/fda.h"

namespace {

using at::Tensor;

// ---- the C ABI, from the library the Python layer names (it may be another build of it) -----------------------
struct Abi {
  decltype(&fda_fwd_workspace_bytes) fwd_workspace_bytes = nullptr;
  decltype(&fda_bwd_workspace_bytes) bwd_workspace_bytes = nullptr;
  decltype(&fda_fwd) fwd = nullptr;
  decltype(&fda_bwd_stages) bwd_stages = nullptr;
  decltype(&fda_strerror) strerror_ = nullptr;
  decltype(&fda_last_cuda_error) last_cuda_error = nullptr;
} abi;

void check_status(int rc) {
  if (rc == FDA_OK) return;
  std::string msg = std::string("fast-diffusion-attention: ") + abi.strerror_(rc);
  const char* detail = abi.last_cuda_error();
  if (rc == FDA_ERR_CUDA && detail[0] != 0) msg += std::string(" [") + detail + "]";
  TORCH_CHECK(false, msg);
}

// ---- one call's options ---------------------------------------------------------------------------------------
struct Options {
  int64_t block_size = 0;
  int64_t max_seqlen = -1;      // -1: not given
  std::optional<double> softmax_scale;   // not given: 1 / sqrt(head dim)
  double softcap = 0.0;
  bool deterministic = false;
  int64_t sm_margin = 0;
  int64_t heads_q = -1;         // packed projections: -1 = a separate axis of size 3
};

struct Shape {
  int64_t batch, seqlen, total, heads, heads_k, head_dim;
  bool varlen;
};

bool is_16bit(const Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }

int32_t dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return FDA_BF16;
    case at::kHalf: return FDA_FP16;
    case at::kFloat8_e4m3fn: return FDA_E4M3;
    default: return -1;
  }
}

// The kernels move tiles with TMA and rows with 16-byte vector accesses: the base address and every stride but the
// last must be multiples of 16 bytes.
bool tile_copy_friendly(const Tensor& t) {
  const int64_t size = t.element_size();
  if (reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 != 0) return false;
  for (int64_t i = 0; i + 1 < t.dim(); ++i) {
    if (t.size(i) > 1 && (t.stride(i) * size) % 16 != 0) return false;
  }
  return true;
}

// An expanded view: the gradient that a sum over tokens or heads hands back, keys that heads share. Tensor maps have no
// stride of 0.
bool repeats_itself(const Tensor& t) {
  for (int64_t i = 0; i < t.dim(); ++i) {
    if (t.size(i) > 1 && t.stride(i) == 0) return true;
  }
  return false;
}

// The reference copies an input only when its last dimension is strided (interface.py:17-18 there); a view whose base
// or strides are not 16-byte multiples, or with a stride of 0, is copied as well, so that every call the reference accepts
// is accepted.
Tensor maybe_contiguous(const Tensor& t) {
  if (!t.is_cuda()) return t;   // refused by the checks
  if (t.dim() >= 1 && (t.stride(-1) != 1 || (t.dim() >= 3 && (!tile_copy_friendly(t) || repeats_itself(t))))) {
    return t.contiguous();
  }
  return t;
}

// Offsets may be a strided view (a column of a table); forward and backward copy it alike.
Tensor contiguous_offsets(const Tensor& cu) { return cu.defined() && cu.dim() == 1 && cu.is_cuda() ? cu.contiguous() : cu; }

// The checks of the reference's check_inputs (csrc/fda/flash_api.cpp:92-139), same key words.
Shape check_inputs(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& cu, const Options& o,
                   bool backward) {
  TORCH_CHECK(backward || dtype_code(q) >= 0,
              "fast-diffusion-attention only supports fp16, bf16, and fp8_e4m3 data type");
  TORCH_CHECK(!backward || is_16bit(q), "fast-diffusion-attention backward only supports fp16 and bf16 data type");
  TORCH_CHECK(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
              "query, key and value must have the same dtype");
  for (const Tensor* t : {&q, &k, &v}) {
    TORCH_CHECK(t->is_cuda(), "Input tensor must be on CUDA device");
    TORCH_CHECK(t->device() == q.device(), "query, key and value must be on the same device");
    TORCH_CHECK(t->dim() >= 2 && t->stride(-1) == 1, "Input tensor must have contiguous last dimension");
  }
  TORCH_CHECK(o.block_size >= 1, "block_size must be a positive integer");
  Shape s;
  s.varlen = cu.defined();
  s.heads = q.size(-2);
  s.head_dim = q.size(-1);
  s.heads_k = k.size(-2);
  if (!s.varlen) {
    TORCH_CHECK(q.dim() == 4, "q must have shape (batch_size, seqlen, num_heads, head_size)");
    s.batch = q.size(0);
    s.seqlen = q.size(1);
    s.total = s.batch * s.seqlen;
    TORCH_CHECK(s.seqlen % 2 == 0, "The sequence length must be even: [noisy half | clean half]");
    const int64_t want[4] = {s.batch, s.seqlen, s.heads_k, s.head_dim};
    TORCH_CHECK(k.sizes() == at::IntArrayRef(want, 4) && v.sizes() == k.sizes(),
                "k and v must have shape (batch_size, seqlen, num_heads_k, head_size)");
  } else {
    TORCH_CHECK(cu.scalar_type() == at::kInt, "cu_seqlens must have dtype torch.int32");
    TORCH_CHECK(cu.is_cuda() && cu.is_contiguous(), "cu_seqlens must be a contiguous CUDA tensor");
    TORCH_CHECK(cu.dim() == 1 && cu.numel() >= 1, "cu_seqlens must be one-dimensional with batch_size + 1 entries");
    TORCH_CHECK(o.max_seqlen >= 0, "max_seqlen must be provided if cu_seqlens is provided");
    TORCH_CHECK(q.dim() == 3, "q must have shape (total, num_heads, head_size) if cu_seqlens is provided");
    s.batch = cu.size(0) - 1;
    s.seqlen = o.max_seqlen;
    s.total = q.size(0);
    const int64_t want[3] = {s.total, s.heads_k, s.head_dim};
    TORCH_CHECK(k.sizes() == at::IntArrayRef(want, 3) && v.sizes() == k.sizes(),
                "k and v must have shape (total, num_heads_k, head_size)");
  }
  TORCH_CHECK(s.head_dim <= 256, "fast-diffusion-attention supports head dimension at most 256");
  TORCH_CHECK(s.heads_k > 0 && s.heads % s.heads_k == 0,
              "Number of heads in key/value must divide number of heads in query");
  const int64_t align = is_16bit(q) ? 8 : 16;
  TORCH_CHECK(s.head_dim % align == 0, "head_size should be a multiple of ", align);
  constexpr int64_t kMax = 0x7fffffff;
  TORCH_CHECK(s.total <= kMax && s.seqlen <= kMax && o.block_size <= kMax && s.heads <= kMax, "tensor sizes beyond 2^31");
  return s;
}

FdaTensor tensor_view(const Tensor& t, bool varlen) {
  FdaTensor f;
  f.ptr = const_cast<void*>(t.const_data_ptr());
  const int row = varlen ? 0 : 1;
  f.head_stride = t.size(row + 1) > 1 ? t.stride(row + 1) : t.size(row + 2);
  f.row_stride = t.size(row) > 1 ? t.stride(row) : t.size(row + 1) * t.size(row + 2);
  f.batch_stride = varlen ? 0 : t.stride(0);
  return f;
}

double scale_of(const Options& o, const Shape& s) {
  return o.softmax_scale ? *o.softmax_scale : 1.0 / std::sqrt(static_cast<double>(s.head_dim));
}

FdaProblem problem_of(const Tensor& q, const Tensor& cu, const Shape& s, const Options& o) {
  FdaProblem p;
  p.dtype = dtype_code(q);
  p.batch = static_cast<int32_t>(s.batch);
  p.seqlen = static_cast<int32_t>(s.seqlen);
  p.total = static_cast<int32_t>(s.total);
  p.heads = static_cast<int32_t>(s.heads);
  p.heads_k = static_cast<int32_t>(s.heads_k);
  p.head_dim = static_cast<int32_t>(s.head_dim);
  p.block_size = static_cast<int32_t>(o.block_size);
  p.softmax_scale = static_cast<float>(scale_of(o, s));
  p.softcap = static_cast<float>(o.softcap);
  p.sm_margin = static_cast<int32_t>(o.sm_margin);
  p.deterministic = o.deterministic ? 1 : 0;
  p.cu_seqlens = cu.defined() ? static_cast<const int32_t*>(cu.const_data_ptr()) : nullptr;
  return p;
}

Tensor empty_on(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& like) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt));
}

// ---- forward / backward on plain tensors ------------------------------------------------------------------------
std::pair<Tensor, Tensor> forward_impl(Tensor q, Tensor k, Tensor v, const Tensor& cu_in, const Tensor* descales,
                                       const Options& o) {
  RECORD_FUNCTION("fda::_diffusion_attn_forward", c10::ArrayRef<const c10::IValue>{});
  q = maybe_contiguous(q);
  k = maybe_contiguous(k);
  v = maybe_contiguous(v);
  const Tensor cu = contiguous_offsets(cu_in);
  const Shape s = check_inputs(q, k, v, cu, o, false);
  const bool fp8 = !is_16bit(q);
  TORCH_CHECK(fp8 || !(descales[0].defined() || descales[1].defined() || descales[2].defined()),
              "q_descale, k_descale and v_descale are only supported for FP8 inputs");
  c10::cuda::OptionalCUDAGuard on_device;
  if (q.device().index() != c10::cuda::current_device()) on_device.set_device(q.device());
  Tensor out = empty_on(q.sizes(), fp8 ? at::kBFloat16 : q.scalar_type(), q);
  Tensor lse = s.varlen ? empty_on({s.heads, s.total}, at::kFloat, q) : empty_on({s.batch, s.heads, s.seqlen}, at::kFloat, q);
  if (s.total == 0 || s.heads == 0) {
    out.zero_();
    lse.fill_(INFINITY);
    return {out, lse};
  }
  FdaFwdArgs a;
  std::memset(&a, 0, sizeof(a));
  a.p = problem_of(q, cu, s, o);
  a.q = tensor_view(q, s.varlen);
  a.k = tensor_view(k, s.varlen);
  a.v = tensor_view(v, s.varlen);
  a.out = tensor_view(out, s.varlen);
  a.lse = static_cast<float*>(lse.mutable_data_ptr());
  const float** slots[3] = {&a.q_descale, &a.k_descale, &a.v_descale};
  const char* names[3] = {"q_descale", "k_descale", "v_descale"};
  for (int i = 0; i < 3; ++i) {
    const Tensor& d = descales[i];
    if (!d.defined()) continue;
    TORCH_CHECK(d.dim() == 2 && d.size(0) == s.batch && d.size(1) == s.heads_k && d.scalar_type() == at::kFloat &&
                    d.is_cuda(),
                names[i], " must be a float32 CUDA tensor of shape (batch_size, num_heads_k)");
    *slots[i] = static_cast<const float*>(d.const_data_ptr());
    a.descale_batch_stride[i] = d.stride(0);
    a.descale_head_stride[i] = d.stride(1);
  }
  a.workspace_bytes = abi.fwd_workspace_bytes(&a.p);
  const Tensor ws = empty_on({static_cast<int64_t>(a.workspace_bytes)}, at::kByte, q);
  a.workspace = ws.mutable_data_ptr();
  check_status(abi.fwd(&a, c10::cuda::getCurrentCUDAStream(q.device().index()).stream()));
  return {out, lse};
}

int64_t padded_half(int64_t seqlen) { return (std::max<int64_t>(seqlen / 2, 1) + 127) / 128 * 128; }

// Returns the workspace: it starts with rowsum(dO * O) in the padded (batch, heads, half, n_pad) layout.
Tensor backward_impl(Tensor dout, Tensor q, Tensor k, Tensor v, Tensor out, const Tensor& lse, const Tensor& dq,
                     const Tensor& dk, const Tensor& dv, const Tensor& cu_in, const Options& o, Tensor workspace,
                     unsigned stages, Shape* shape) {
  RECORD_FUNCTION("fda::_diffusion_attn_backward", c10::ArrayRef<const c10::IValue>{});
  dout = maybe_contiguous(dout);
  q = maybe_contiguous(q);
  k = maybe_contiguous(k);
  v = maybe_contiguous(v);
  out = maybe_contiguous(out);
  const Tensor cu = contiguous_offsets(cu_in);
  const Shape s = check_inputs(q, k, v, cu, o, true);
  if (shape) *shape = s;
  TORCH_CHECK(out.scalar_type() == q.scalar_type() && dout.scalar_type() == q.scalar_type(),
              "query, out and dout must have the same dtype");
  TORCH_CHECK(out.sizes() == q.sizes() && dout.sizes() == q.sizes(), "out and dout must have the same shape as q");
  const Tensor* grads[3] = {&dq, &dk, &dv};
  const Tensor* of[3] = {&q, &k, &v};
  const char* names[3] = {"dq", "dk", "dv"};
  for (int i = 0; i < 3; ++i) {
    TORCH_CHECK(grads[i]->scalar_type() == q.scalar_type() && grads[i]->sizes() == of[i]->sizes() &&
                    grads[i]->stride(-1) == 1,
                names[i], " must have the dtype and shape of its input and a contiguous last dimension");
  }
  // the same checks as mha_bwd makes on its arguments (csrc/fda/flash_api.cpp:491, :523-529 of the reference): the
  // kernels index these tensors without looking at them again
  const std::pair<const char*, const Tensor*> on[6] = {{"out", &out}, {"dout", &dout}, {"dq", &dq},
                                                       {"dk", &dk},   {"dv", &dv},     {"softmax_lse", &lse}};
  for (const auto& e : on) TORCH_CHECK(e.second->device() == q.device(), e.first, " must be on the same device as q");
  TORCH_CHECK(lse.scalar_type() == at::kFloat, "softmax_lse must have dtype float32");
  const int64_t want3[3] = {s.batch, s.heads, s.seqlen}, want2[2] = {s.heads, s.total};
  const at::IntArrayRef want = s.varlen ? at::IntArrayRef(want2, 2) : at::IntArrayRef(want3, 3);
  TORCH_CHECK(lse.sizes() == want, "softmax_lse must have shape ", want);
  TORCH_CHECK(lse.is_contiguous(), "softmax_lse must be contiguous");
  for (int i = 0; i < 3; ++i) {
    TORCH_CHECK(tile_copy_friendly(*grads[i]), names[i],
                " must have a 16-byte aligned base address and row/head/batch strides");
  }
  c10::cuda::OptionalCUDAGuard on_device;
  if (q.device().index() != c10::cuda::current_device()) on_device.set_device(q.device());
  if (s.total == 0 || s.heads == 0) {
    for (const Tensor* g : grads) g->zero_();
    return at::zeros({s.batch * s.heads * 2 * padded_half(s.seqlen) * 4}, q.options().dtype(at::kByte));
  }
  FdaBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  a.p = problem_of(q, cu, s, o);
  a.q = tensor_view(q, s.varlen);
  a.k = tensor_view(k, s.varlen);
  a.v = tensor_view(v, s.varlen);
  a.out = tensor_view(out, s.varlen);
  a.dout = tensor_view(dout, s.varlen);
  a.dq = tensor_view(dq, s.varlen);
  a.dk = tensor_view(dk, s.varlen);
  a.dv = tensor_view(dv, s.varlen);
  a.lse = static_cast<const float*>(lse.const_data_ptr());
  a.workspace_bytes = abi.bwd_workspace_bytes(&a.p);
  if (!workspace.defined()) {
    workspace = empty_on({static_cast<int64_t>(a.workspace_bytes)}, at::kByte, q);
  } else {
    TORCH_CHECK(workspace.numel() >= static_cast<int64_t>(a.workspace_bytes) && workspace.scalar_type() == at::kByte,
                "workspace must be a uint8 CUDA tensor of at least fda_bwd_workspace_bytes bytes");
  }
  a.workspace = workspace.mutable_data_ptr();
  check_status(abi.bwd_stages(&a, stages, c10::cuda::getCurrentCUDAStream(q.device().index()).stream()));
  return workspace;
}

// Views (q, k, v) of a packed projection: behind the leading axes either (3, heads, dim) or (heads_q + 2 heads_k, dim).
struct Views {
  Tensor q, k, v;
};
Views split_packed(const Tensor& qkv, int64_t heads_q, bool varlen) {
  const int64_t lead = varlen ? 1 : 2;
  if (qkv.dim() == lead + 3) return {qkv.select(lead, 0), qkv.select(lead, 1), qkv.select(lead, 2)};
  const int64_t heads_k = (qkv.size(-2) - heads_q) / 2;
  return {qkv.narrow(-2, 0, heads_q), qkv.narrow(-2, heads_q, heads_k), qkv.narrow(-2, heads_q + heads_k, heads_k)};
}

Tensor gradient_like(const Tensor& t) {
  return t.is_contiguous() ? empty_on(t.sizes(), t.scalar_type(), t) : at::empty_like(t);
}

// ---- who may be passed by -----------------------------------------------------------------------------------------
// No dispatch or function mode, function transform or tracer wants to see the operators.
bool plain_context() {
  return !c10::impl::dispatch_mode_enabled() && !at::impl::torch_function_mode_enabled() && !torch::jit::tracer::isTracing() &&
         !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

// A CUDA tensor whose memory holds its values: no subclass, wrapper or lazily applied operation in between.
bool plain_values(const Tensor& t) {
  return t.is_cuda() && t.layout() == at::kStrided && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
         !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                   c10::DispatchKey::Functionalize, c10::DispatchKey::Batched,
                                                   c10::DispatchKey::ZeroTensor, c10::DispatchKey::Negative,
                                                   c10::DispatchKey::Conjugate}));
}

// The Python layer's backward through the operators (interface.py `_gradients`), for calls that somebody wants to see.
PyObject* operator_backward = nullptr;

PyObject* none() {
  Py_INCREF(Py_None);
  return Py_None;
}

struct Gil {
  PyGILState_STATE st = PyGILState_Ensure();
  ~Gil() { PyGILState_Release(st); }
};

// ---- autograd node ----------------------------------------------------------------------------------------------
// One node for separate q, k, v and for one packed projection, batched or packed samples. Saves q, k, v (or qkv), out,
// lse and cu_seqlens, the set the reference saves (interface.py:158, :189 there). The gradients have no derivative of their
// own: under create_graph they come back as constants, as from the operators.
struct DiffusionAttentionBackward : public torch::autograd::Node {
  torch::autograd::SavedVariable in[3], out, lse, cu;   // cu: only of packed samples
  bool varlen = false;
  int n_in = 0;
  Options opts;

  std::string name() const override { return "_DiffusionAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& s : in) s.reset_data();
    out.reset_data();
    lse.reset_data();
    cu.reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& g) override {
    auto self = getptr();
    Tensor x[3];
    Tensor o, l, offsets;
    {
      std::lock_guard<std::mutex> lock(mutex_);   // another thread may be releasing the same graph
      for (int i = 0; i < n_in; ++i) x[i] = in[i].unpack();
      o = out.unpack(self);
      l = lse.unpack(self);
      if (varlen) offsets = cu.unpack();
    }
    const Tensor dout = g[0].defined() ? g[0] : at::zeros_like(o);
    torch::autograd::variable_list r(n_in);
    // The graph was built by an eager call, but the backward may run where a mode is on, or get a gradient that is more
    // than its memory.
    bool plain = plain_context() && plain_values(dout) && plain_values(o) && plain_values(l) && (!varlen || plain_values(offsets));
    for (int i = 0; i < n_in; ++i) plain = plain && plain_values(x[i]);
    if (!plain) {
      by_operator(x, dout, o, l, offsets, &r);
    } else {
      at::AutoDispatchBelowADInplaceOrView below;
      if (n_in == 3) {
        for (int i = 0; i < 3; ++i) r[i] = gradient_like(x[i]);
        backward_impl(dout, x[0], x[1], x[2], o, l, r[0], r[1], r[2], offsets, opts, Tensor(), 7u, nullptr);
      } else {
        r[0] = empty_on(x[0].sizes(), x[0].scalar_type(), x[0]);
        const Views v = split_packed(x[0], opts.heads_q, varlen);
        const Views d = split_packed(r[0], opts.heads_q, varlen);
        backward_impl(dout, v.q, v.k, v.v, o, l, d.q, d.k, d.v, offsets, opts, Tensor(), 7u, nullptr);
      }
    }
    return r;
  }

  // Compiled autograd: `apply` runs on traced stand-ins of the saved tensors, under the tracer's modes and so through the
  // operators, whose shape functions are registered.
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    for (int i = 0; i < n_in; ++i) args.collect(in[i], false);
    args.collect(out, true);
    args.collect(lse, true);
    if (varlen) args.collect(cu, false);
    args.collect(varlen);
    args.collect(n_in);
    args.collect(opts.block_size);
    args.collect(opts.max_seqlen);
    args.collect(opts.softmax_scale);
    args.collect(opts.softcap);
    args.collect(opts.deterministic);
    args.collect(opts.sm_margin);
    args.collect(opts.heads_q);
  }
  torch::autograd::variable_list apply_with_saved(const torch::autograd::variable_list& g,
                                                  torch::dynamo::autograd::SwapSavedVariables& saved) override {
    auto each = [&](auto&& fn) {
      for (int i = 0; i < n_in; ++i) fn(in[i]);
      fn(out);
      fn(lse);
      if (varlen) fn(cu);
    };
    each([&](torch::autograd::SavedVariable& v) { saved.before(v); });
    auto r = apply(torch::autograd::variable_list(g));
    each([&](torch::autograd::SavedVariable& v) { saved.after(v); });
    return r;
  }

  // _gradients(inputs, dout, out, lse, cu_seqlens, num_heads_q, max_seqlen, block_size, softmax_scale, softcap,
  //            deterministic, sm_margin) -> the inputs' gradients
  void by_operator(const Tensor* x, const Tensor& dout, const Tensor& o, const Tensor& l, const Tensor& offsets,
                   torch::autograd::variable_list* r) {
    Gil gil;
    auto own = [](PyObject* p) {
      if (!p) {
        python_error e;
        e.persist();
        throw e;
      }
      return THPObjectPtr(p);
    };
    auto integer = [](int64_t v) { return v < 0 ? none() : PyLong_FromLongLong(v); };
    THPObjectPtr inputs = own(PyTuple_New(n_in));
    for (int i = 0; i < n_in; ++i) PyTuple_SET_ITEM(inputs.get(), i, own(THPVariable_Wrap(x[i])).release());
    THPObjectPtr args = own(PyTuple_New(12));
    int at = 0;
    auto add = [&](PyObject* p) { PyTuple_SET_ITEM(args.get(), at++, own(p).release()); };
    add(inputs.release());
    for (const Tensor& t : {dout, o, l, offsets}) add(THPVariable_Wrap(t));
    add(integer(opts.heads_q));
    add(integer(opts.max_seqlen));
    add(PyLong_FromLongLong(opts.block_size));
    add(opts.softmax_scale ? PyFloat_FromDouble(*opts.softmax_scale) : none());
    add(PyFloat_FromDouble(opts.softcap));
    add(PyBool_FromLong(opts.deterministic));
    add(PyLong_FromLongLong(opts.sm_margin));
    THPObjectPtr grads = own(PyObject_CallObject(operator_backward, args.get()));
    TORCH_CHECK(PyTuple_Check(grads.get()) && PyTuple_GET_SIZE(grads.get()) == n_in, "one gradient for every input");
    for (int i = 0; i < n_in; ++i) (*r)[i] = THPVariable_Unpack(PyTuple_GET_ITEM(grads.get(), i));
  }
};

std::pair<Tensor, Tensor> attention(const Tensor* x, int n_in, const Tensor& cu, const Tensor* descales,
                                    const Options& o) {
  bool needs_grad = false;
  if (at::GradMode::is_enabled()) {
    for (int i = 0; i < n_in; ++i) needs_grad = needs_grad || x[i].requires_grad();
  }
  std::shared_ptr<DiffusionAttentionBackward> node;
  if (needs_grad) {
    node = std::shared_ptr<DiffusionAttentionBackward>(new DiffusionAttentionBackward(), torch::autograd::deleteNode);
    torch::autograd::edge_list edges;
    for (int i = 0; i < n_in; ++i) edges.push_back(torch::autograd::impl::gradient_edge(x[i]));
    node->set_next_edges(std::move(edges));
    node->n_in = n_in;
    node->varlen = cu.defined();
    node->opts = o;
  }
  std::pair<Tensor, Tensor> r;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    if (n_in == 3) {
      r = forward_impl(x[0], x[1], x[2], cu, descales, o);
    } else {
      const Views v = split_packed(x[0], o.heads_q, cu.defined());
      r = forward_impl(v.q, v.k, v.v, cu, descales, o);
    }
  }
  if (node) {
    torch::autograd::set_history(r.first, node);
    torch::autograd::set_history(r.second, node);
    // everything through hooks on saved tensors, in the order in which the Python node saves
    for (int i = 0; i < n_in; ++i) node->in[i] = torch::autograd::SavedVariable(x[i], false);
    node->out = torch::autograd::SavedVariable(r.first, true);
    node->lse = torch::autograd::SavedVariable(r.second, true);
    if (cu.defined()) node->cu = torch::autograd::SavedVariable(cu, false);
  }
  return r;
}

// ---- Python side ------------------------------------------------------------------------------------------------
// Conversions for the eager path: false where the object is not of the exact plain type (the caller then answers None
// and the Python layer takes the general path, which converts or refuses it as the operators do).
bool to_int(PyObject* o, int64_t* out) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  *out = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}
bool to_double(PyObject* o, double* out) {
  if (PyFloat_CheckExact(o)) { *out = PyFloat_AS_DOUBLE(o); return true; }
  int64_t i;
  if (PyLong_CheckExact(o) && to_int(o, &i)) { *out = static_cast<double>(i); return true; }
  return false;
}
bool to_bool(PyObject* o, bool* out) {
  if (!PyBool_Check(o)) return false;
  *out = o == Py_True;
  return true;
}
// An ordinary eager CUDA tensor (or parameter) without forward-mode tangents.
bool plain_tensor(PyObject* o, Tensor* out) {
  if (!THPVariable_CheckExact(o)) return false;
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !plain_values(t) || t._fw_grad(0).defined()) return false;
  *out = t;
  return true;
}
bool optional_plain_tensor(PyObject* o, Tensor* out) { return o == Py_None || plain_tensor(o, out); }

bool to_scale(PyObject* o, std::optional<double>* out) {
  if (o == Py_None) return true;
  double v;
  if (!to_double(o, &v)) return false;
  *out = v;
  return true;
}

PyObject* pair_to_python(const std::pair<Tensor, Tensor>& r) {
  PyObject* a = THPVariable_Wrap(r.first);
  PyObject* b = a ? THPVariable_Wrap(r.second) : nullptr;
  if (!b) { Py_XDECREF(a); return nullptr; }
  PyObject* t = PyTuple_New(2);
  if (!t) { Py_DECREF(a); Py_DECREF(b); return nullptr; }
  PyTuple_SET_ITEM(t, 0, a);
  PyTuple_SET_ITEM(t, 1, b);
  return t;
}

struct NoGil {
  PyThreadState* st = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(st); }
};

// attention(q, k, v, cu_seqlens, max_seqlen, block_size, softmax_scale, q_descale, k_descale, v_descale, softcap,
//           deterministic, sm_margin) -> (out, lse), or None when this is not an ordinary eager call
PyObject* py_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 13, "attention takes 13 arguments");
  Tensor x[3], cu, ds[3];
  Options o;
  if (!plain_context() || !plain_tensor(args[0], &x[0]) || !plain_tensor(args[1], &x[1]) || !plain_tensor(args[2], &x[2]) ||
      !optional_plain_tensor(args[3], &cu) || (args[4] != Py_None && !to_int(args[4], &o.max_seqlen)) ||
      !to_int(args[5], &o.block_size) || !to_scale(args[6], &o.softmax_scale) || !optional_plain_tensor(args[7], &ds[0]) ||
      !optional_plain_tensor(args[8], &ds[1]) || !optional_plain_tensor(args[9], &ds[2]) ||
      !to_double(args[10], &o.softcap) || !to_bool(args[11], &o.deterministic) || !to_int(args[12], &o.sm_margin)) {
    Py_RETURN_NONE;
  }
  // e4m3 inputs have no backward: what their autograd node does is the general path's business
  if (!is_16bit(x[0]) && at::GradMode::is_enabled() &&
      (x[0].requires_grad() || x[1].requires_grad() || x[2].requires_grad())) {
    Py_RETURN_NONE;
  }
  std::pair<Tensor, Tensor> r;
  {
    NoGil nogil;
    r = attention(x, 3, cu, ds, o);
  }
  return pair_to_python(r);
  END_HANDLE_TH_ERRORS
}

// attention_packed(qkv, num_heads_q, cu_seqlens, max_seqlen, block_size, softmax_scale, softcap, deterministic,
//                  sm_margin) -> (out, lse) or None, also for shapes that the Python layer explains and refuses
PyObject* py_attention_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 9, "attention_packed takes 9 arguments");
  Tensor x[3], cu, ds[3];
  Options o;
  if (!plain_context() || !plain_tensor(args[0], &x[0]) || (args[1] != Py_None && (!to_int(args[1], &o.heads_q) || o.heads_q < 0)) ||
      !optional_plain_tensor(args[2], &cu) || (args[3] != Py_None && !to_int(args[3], &o.max_seqlen)) ||
      !to_int(args[4], &o.block_size) || !to_scale(args[5], &o.softmax_scale) || !to_double(args[6], &o.softcap) ||
      !to_bool(args[7], &o.deterministic) || !to_int(args[8], &o.sm_margin)) {
    Py_RETURN_NONE;
  }
  const int64_t lead = cu.defined() ? 1 : 2;
  const bool three = x[0].dim() == lead + 3 && x[0].size(lead) == 3 && (o.heads_q < 0 || o.heads_q == x[0].size(-2));
  const bool flat = x[0].dim() == lead + 2 && o.heads_q > 0 && x[0].size(-2) > o.heads_q && (x[0].size(-2) - o.heads_q) % 2 == 0;
  if (!is_16bit(x[0]) || !(three || flat)) Py_RETURN_NONE;
  std::pair<Tensor, Tensor> r;
  {
    NoGil nogil;
    r = attention(x, 1, cu, ds, o);
  }
  return pair_to_python(r);
  END_HANDLE_TH_ERRORS
}

Tensor any_tensor(PyObject* o, const char* name) {
  if (o == Py_None) return Tensor();
  TORCH_CHECK(THPVariable_Check(o), name, " must be a tensor");
  return THPVariable_Unpack(o);
}
int64_t any_int(PyObject* o, const char* name) {
  int64_t v = 0;
  TORCH_CHECK(to_int(o, &v), name, " must be an integer");
  return v;
}
double any_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
bool any_bool(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}

// forward(...) with attention's arguments: the operator's body, without autograd
PyObject* py_forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 13, "forward takes 13 arguments");
  Tensor x[3] = {any_tensor(args[0], "q"), any_tensor(args[1], "k"), any_tensor(args[2], "v")};
  const Tensor cu = any_tensor(args[3], "cu_seqlens");
  const Tensor ds[3] = {any_tensor(args[7], "q_descale"), any_tensor(args[8], "k_descale"), any_tensor(args[9], "v_descale")};
  Options o;
  if (args[4] != Py_None) o.max_seqlen = any_int(args[4], "max_seqlen");
  TORCH_CHECK(PyLong_Check(args[5]), "block_size must be a positive integer");
  o.block_size = any_int(args[5], "block_size");
  if (args[6] != Py_None) o.softmax_scale = any_double(args[6]);
  o.softcap = any_double(args[10]);
  o.deterministic = any_bool(args[11]);
  o.sm_margin = any_int(args[12], "sm_margin");
  std::pair<Tensor, Tensor> r;
  {
    NoGil nogil;
    r = forward_impl(x[0], x[1], x[2], cu, ds, o);
  }
  return pair_to_python(r);
  END_HANDLE_TH_ERRORS
}

// backward(dout, q, k, v, out, lse, dq, dk, dv, block_size, cu_seqlens, max_seqlen, softmax_scale, softcap,
//          deterministic, sm_margin, workspace, stages) -> view of rowsum(dO * O), (batch, heads, 2, n_pad)
PyObject* py_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 18, "backward takes 18 arguments");
  static const char* names[9] = {"dout", "q", "k", "v", "out", "softmax_lse", "dq", "dk", "dv"};
  Tensor t[9];
  for (int i = 0; i < 9; ++i) {
    t[i] = any_tensor(args[i], names[i]);
    TORCH_CHECK(t[i].defined(), names[i], " must be a tensor");
  }
  Options o;
  TORCH_CHECK(PyLong_Check(args[9]), "block_size must be a positive integer");
  o.block_size = any_int(args[9], "block_size");
  const Tensor cu = any_tensor(args[10], "cu_seqlens");
  if (args[11] != Py_None) o.max_seqlen = any_int(args[11], "max_seqlen");
  if (args[12] != Py_None) o.softmax_scale = any_double(args[12]);
  o.softcap = any_double(args[13]);
  o.deterministic = any_bool(args[14]);
  o.sm_margin = any_int(args[15], "sm_margin");
  Tensor ws = any_tensor(args[16], "workspace");
  const unsigned stages = static_cast<unsigned>(any_int(args[17], "stages"));
  Tensor delta;
  {
    NoGil nogil;
    Shape s;
    ws = backward_impl(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], cu, o, ws, stages, &s);
    const int64_t n_pad = padded_half(s.seqlen);
    delta = ws.narrow(0, 0, s.batch * s.heads * 2 * n_pad * 4).view(at::kFloat).view({s.batch, s.heads, 2, n_pad});
  }
  return THPVariable_Wrap(delta);
  END_HANDLE_TH_ERRORS
}

PyObject* py_bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 2, "bind takes 2 arguments");
  const char* path = PyUnicode_AsUTF8(args[0]);
  if (!path) throw python_error();
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(lib, "cannot load ", path, ": ", dlerror());
  auto sym = [&](const char* name) {
    void* p = dlsym(lib, name);
    TORCH_CHECK(p, name, " is missing in ", path);
    return p;
  };
  abi.fwd_workspace_bytes = reinterpret_cast<decltype(abi.fwd_workspace_bytes)>(sym("fda_fwd_workspace_bytes"));
  abi.bwd_workspace_bytes = reinterpret_cast<decltype(abi.bwd_workspace_bytes)>(sym("fda_bwd_workspace_bytes"));
  abi.fwd = reinterpret_cast<decltype(abi.fwd)>(sym("fda_fwd"));
  abi.bwd_stages = reinterpret_cast<decltype(abi.bwd_stages)>(sym("fda_bwd_stages"));
  abi.strerror_ = reinterpret_cast<decltype(abi.strerror_)>(sym("fda_strerror"));
  abi.last_cuda_error = reinterpret_cast<decltype(abi.last_cuda_error)>(sym("fda_last_cuda_error"));
  Py_INCREF(args[1]);
  Py_XSETREF(operator_backward, args[1]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

template <typename F>
PyCFunction as_pycfunction(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }

PyMethodDef methods[] = {
    {"attention", as_pycfunction(py_attention), METH_FASTCALL, "eager attention with autograd, or None"},
    {"attention_packed", as_pycfunction(py_attention_packed), METH_FASTCALL, "the same on one packed projection"},
    {"forward", as_pycfunction(py_forward), METH_FASTCALL, "body of the forward operator"},
    {"backward", as_pycfunction(py_backward), METH_FASTCALL, "body of the backward operator"},
    {"bind", as_pycfunction(py_bind), METH_FASTCALL, "path of the kernel library, backward through the operators"},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fda_torch", "host path of fast_diffusion_attention", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fda_torch() { return PyModule_Create(&module); }
