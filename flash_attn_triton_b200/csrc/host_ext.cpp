// Host path between PyTorch and the C ABI: allocation of outputs, argument blocks, autograd nodes
// and stream lookup in C++.
//
// A small attention call is bounded by the host, not by the GPU: the same steps as
// torch.autograd.Function classes with ctypes argument blocks cost about 25 us per forward and
// 70 us per backward on the host, against kernels of 5-20 us.  The kernels themselves are reached
// through the addresses of libfa_b200.so's C functions, handed over once by init(), so that any build
// of that library can be driven.
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <string.h>

#include <array>
#include <list>
#include <mutex>

#include "../../include/fa_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------------
// the C ABI
// ---------------------------------------------------------------------------------------
typedef int (*AttnFn)(const fa_attn_args*, void*);
struct Abi {
  AttnFn fwd, varlen_fwd, preprocess, bwd_dq, bwd_dkdv, varlen_bwd_dq, varlen_bwd_dkdv;
  size_t (*bits_bytes)(const fa_attn_args*, int32_t);
  int (*bits)(const fa_attn_args*, void*, void*);
  int (*fwd_bits)(const fa_attn_args*, const void*, void*);
  int (*bwd_dq_bits)(const fa_attn_args*, const void*, void*);
  int (*bwd_dkdv_bits)(const fa_attn_args*, const void*, void*);
  int (*quantize_k)(const void*, int8_t*, float*, int64_t, int32_t, int32_t, void*);
  int (*fwd_int8)(const fa_int8_args*, void*);
  size_t (*int8_codes16_bytes)(const fa_int8_args*);
  int (*fwd_int8_codes16)(const fa_int8_args*, const void*, float*, void*, void*);
  int (*varlen_check)(const int32_t*, const int32_t*, int32_t, int64_t, int64_t, int32_t, int64_t, int64_t, int32_t, int32_t*, void*);
  int (*check_result)(int32_t, uint32_t*, void*);
  int (*decode)(const fa_decode_args*, void*);
  int (*decode_checked)(const fa_decode_args*, uint32_t*, void*);
  int32_t (*decode_counters)(const fa_decode_args*);
  size_t (*decode_workspace)(const fa_decode_args*);
  size_t (*decode_checked_workspace)(const fa_decode_args*);
  PyObject* check;   // _native.check(status, what): raises the Python exception of a status
};
Abi g_abi = {};

// Raises the Python exception of a non-zero status, from whichever thread runs the call.
void check(int status, const char* what) {
  if (status == 0) return;
  pybind11::gil_scoped_acquire gil;
  PyObject* r = PyObject_CallFunction(g_abi.check, "is", status, what);
  Py_XDECREF(r);
  if (r == nullptr) {
    python_error e;
    e.persist();
    throw std::move(e);
  }
  TORCH_CHECK(false, what, " failed (status ", status, ")");
}

// ---------------------------------------------------------------------------------------
// tensors as the kernels see them
// ---------------------------------------------------------------------------------------
enum Layout { kBSHD = 0, kBHSD = 1, kTHD = 2 };
enum Packing { kSeparate = 0, kQKV = 1, kKV = 2 };

// unit inner stride, 16-byte aligned rows
bool kernel_ready(const Tensor& t) {
  const auto st = t.strides();
  const size_t n = st.size();
  if (n == 0 || st[n - 1] != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) != 0) return false;
  for (size_t i = 0; i + 1 < n; ++i)
    if (st[i] % 8 != 0) return false;
  return true;
}
Tensor prep(const Tensor& t) { return kernel_ready(t) ? t : t.contiguous(); }

struct View {
  char* p;
  int64_t stride[3];                 // batch, row, head
  int64_t batch, rows, heads, dim;
};

// `packed` >= 0: dimension of t that holds q/k/v (or k/v), `which` the slice taken from it
View view_of(const Tensor& t, Layout layout, int packed, int which) {
  int64_t sz[4], st[4];
  int n = 0;
  for (int i = 0; i < t.dim(); ++i) {
    if (i == packed) continue;
    sz[n] = t.size(i);
    st[n] = t.stride(i);
    ++n;
  }
  View v;
  v.p = static_cast<char*>(t.data_ptr());
  if (packed >= 0) v.p += which * t.stride(packed) * t.element_size();
  v.dim = sz[n - 1];
  if (layout == kTHD) {
    v.batch = 1; v.rows = sz[0]; v.heads = sz[1];
    v.stride[0] = 0; v.stride[1] = st[0]; v.stride[2] = st[1];
  } else {
    const int r = layout == kBSHD ? 1 : 2, h = layout == kBSHD ? 2 : 1;
    v.batch = sz[0]; v.rows = sz[r]; v.heads = sz[h];
    v.stride[0] = st[0]; v.stride[1] = st[r]; v.stride[2] = st[h];
  }
  return v;
}

Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& dev) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, dev, std::nullopt));
}

// What a call is made with, beyond its tensors.
struct Params {
  Layout layout = kBSHD;
  Packing packing = kSeparate;
  int packed_dim = -1;
  double scale = 1.0, softcap = 0.0;
  int causal = 0, wl = -1, wr = -1, q_pos_offset = 0, impl = FA_IMPL_AUTO;
  int max_q = 0, max_k = 0;          // packed sequences
  int k_valid = 0;                   // keys used of each (batch, head); 0 = all (padded INT8 calls)
  double dropout_p = 0.0;
  uint64_t seed = 0;
  int row_stride = 0;
  // optional tensors
  Tensor cu_q, cu_k, used_q, used_k, alibi, bias;
};

void split(const Params& c, const variable_list& in, View& q, View& k, View& v) {
  switch (c.packing) {
    case kSeparate:
      q = view_of(in[0], c.layout, -1, 0); k = view_of(in[1], c.layout, -1, 0); v = view_of(in[2], c.layout, -1, 0);
      break;
    case kQKV:
      q = view_of(in[0], c.layout, c.packed_dim, 0); k = view_of(in[0], c.layout, c.packed_dim, 1);
      v = view_of(in[0], c.layout, c.packed_dim, 2);
      break;
    case kKV:
      q = view_of(in[0], c.layout, -1, 0); k = view_of(in[1], c.layout, c.packed_dim, 0);
      v = view_of(in[1], c.layout, c.packed_dim, 1);
      break;
  }
  if (c.k_valid > 0) k.rows = v.rows = c.k_valid;
}

void set_strides(int64_t* dst, const View& v) { memcpy(dst, v.stride, sizeof(v.stride)); }

void fill(fa_attn_args& a, const Params& c, const Tensor& first, const View& q, const View& k, const View& v,
          const View& o, float* lse) {
  memset(&a, 0, sizeof(a));
  a.dtype = first.scalar_type() == at::kBFloat16 ? FA_BF16 : FA_F16;
  TORCH_CHECK_VALUE(a.dtype == FA_BF16 || first.scalar_type() == at::kHalf, "unsupported dtype ", first.scalar_type());
  a.device = first.device().index();
  a.impl = c.impl;
  const bool packed = c.layout == kTHD;
  a.batch = packed ? (int)c.cu_q.numel() - 1 : (int)q.batch;
  a.seqlen_q = packed ? c.max_q : (int)q.rows;
  a.seqlen_k = packed ? c.max_k : (int)k.rows;
  a.heads_q = (int)q.heads; a.heads_kv = (int)k.heads; a.head_dim = (int)q.dim;
  a.q = q.p; a.k = k.p; a.v = v.p; a.o = o.p;
  set_strides(a.q_stride, q); set_strides(a.k_stride, k); set_strides(a.v_stride, v); set_strides(a.o_stride, o);
  if (packed) {
    a.cu_seqlens_q = c.cu_q.const_data_ptr<int32_t>();
    a.cu_seqlens_k = c.cu_k.const_data_ptr<int32_t>();
    a.total_q = (int)q.rows; a.total_k = (int)k.rows;
  }
  // base-2 LSE: (batch, heads, rows), packed (heads, tokens)
  a.lse2 = lse;
  a.lse_stride[0] = packed ? 0 : q.heads * q.rows;
  a.lse_stride[1] = 1;
  a.lse_stride[2] = q.rows;
  a.softmax_scale = (float)c.scale;
  a.softcap = (float)c.softcap;
  a.alibi_slopes = c.alibi.defined() ? c.alibi.const_data_ptr<float>() : nullptr;
  a.causal = c.causal; a.window_left = c.wl; a.window_right = c.wr; a.q_pos_offset = c.q_pos_offset;
  if (c.bias.defined()) {
    a.attn_bias = c.bias.const_data_ptr<float>();
    for (int i = 0; i < 4; ++i) a.bias_stride[i] = c.bias.stride(i);
  }
  if (c.dropout_p > 0.0) {
    a.dropout_p = (float)c.dropout_p;
    a.dropout_seed = c.seed;
    a.dropout_row_stride = c.row_stride;
  }
  if (c.used_q.defined()) a.seqused_q = c.used_q.const_data_ptr<int32_t>();
  if (c.used_k.defined()) a.seqused_k = c.used_k.const_data_ptr<int32_t>();
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

c10::SmallVector<int64_t, 4> lse_shape(const Params& c, const View& q) {
  if (c.layout == kTHD) return {q.heads, q.rows};
  return {q.batch, q.heads, q.rows};
}

// shape of one of q/k/v (the output has q's)
c10::SmallVector<int64_t, 4> shape_of(const Params& c, const View& v) {
  if (c.layout == kTHD) return {v.rows, v.heads, v.dim};
  if (c.layout == kBSHD) return {v.batch, v.rows, v.heads, v.dim};
  return {v.batch, v.heads, v.rows, v.dim};
}

// The dropout mask of a call as bits, where its kernels read it that way; an undefined tensor otherwise.  It
// is drawn again in the backward: that costs a few microseconds, keeping it would hold memory per layer.
Tensor dropout_bits(const fa_attn_args& a, const Tensor& t, bool backward) {
  if (!(a.dropout_p > 0.f)) return Tensor();
  const size_t bytes = g_abi.bits_bytes(&a, backward);
  if (bytes == 0) return Tensor();
  Tensor bits = empty_cuda({(int64_t)bytes}, at::kByte, t.device());
  check(g_abi.bits(&a, bits.mutable_data_ptr(), stream_of(t)), "fa_dropout_bits");
  return bits;
}

// The value checks of a packed call (the reference's, flash_attn_interface.py:588-626): started before the host work
// of the call, whose result is awaited before anything reads by cu_seqlens.
class VarlenCheck {
 public:
  void start(const Tensor& q, const Tensor& k, const Tensor& cu_q, const Tensor& cu_k, bool k_at_most, int64_t max_q, int64_t max_k) {
    stream_ = stream_of(q);
    const int n = (int)cu_q.numel() - 1;
    const int r = g_abi.varlen_check(cu_q.const_data_ptr<int32_t>(), cu_k.const_data_ptr<int32_t>(), n, q.size(0), k.size(0), k_at_most,
                                     max_q, max_k, q.device().index(), &ticket_, stream_);
    if (r != FA_ERR_UNSUPPORTED) {
      check(r, "fa_varlen_check");
      open_ = true;
      return;
    }
    // no mapped host memory, or too many tickets out: by a copy
    const Tensor hq = cu_q.cpu(), hk = cu_k.cpu();
    const int32_t *a = hq.const_data_ptr<int32_t>(), *b = hk.const_data_ptr<int32_t>();
    if (a[0] != 0 || b[0] != 0) failed_ |= FA_VARLEN_START;
    for (int i = 0; i < n; ++i) {
      const int64_t lq = (int64_t)a[i + 1] - a[i], lk = (int64_t)b[i + 1] - b[i];
      if (lq < 0 || lk < 0) failed_ |= FA_VARLEN_ORDER;
      if (lq > max_q || lk > max_k) failed_ |= FA_VARLEN_LONGEST;
    }
    if (a[n] != q.size(0) || (k_at_most ? b[n] > k.size(0) : b[n] != k.size(0))) failed_ |= FA_VARLEN_COVER;
    open_ = true;
  }
  // Raises what the values are refused for, once.
  void finish() {
    if (!open_) return;
    open_ = false;
    check(result(), "fa_check_result");
    const char* what = failed_ & FA_VARLEN_START     ? "cu_seqlens arrays must start at zero and contain a batch boundary"
                       : failed_ & FA_VARLEN_ORDER   ? "cu_seqlens arrays must be monotonically non-decreasing"
                       : failed_ & FA_VARLEN_COVER   ? "cu_seqlens arrays must cover the packed q and KV tensors"
                       : failed_ & FA_VARLEN_LONGEST ? "max sequence lengths must cover every packed sequence"
                                                     : nullptr;
    if (what == nullptr) return;
    PyErr_SetString(PyExc_ValueError, what);
    throw python_error();
  }
  ~VarlenCheck() { result(); }     // an exception in between: the ticket is handed in all the same
  VarlenCheck() = default;
  VarlenCheck(const VarlenCheck&) = delete;
  VarlenCheck& operator=(const VarlenCheck&) = delete;

 private:
  int result() {
    if (ticket_ < 0) return FA_OK;
    const int32_t t = ticket_;
    ticket_ = -1;
    uint32_t bad = 0;
    int r;
    {
      pybind11::gil_scoped_release nogil;
      r = g_abi.check_result(t, &bad, stream_);
    }
    failed_ |= bad;
    return r;
  }
  bool open_ = false;              // checks made or under way, the answer not looked at yet
  int32_t ticket_ = -1;
  uint32_t failed_ = 0;
  void* stream_ = nullptr;
};

// in: prepared inputs.  Fills out and (when wanted) lse.
void run_forward(const Params& c, const variable_list& in, bool want_lse, Tensor& out, Tensor& lse, VarlenCheck* values = nullptr) {
  View q, k, v;
  split(c, in, q, k, v);
  const Tensor& t = in[0];
  out = empty_cuda(shape_of(c, q), t.scalar_type(), t.device());
  if (want_lse) lse = empty_cuda(lse_shape(c, q), at::kFloat, t.device());
  fa_attn_args a;
  fill(a, c, t, q, k, v, view_of(out, c.layout, -1, 0), want_lse ? lse.mutable_data_ptr<float>() : nullptr);
  const Tensor bits = dropout_bits(a, t, false);
  if (values != nullptr) values->finish();
  if (bits.defined()) check(g_abi.fwd_bits(&a, bits.const_data_ptr(), stream_of(t)), "fa_fwd_dropout");
  else if (c.layout == kTHD) check(g_abi.varlen_fwd(&a, stream_of(t)), "fa_varlen_fwd");
  else check(g_abi.fwd(&a, stream_of(t)), "fa_fwd");
}

// Gradients of the inputs, in the inputs' own packing.  need[0..2]: dq, dk, dv wanted.
variable_list run_backward(const Params& c, const variable_list& in, const Tensor& out, const Tensor& lse,
                           const Tensor& grad, bool need_dq, bool need_dkdv) {
  View q, k, v;
  split(c, in, q, k, v);
  const Tensor& t = in[0];
  const Tensor dout = prep(grad);
  // rows past cu_seqlens[-1] or past a used length (and padded keys) get no writer: they start from zero
  const bool partial = c.used_q.defined() || c.used_k.defined() || c.k_valid > 0;
  auto alloc = [&](at::IntArrayRef sizes) {
    return partial ? at::zeros(sizes, t.options()) : empty_cuda(sizes, t.scalar_type(), t.device());
  };
  variable_list g(in.size());
  View dq = q, dk = k, dv = v;
  switch (c.packing) {
    case kSeparate:
      if (need_dq) { g[0] = alloc(in[0].sizes()); dq = view_of(g[0], c.layout, -1, 0); }
      if (need_dkdv) {
        g[1] = alloc(in[1].sizes()); dk = view_of(g[1], c.layout, -1, 0);
        g[2] = alloc(in[2].sizes()); dv = view_of(g[2], c.layout, -1, 0);
      }
      break;
    case kQKV:
      g[0] = alloc(in[0].sizes());
      dq = view_of(g[0], c.layout, c.packed_dim, 0);
      dk = view_of(g[0], c.layout, c.packed_dim, 1);
      dv = view_of(g[0], c.layout, c.packed_dim, 2);
      break;
    case kKV:
      if (need_dq) { g[0] = alloc(in[0].sizes()); dq = view_of(g[0], c.layout, -1, 0); }
      if (need_dkdv) {
        g[1] = alloc(in[1].sizes());
        dk = view_of(g[1], c.layout, c.packed_dim, 0);
        dv = view_of(g[1], c.layout, c.packed_dim, 1);
      }
      break;
  }
  Tensor delta = empty_cuda(lse.sizes(), at::kFloat, t.device());
  fa_attn_args a;
  fill(a, c, t, q, k, v, view_of(out, c.layout, -1, 0), lse.data_ptr<float>());
  const View vd = view_of(dout, c.layout, -1, 0);
  a.dout = vd.p;
  set_strides(a.do_stride, vd);
  a.delta = delta.mutable_data_ptr<float>();
  a.dq = dq.p; a.dk = dk.p; a.dv = dv.p;
  set_strides(a.dq_stride, dq); set_strides(a.dk_stride, dk); set_strides(a.dv_stride, dv);
  void* st = stream_of(t);
  check(g_abi.preprocess(&a, st), "fa_bwd_preprocess");
  const Tensor bits = dropout_bits(a, t, true);
  if (bits.defined()) {
    if (need_dq) check(g_abi.bwd_dq_bits(&a, bits.const_data_ptr(), st), "fa_bwd_dq_dropout");
    if (need_dkdv) check(g_abi.bwd_dkdv_bits(&a, bits.const_data_ptr(), st), "fa_bwd_dkdv_dropout");
  } else if (c.layout == kTHD) {
    if (need_dq) check(g_abi.varlen_bwd_dq(&a, st), "fa_varlen_bwd_dq");
    if (need_dkdv) check(g_abi.varlen_bwd_dkdv(&a, st), "fa_varlen_bwd_dkdv");
  } else {
    if (need_dq) check(g_abi.bwd_dq(&a, st), "fa_bwd_dq");
    if (need_dkdv) check(g_abi.bwd_dkdv(&a, st), "fa_bwd_dkdv");
  }
  return g;
}

// Every tensor that the backward reads is a saved variable: one that was changed in place since the forward is
// refused, and the saved-tensor hooks (offloading, checkpointing) see all of them.  Params::bias alone is held as it
// is: expanded over broadcast dimensions, it would be written out in full by a hook that copies.
struct AttnBackward : public Node {
  Params c;                                      // without the tensors of `side`
  std::vector<SavedVariable> in;
  SavedVariable out, lse;
  SavedVariable side[5];                         // cu_q, cu_k, used_q, used_k, alibi

  static std::array<Tensor Params::*, 5> side_members() {
    return {&Params::cu_q, &Params::cu_k, &Params::used_q, &Params::used_k, &Params::alibi};
  }

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);    // against release_variables() of a backward on another thread
    // no gradient came back to the output (a node behind it returned none): the inputs have one of zeros
    const Tensor grad = grads[0].defined() ? grads[0] : input_metadata(0).zeros_like();
    // Unpacked before autograd is switched off: the hook of a checkpointed region runs that region's forward again
    // here, and its nodes have to save what this one saved.
    variable_list x;
    x.reserve(in.size());
    for (auto& s : in) x.push_back(s.unpack());
    const Tensor o = out.unpack(getptr()), l = lse.unpack();
    Params p = c;
    for (size_t i = 0; i < 5; ++i) p.*side_members()[i] = side[i].unpack();
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::CUDAGuard guard(x[0].device());
    bool dq = true, dkdv = true;
    if (p.packing != kQKV) {
      dq = task_should_compute_output(0);
      dkdv = task_should_compute_output(1) || (p.packing == kSeparate && task_should_compute_output(2));
    }
    return run_backward(p, x, o, l, grad, dq, dkdv);
  }
  std::string name() const override { return "FlashAttnBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& s : in) s.reset_data();
    for (auto& s : side) s.reset_data();
    out.reset_data();
    lse.reset_data();
  }
};

// Forward of `in` (1 to 3 tensors by packing) with the autograd node when a gradient is wanted.
// `forward` computes out and lse from the prepared inputs.
template <typename F>
Tensor with_grad(const Params& c, variable_list in, bool want_lse, Tensor& lse, F forward) {
  c10::cuda::CUDAGuard guard(in[0].device());
  auto no_tangent = [](const Tensor& t) {
    TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(/*level=*/0).defined(),
                                "the attention functions have no forward-mode derivative");
  };
  for (const auto& t : in) no_tangent(t);
  no_tangent(c.alibi);
  const bool need = at::GradMode::is_enabled() && torch::autograd::any_variable_requires_grad(in);
  std::shared_ptr<AttnBackward> node;
  if (need) {
    node = std::shared_ptr<AttnBackward>(new AttnBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(in));
  }
  Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    for (auto& t : in) t = prep(t);
    forward(in, need || want_lse, out, lse);
  }
  if (need) {
    torch::autograd::set_history(out, node);
    node->c = c;
    node->in.reserve(in.size());
    for (auto& t : in) node->in.emplace_back(t, false);
    node->out = SavedVariable(out, true);
    node->lse = SavedVariable(lse, false);
    for (size_t i = 0; i < 5; ++i) {
      Tensor& t = node->c.*AttnBackward::side_members()[i];
      node->side[i] = SavedVariable(t, false);
      t.reset();
    }
  }
  return out;
}

// ---------------------------------------------------------------------------------------
// Python entry points (positional arguments only)
// ---------------------------------------------------------------------------------------
struct Args {
  PyObject* const* v;
  Py_ssize_t n, i = 0;
  PyObject* next() {
    TORCH_CHECK(i < n, "missing argument");
    return v[i++];
  }
  Tensor tensor() {
    PyObject* o = next();
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
    return THPVariable_Unpack(o);
  }
  Tensor tensor_or_none() {
    PyObject* o = next();
    if (o == Py_None) return Tensor();
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor or None");
    return THPVariable_Unpack(o);
  }
  int64_t integer() {
    const long long x = PyLong_AsLongLong(next());
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
  }
  double real() {
    const double x = PyFloat_AsDouble(next());
    if (x == -1.0 && PyErr_Occurred()) throw python_error();
    return x;
  }
  bool truth() {
    const int x = PyObject_IsTrue(next());
    if (x < 0) throw python_error();
    return x != 0;
  }
};

void score_params(Args& a, Params& c) {
  c.scale = a.real();
  c.causal = a.truth();
  c.wl = (int)a.integer();
  c.wr = (int)a.integer();
  c.softcap = a.real();
  c.alibi = a.tensor_or_none();
}

variable_list input_list(Args& a, Params& c) {
  c.packing = (Packing)a.integer();
  c.packed_dim = (int)a.integer();
  variable_list in;
  in.push_back(a.tensor());
  for (int i = 1; i < (c.packing == kSeparate ? 3 : c.packing == kKV ? 2 : 1); ++i) in.push_back(a.tensor());
  return in;
}

PyObject* result(const Tensor& out, const Tensor& lse, bool want_lse) {
  if (!want_lse) return THPVariable_Wrap(out);
  PyObject* t = PyTuple_New(2);
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(out));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(lse));
  return t;
}

// dense(packing, packed_dim, inputs.., scale, causal, wl, wr, softcap, alibi, q_pos_offset, impl, head_major,
//       bias, dropout_p, seed, row_stride, want_lse) -> out | (out, lse2)
PyObject* py_dense(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  Params c;
  variable_list in = input_list(a, c);
  score_params(a, c);
  c.q_pos_offset = (int)a.integer();
  c.impl = (int)a.integer();
  c.layout = a.truth() ? kBHSD : kBSHD;
  c.bias = a.tensor_or_none();
  c.dropout_p = a.real();
  c.seed = (uint64_t)a.integer();
  c.row_stride = (int)a.integer();
  const bool want_lse = a.truth();
  Tensor lse;
  Tensor out = with_grad(c, std::move(in), want_lse, lse, [&](const variable_list& x, bool w, Tensor& o, Tensor& l) {
    run_forward(c, x, w, o, l);
  });
  return result(out, lse, want_lse);
  END_HANDLE_TH_ERRORS
}

// varlen(q, k, v, cu_q, cu_k, max_q, max_k, checks, scale, causal, wl, wr, softcap, alibi, impl,
//        dropout_p, seed, row_stride, used_q, used_k, want_lse) -> out | (out, lse2)
// checks: 0 none, 1 the values of cu_seqlens, 2 the same with rows of k and v past the last sequence.  What they are refused for
// comes before anything else that the call is refused for.
PyObject* py_varlen(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  Params c;
  variable_list in;
  for (int i = 0; i < 3; ++i) in.push_back(a.tensor());
  c.layout = kTHD;
  c.cu_q = a.tensor();
  c.cu_k = a.tensor();
  c.max_q = (int)a.integer();
  c.max_k = (int)a.integer();
  const int checks = (int)a.integer();
  VarlenCheck values;
  if (checks != 0) {
    c10::cuda::CUDAGuard guard(in[0].device());
    at::AutoDispatchBelowADInplaceOrView below;
    values.start(in[0], in[1], c.cu_q, c.cu_k, checks == 2, c.max_q, c.max_k);
  }
  try {
    score_params(a, c);
    c.impl = (int)a.integer();
    c.dropout_p = a.real();
    c.seed = (uint64_t)a.integer();
    c.row_stride = (int)a.integer();
    c.used_q = a.tensor_or_none();
    c.used_k = a.tensor_or_none();
    const bool want_lse = a.truth();
    Tensor lse;
    Tensor out = with_grad(c, std::move(in), want_lse, lse, [&](const variable_list& x, bool w, Tensor& o, Tensor& l) {
      run_forward(c, x, w, o, l, &values);
    });
    return result(out, lse, want_lse);
  } catch (python_error& e) {
    e.persist();
    values.finish();
    throw;
  } catch (...) {
    values.finish();
    throw;
  }
  END_HANDLE_TH_ERRORS
}

// varlen_check(q, k, cu_q, cu_k, max_q, max_k, k_at_most): the same checks by themselves
PyObject* py_varlen_check(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  const Tensor q = a.tensor(), k = a.tensor(), cu_q = a.tensor(), cu_k = a.tensor();
  const int64_t max_q = a.integer(), max_k = a.integer();
  const bool k_at_most = a.truth();
  c10::cuda::CUDAGuard guard(q.device());
  at::AutoDispatchBelowADInplaceOrView below;
  VarlenCheck values;
  values.start(q, k, cu_q, cu_k, k_at_most, max_q, max_k);
  values.finish();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// backward(packing, packed_dim, inputs.., out, lse2, dout, layout, cu_q, cu_k, max_q, max_k, scale, causal, wl, wr,
//          softcap, alibi, q_pos_offset, impl, bias, dropout_p, seed, row_stride, used_q, used_k) -> gradients
PyObject* py_backward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  Params c;
  variable_list in = input_list(a, c);
  Tensor out = a.tensor(), lse = a.tensor(), dout = a.tensor();
  c.layout = (Layout)a.integer();
  c.cu_q = a.tensor_or_none();
  c.cu_k = a.tensor_or_none();
  c.max_q = (int)a.integer();
  c.max_k = (int)a.integer();
  score_params(a, c);
  c.q_pos_offset = (int)a.integer();
  c.impl = (int)a.integer();
  c.bias = a.tensor_or_none();
  c.dropout_p = a.real();
  c.seed = (uint64_t)a.integer();
  c.row_stride = (int)a.integer();
  c.used_q = a.tensor_or_none();
  c.used_k = a.tensor_or_none();
  c10::cuda::CUDAGuard guard(in[0].device());
  at::AutoDispatchBelowADInplaceOrView below;
  const variable_list g = run_backward(c, in, out, lse, dout, true, true);
  PyObject* t = PyTuple_New((Py_ssize_t)g.size());
  for (size_t i = 0; i < g.size(); ++i) PyTuple_SET_ITEM(t, (Py_ssize_t)i, THPVariable_Wrap(g[i]));
  return t;
  END_HANDLE_TH_ERRORS
}

// int8(q, k, v, causal, scale, impl, k_valid, q_pos_offset) -> out; fp16 backward (head-major tensors)
PyObject* py_int8(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  Params c;
  variable_list in;
  for (int i = 0; i < 3; ++i) in.push_back(a.tensor());
  c.layout = kBHSD;
  c.causal = a.truth();
  c.scale = a.real();
  const int impl = (int)a.integer();
  c.k_valid = (int)a.integer();
  c.q_pos_offset = (int)a.integer();
  Tensor lse;
  Tensor out = with_grad(c, std::move(in), false, lse, [&](const variable_list& x, bool want_lse, Tensor& o, Tensor& l) {
    const Tensor &q = x[0], &k = x[1], &v = x[2];
    const auto dev = q.device();
    const int64_t D = q.size(3), rows = k.numel() / D;
    void* st = stream_of(q);
    Tensor s_k = empty_cuda({rows}, at::kFloat, dev), k8, q8, s_q;
    o = empty_cuda(q.sizes(), at::kHalf, dev);
    fa_int8_args p;
    memset(&p, 0, sizeof(p));
    p.device = dev.index();
    p.impl = impl;
    p.batch = (int)q.size(0); p.heads = (int)q.size(1); p.seqlen = (int)q.size(2); p.head_dim = (int)D;
    p.q = q.data_ptr(); p.s_k = s_k.data_ptr<float>(); p.v = v.data_ptr();
    p.o = o.data_ptr();
    if (want_lse) {
      l = empty_cuda({q.size(0), q.size(1), q.size(2)}, at::kFloat, dev);
      p.lse2 = l.mutable_data_ptr<float>();
    }
    p.softmax_scale = (float)c.scale;
    p.causal = c.causal;
    p.seqlen_k_valid = c.k_valid;
    p.q_pos_offset = c.q_pos_offset;
    if (const size_t bytes = g_abi.int8_codes16_bytes(&p)) {
      const Tensor codes = empty_cuda({(int64_t)bytes}, at::kByte, dev);
      s_q = empty_cuda({rows}, at::kFloat, dev);
      p.sq_scratch = s_q.data_ptr<float>();
      check(g_abi.fwd_int8_codes16(&p, k.data_ptr(), s_k.data_ptr<float>(), codes.data_ptr(), st), "fa_fwd_int8_codes16");
      return;
    }
    k8 = empty_cuda(k.sizes(), at::kChar, dev);
    check(g_abi.quantize_k(k.data_ptr(), k8.data_ptr<int8_t>(), s_k.data_ptr<float>(), rows, (int)D, dev.index(), st),
          "fa_quantize_k_int8");
    p.k8 = k8.data_ptr<int8_t>();
    if (D == 128 && impl != FA_IMPL_MMA) {
      q8 = empty_cuda(q.sizes(), at::kChar, dev);
      s_q = empty_cuda({rows}, at::kFloat, dev);
      p.q8_scratch = q8.data_ptr<int8_t>();
      p.sq_scratch = s_q.data_ptr<float>();
    }
    check(g_abi.fwd_int8(&p, st), "fa_fwd_int8");
  });
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// Zeroed counters of the split-KV merge, one buffer per (device, stream): calls on a stream run one
// after the other and leave them zero.  At most kCounterBuffers of them are kept (least recently
// used first out; the allocator hands a dropped one out again on the same stream only).
constexpr int kCounterWords = 8192;
constexpr size_t kCounterBuffers = 32;
Tensor decode_counters(const at::Device& dev, cudaStream_t stream) {
  struct Entry {
    int device;
    cudaStream_t stream;
    Tensor words;
  };
  static std::mutex mu;
  static std::list<Entry>* pool = new std::list<Entry>();     // never destroyed: outlives the CUDA context's teardown
  std::lock_guard<std::mutex> lock(mu);
  for (auto it = pool->begin(); it != pool->end(); ++it)
    if (it->device == dev.index() && it->stream == stream) {
      pool->splice(pool->begin(), *pool, it);
      return it->words;
    }
  if (pool->size() >= kCounterBuffers) pool->pop_back();
  pool->push_front(Entry{dev.index(), stream, at::zeros({kCounterWords}, at::TensorOptions().device(dev).dtype(at::kInt))});
  return pool->front().words;
}

// kvcache(q, k_cache, v_cache, k_new, v_new, cos, sin, seqlens, batch_idx, leftpad, block_table, scale, causal, wl, wr,
//         interleaved, alibi, num_splits, checks) -> out, or the mask of the value checks that failed
PyObject* py_kvcache(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  Tensor q = a.tensor(), kc = a.tensor(), vc = a.tensor(), kn = a.tensor_or_none(), vn = a.tensor_or_none();
  Tensor cos = a.tensor_or_none(), sin = a.tensor_or_none(), lens = a.tensor(), idx = a.tensor_or_none();
  Tensor pads = a.tensor_or_none(), table = a.tensor_or_none();
  fa_decode_args p;
  memset(&p, 0, sizeof(p));
  p.softmax_scale = (float)a.real();
  p.causal = a.truth();
  p.window_left = (int)a.integer();
  p.window_right = (int)a.integer();
  p.rotary_interleaved = a.truth();
  Tensor alibi = a.tensor_or_none();
  p.num_splits = (int)a.integer();
  const bool checks = a.truth();

  c10::cuda::CUDAGuard guard(q.device());
  at::AutoDispatchBelowADInplaceOrView below;
  const auto dev = q.device();
  q = prep(q);
  Tensor out = empty_cuda(q.sizes(), q.scalar_type(), dev);
  p.dtype = q.scalar_type() == at::kBFloat16 ? FA_BF16 : FA_F16;
  p.device = dev.index();
  const View vq = view_of(q, kBSHD, -1, 0), vo = view_of(out, kBSHD, -1, 0), vkc = view_of(kc, kBSHD, -1, 0),
             vvc = view_of(vc, kBSHD, -1, 0);
  p.batch = (int)vq.batch; p.seqlen_q = (int)vq.rows; p.heads_q = (int)vq.heads; p.head_dim = (int)vq.dim;
  p.heads_kv = (int)vkc.heads;
  p.q = vq.p; p.o = vo.p;
  set_strides(p.q_stride, vq); set_strides(p.o_stride, vo);
  p.k_cache = vkc.p; p.v_cache = vvc.p;
  set_strides(p.kc_stride, vkc); set_strides(p.vc_stride, vvc);
  p.page_size = (int)vkc.rows; p.num_pages = (int)vkc.batch;
  if (table.defined()) {
    p.block_table = table.const_data_ptr<int32_t>();
    p.block_table_stride = (int)table.size(1);       // contiguous
  }
  if (idx.defined()) p.cache_batch_idx = idx.const_data_ptr<int32_t>();
  p.cache_seqlens = lens.const_data_ptr<int32_t>();
  if (pads.defined()) p.cache_leftpad = pads.const_data_ptr<int32_t>();
  if (kn.defined()) {
    kn = prep(kn);
    vn = prep(vn);
    const View vkn = view_of(kn, kBSHD, -1, 0), vvn = view_of(vn, kBSHD, -1, 0);
    p.k_new = vkn.p; p.v_new = vvn.p;
    set_strides(p.kn_stride, vkn); set_strides(p.vn_stride, vvn);
    p.seqlen_new = (int)vkn.rows;
  }
  if (cos.defined()) {
    p.rotary_cos = cos.data_ptr(); p.rotary_sin = sin.data_ptr();
    p.rotary_dim = (int)cos.size(1) * 2;
    p.rotary_seqlen = (int)cos.size(0);
  }
  if (alibi.defined()) p.alibi_slopes = alibi.const_data_ptr<float>();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  Tensor ws, ctr;
  if (const size_t need = checks ? g_abi.decode_checked_workspace(&p) : g_abi.decode_workspace(&p)) {
    ws = empty_cuda({(int64_t)need}, at::kByte, dev);
    p.workspace = ws.data_ptr();
    p.workspace_bytes = need;
    const int words = g_abi.decode_counters(&p);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (words <= kCounterWords && cudaStreamIsCapturing(st, &cap) == cudaSuccess) {
      // a captured call keeps counters of its own, zeroed inside the graph
      ctr = cap == cudaStreamCaptureStatusNone ? decode_counters(dev, st)
                                               : at::zeros({words}, at::TensorOptions().device(dev).dtype(at::kInt));
      p.counters = reinterpret_cast<uint32_t*>(ctr.data_ptr<int32_t>());
      p.num_counters = (int)ctr.numel();
    }
  }
  uint32_t failed = 0;
  int status;
  if (checks) {
    pybind11::gil_scoped_release nogil;
    status = g_abi.decode_checked(&p, &failed, st);
  } else {
    status = g_abi.decode(&p, st);
  }
  check(status, "fa_decode_paged");
  if (failed) return PyLong_FromUnsignedLong(failed);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// init({name: address}, check): addresses of the C functions, once per loaded library
PyObject* py_init(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Args a{args, n};
  PyObject* addr = a.next();
  PyObject* chk = a.next();
  auto get = [&](const char* name) {
    PyObject* o = PyDict_GetItemString(addr, name);
    TORCH_CHECK(o != nullptr, "no address for ", name);
    void* p = PyLong_AsVoidPtr(o);
    if (p == nullptr && PyErr_Occurred()) throw python_error();
    return p;
  };
  g_abi.fwd = (AttnFn)get("fa_fwd");
  g_abi.varlen_fwd = (AttnFn)get("fa_varlen_fwd");
  g_abi.preprocess = (AttnFn)get("fa_bwd_preprocess");
  g_abi.bwd_dq = (AttnFn)get("fa_bwd_dq");
  g_abi.bwd_dkdv = (AttnFn)get("fa_bwd_dkdv");
  g_abi.varlen_bwd_dq = (AttnFn)get("fa_varlen_bwd_dq");
  g_abi.varlen_bwd_dkdv = (AttnFn)get("fa_varlen_bwd_dkdv");
  g_abi.bits_bytes = (decltype(g_abi.bits_bytes))get("fa_dropout_bits_bytes");
  g_abi.bits = (decltype(g_abi.bits))get("fa_dropout_bits");
  g_abi.fwd_bits = (decltype(g_abi.fwd_bits))get("fa_fwd_dropout");
  g_abi.bwd_dq_bits = (decltype(g_abi.bwd_dq_bits))get("fa_bwd_dq_dropout");
  g_abi.bwd_dkdv_bits = (decltype(g_abi.bwd_dkdv_bits))get("fa_bwd_dkdv_dropout");
  g_abi.quantize_k = (decltype(g_abi.quantize_k))get("fa_quantize_k_int8");
  g_abi.fwd_int8 = (decltype(g_abi.fwd_int8))get("fa_fwd_int8");
  g_abi.int8_codes16_bytes = (decltype(g_abi.int8_codes16_bytes))get("fa_int8_codes16_bytes");
  g_abi.fwd_int8_codes16 = (decltype(g_abi.fwd_int8_codes16))get("fa_fwd_int8_codes16");
  g_abi.varlen_check = (decltype(g_abi.varlen_check))get("fa_varlen_check");
  g_abi.check_result = (decltype(g_abi.check_result))get("fa_check_result");
  g_abi.decode = (decltype(g_abi.decode))get("fa_decode_paged");
  g_abi.decode_checked = (decltype(g_abi.decode_checked))get("fa_decode_paged_checked");
  g_abi.decode_counters = (decltype(g_abi.decode_counters))get("fa_decode_counters");
  g_abi.decode_workspace = (decltype(g_abi.decode_workspace))get("fa_decode_workspace_bytes");
  g_abi.decode_checked_workspace = (decltype(g_abi.decode_checked_workspace))get("fa_decode_checked_workspace_bytes");
  Py_INCREF(chk);
  Py_XDECREF(g_abi.check);
  g_abi.check = chk;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL
PyMethodDef g_methods[] = {
    {"init", FAST(py_init), "addresses of the C ABI functions and the status check"},
    {"dense", FAST(py_dense), "dense attention"},
    {"varlen", FAST(py_varlen), "packed variable-length attention"},
    {"varlen_check", FAST(py_varlen_check), "value checks of a packed call"},
    {"backward", FAST(py_backward), "gradients from a forward's output and LSE"},
    {"kvcache", FAST(py_kvcache), "append to a KV cache and attend to it"},
    {"int8", FAST(py_int8), "INT8 scores forward"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_fa_host", "host path of the attention kernels", -1, g_methods};

}  // namespace

PyMODINIT_FUNC PyInit__fa_host(void) {
  PyObject* m = PyModule_Create(&g_module);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", FA_TORCH) != 0) Py_CLEAR(m);
  return m;
}
