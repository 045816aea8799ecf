// The host path of the public functions in native code: argument checks, output and workspace
// allocation, autograd and the call into libspsattn.so, as one CPython extension
// (sps_b200._native).  A small attention call is bound by its host path, not by its kernels: the
// same steps in Python with ctypes took 32-38 us per forward call and about 40 us more per
// backward, against 8-13 us of kernel time.  Functions take positional arguments only and raise what
// their Python wrappers document; nothing here synchronises.  Whatever may launch or allocate runs without
// the interpreter lock (a launch blocks while its stream's queue is full, and what empties the queue may
// need another Python thread).
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime_api.h>

#include <algorithm>
#include <cmath>
#include <limits>
#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/spsattn.h"

namespace {

using at::Tensor;
using c10::optional;

// ------------------------------------------------------------------------------------- errors

struct PyError {
  PyObject* type;
  std::string message;
};

PyObject* g_spsattn_error = nullptr;   // sps_b200._lib.SpsAttnError
PyObject* g_packed_type = nullptr;     // sps_b200.decode.PackedKVSegment

[[noreturn]] void fail(PyObject* type, const std::string& message) { throw PyError{type, message}; }

// As the exception that torch carries through its own code; the interpreter lock is held.
[[noreturn]] void raise(const PyError& e) {
  PyErr_SetString(e.type ? e.type : PyExc_RuntimeError, e.message.c_str());
  python_error err;
  err.persist();
  throw err;
}

void require(bool ok, const char* message) {
  if (!ok) fail(PyExc_AssertionError, message);
}

// A negative or CUDA error code of the C ABI as the package's exception.
void check_rc(int rc, const char* what) {
  if (rc == 0) return;
  fail(g_spsattn_error, std::string(what) + " failed: " + spsattn_strerror(rc) + " (code " + std::to_string(rc) + ")");
}

// ------------------------------------------------------------------------------------- arguments

const Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, std::string(name) + " must be a tensor, got " + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}

optional<Tensor> optional_tensor(PyObject* o, const char* name) {
  if (o == Py_None) return c10::nullopt;
  return tensor_arg(o, name);
}

// int(o); with `saturate`, a value past the range of 64 bits is its end (a window longer than any row)
long long int_arg(PyObject* o, bool saturate = false) {
  PyObject* whole = PyLong_CheckExact(o) ? Py_NewRef(o) : PyNumber_Long(o);
  if (!whole) throw python_error();
  int past = 0;
  const long long v = PyLong_AsLongLongAndOverflow(whole, &past);
  Py_DECREF(whole);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  if (past == 0) return v;
  if (!saturate) fail(PyExc_OverflowError, "the number does not fit 64 bits");
  return past > 0 ? std::numeric_limits<long long>::max() : std::numeric_limits<long long>::min();
}

double float_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}

bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}

at::ScalarType dtype_arg(PyObject* o) {
  if (!THPDtype_Check(o)) fail(PyExc_TypeError, "expected a torch.dtype");
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

struct Unlocked {         // the interpreter lock is given up while one of these lives
  PyThreadState* state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

template <typename F>
auto unlocked(F&& f) {
  const Unlocked u;
  return f();
}

struct PyRef {            // owned reference
  PyObject* p;
  explicit PyRef(PyObject* o) : p(o) {
    if (!p) throw python_error();
  }
  ~PyRef() { Py_DECREF(p); }
  PyRef(const PyRef&) = delete;
};

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return SPSATTN_DTYPE_BF16;
  if (t.scalar_type() == at::kHalf) return SPSATTN_DTYPE_FP16;
  fail(PyExc_TypeError, std::string("sps_b200 attention computes in bf16 or fp16, got ") + at::toString(t.scalar_type()));
}

// ------------------------------------------------------------------------------------- status word

constexpr int kMaxDevices = 64;

// One int32 word of SPSATTN_STATUS bits per device; lives as long as the process.
const Tensor& status_word(int device) {
  static std::once_flag once[kMaxDevices];
  static Tensor* words[kMaxDevices];
  TORCH_CHECK(device >= 0 && device < kMaxDevices, "device index out of range");
  std::call_once(once[device], [device] {
    words[device] = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device)));
  });
  return *words[device];
}

int* status_ptr(const Tensor& like) { return status_word(like.get_device()).data_ptr<int>(); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor empty_bytes(size_t n, const Tensor& like) {
  return at::detail::empty_cuda({static_cast<int64_t>(n)}, at::kByte, like.device(), c10::nullopt);
}

// ------------------------------------------------------------------------------------- prefill

bool supported_head_dim(int64_t d) { return d == 16 || d == 32 || d == 64 || d == 128 || d == 256; }
bool backward_head_dim(int64_t d) { return d == 64 || d == 128; }

// rows of D contiguous elements, 16-byte aligned, batch / head / row strides multiples of 8
bool addressable(const Tensor& t) {
  const int64_t d = t.size(3);
  if (t.stride(3) != 1 || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u)) return false;
  for (int i = 0; i < 3; ++i)
    if (t.stride(i) % 8 || t.stride(i) < d) return false;
  return true;
}

// [B, H, N, D] result: token-major (what the caller's transpose(1, 2).contiguous() wants) when
// the operand is, else dense
Tensor empty_like_layout(const Tensor& x) {
  const int64_t b = x.size(0), h = x.size(1), n = x.size(2), d = x.size(3);
  if (x.stride(2) > x.stride(1))
    return at::detail::empty_strided_cuda({b, h, n, d}, {n * h * d, d, h * d, 1}, x.scalar_type(), x.device());
  return at::detail::empty_cuda({b, h, n, d}, x.scalar_type(), x.device(), c10::nullopt);
}

struct MaskArgs {
  double sm_scale;
  int64_t parity, temporary_window, persistent_window, flags;
  bool has_persistent_window;

  int temporary(int64_t n) const { return (int)std::max<int64_t>(-1, std::min(temporary_window, n)); }
  int persistent(int64_t n) const {
    return has_persistent_window ? (int)std::max<int64_t>(-1, std::min(persistent_window, n)) : SPSATTN_NO_WINDOW;
  }
};

struct DocArgs {
  Tensor keep;
  const void* ptr = nullptr;
  int is_i64 = 0;
  int64_t stride_b = 0, stride_t = 0;

  DocArgs(const optional<Tensor>& ids, int64_t batch, int64_t rows, const Tensor& like) {
    if (!ids.has_value()) return;
    keep = *ids;
    require(keep.dim() == 2 && keep.size(0) == batch && keep.size(1) == rows, "document ids must be [B, N]");
    require(keep.is_cuda() && keep.device() == like.device(), "document ids must be on the device of the operands");
    if (keep.scalar_type() != at::kLong && keep.scalar_type() != at::kInt) keep = keep.to(at::kLong);
    ptr = keep.data_ptr();
    is_i64 = keep.scalar_type() == at::kLong;
    stride_b = keep.stride(0);
    stride_t = keep.stride(1);
  }
};

struct Forward {
  Tensor o, lse, ws;       // ws: what the call found out about the documents (undefined without ids)
};

Forward prefill_forward(Tensor q, Tensor k, Tensor v, const MaskArgs& m, const optional<Tensor>& docs, bool return_lse,
                        const optional<Tensor>& out) {
  if (!q.is_cuda()) fail(PyExc_RuntimeError, "sps_b200 attention needs CUDA tensors; there is no CPU path");
  if (q.dim() != 4) fail(PyExc_ValueError, "q must be [B, H, N, D]");
  require(k.sizes() == q.sizes() && v.sizes() == q.sizes(), "q, k, v must have the same shape");
  require(k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(), "q, k, v must have the same dtype");
  const int64_t b = q.size(0), h = q.size(1), n = q.size(2), d = q.size(3);
  require(supported_head_dim(d), "head_dim must be one of (16, 32, 64, 128, 256)");
  if (m.parity != SPSATTN_PARITY_NONE) require(n % 2 == 0, "Expected doubled sequence length (2T).");
  const int dt = dtype_code(q);
  // the tensor-core kernels read any layout whose rows are contiguous (the transposed views of
  // token-major projections that the reference's modules pass); only what they cannot address is
  // copied, where the reference copies always (triton_sps_flash_attention.py:504-506)
  for (Tensor* x : {&q, &k, &v})
    if (!addressable(*x)) *x = x->contiguous();
  const DocArgs ids(docs, b, n, q);
  const c10::cuda::CUDAGuard guard(q.device());
  Forward r;
  r.o = out.has_value() ? *out : empty_like_layout(q);
  if (return_lse) r.lse = at::detail::empty_cuda({b, h, n}, at::kFloat, q.device(), c10::nullopt);
  const size_t ws_bytes = ids.ptr ? spsattn_prefill_workspace_bytes(b, h, n, d) : 0;
  if (ws_bytes) r.ws = empty_bytes(ws_bytes, q);
  const int rc = spsattn_prefill_fwd_strided(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), r.o.data_ptr(), return_lse ? r.lse.data_ptr<float>() : nullptr,
      q.strides().data(), k.strides().data(), v.strides().data(), r.o.strides().data(), ids.ptr, ids.is_i64, ids.stride_b,
      ids.stride_t, b, h, n, d, dt, (float)m.sm_scale, (int)m.parity, m.temporary(n), m.persistent(n), (int)m.flags,
      ws_bytes ? r.ws.data_ptr() : nullptr, ws_bytes, status_ptr(q), stream_of(q));
  check_rc(rc, "spsattn_prefill_fwd");
  return r;
}

struct Gradients {
  Tensor dq, dk, dv;
};

Gradients prefill_backward(Tensor q, Tensor k, Tensor v, Tensor o, Tensor lse, Tensor d_o, const MaskArgs& m,
                           const optional<Tensor>& docs, const Tensor& forward_ws = Tensor()) {
  const int64_t b = q.size(0), h = q.size(1), n = q.size(2), d = q.size(3);
  if (!backward_head_dim(d))
    fail(PyExc_RuntimeError, "the backward kernels cover head_dim (64, 128), got " + std::to_string(d));
  const int dt = dtype_code(q);
  if (d_o.scalar_type() != q.scalar_type()) d_o = d_o.to(q.scalar_type());
  // operands are read where they lie when their rows are addressable; the reference copies all
  // five (triton_sps_flash_attention.py:629-633)
  for (Tensor* x : {&q, &k, &v, &o, &d_o})
    if (!addressable(*x)) *x = x->contiguous();
  if (!lse.is_contiguous()) lse = lse.contiguous();
  require(lse.dim() == 3 && lse.size(0) == b && lse.size(1) == h && lse.size(2) == n && lse.scalar_type() == at::kFloat,
          "lse must be fp32 [B, H, N]");
  const DocArgs ids(docs, b, n, q);
  const c10::cuda::CUDAGuard guard(q.device());
  Gradients g{empty_like_layout(q), empty_like_layout(k), empty_like_layout(v)};
  int64_t strides[24];
  int at_ = 0;
  for (const Tensor* x : {&q, &k, &v, &o, &d_o, &g.dq, &g.dk, &g.dv})
    for (int i = 0; i < 3; ++i) strides[at_++] = x->stride(i);
  const size_t ws_bytes = spsattn_prefill_bwd_workspace_bytes(b, h, n, d);
  const Tensor ws = empty_bytes(ws_bytes, q);
  const int rc = spsattn_prefill_bwd_after(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), d_o.data_ptr(), lse.data_ptr<float>(), g.dq.data_ptr(),
      g.dk.data_ptr(), g.dv.data_ptr(), strides, ids.ptr, ids.is_i64, ids.stride_b, ids.stride_t, b, h, n, d, dt,
      (float)m.sm_scale, (int)m.parity, m.temporary(n), m.persistent(n), (int)m.flags,
      forward_ws.defined() ? forward_ws.data_ptr() : nullptr, ws.data_ptr(), ws_bytes,
      status_ptr(q), stream_of(q));
  check_rc(rc, "spsattn_prefill_bwd");
  return g;
}

// Differentiable prefill attention (head_dim 64 and 128), once differentiable.
struct PrefillAttention : public torch::autograd::Function<PrefillAttention> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v,
                        const MaskArgs& m, const optional<Tensor>& docs) {
    Forward r = prefill_forward(q, k, v, m, docs, true, c10::nullopt);
    ctx->save_for_backward({q, k, v, r.o, r.lse});
    if (docs.has_value()) ctx->saved_data["docs"] = *docs;
    // not a saved tensor: hooks on those may give back other values (compressed ones, say), and these
    // are row indices
    if (r.ws.defined()) ctx->saved_data["runs"] = r.ws;
    ctx->saved_data["scale"] = m.sm_scale;
    ctx->saved_data["mask"] = std::vector<int64_t>{m.parity, m.temporary_window, m.persistent_window, m.flags,
                                                   (int64_t)m.has_persistent_window};
    return r.o;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto mask = ctx->saved_data["mask"].toIntVector();
    MaskArgs m{ctx->saved_data["scale"].toDouble(), mask[0], mask[1], mask[2], mask[3], mask[4] != 0};
    auto kept = [ctx](const char* name) {
      const auto it = ctx->saved_data.find(name);
      return it == ctx->saved_data.end() ? optional<Tensor>() : it->second.toTensor();
    };
    const optional<Tensor> docs = kept("docs"), runs = kept("runs");
    torch::autograd::variable_list out(5);
    try {
      const at::AutoGradMode no_grad(false);
      Gradients g = prefill_backward(saved[0], saved[1], saved[2], saved[3], saved[4], grads[0].detach(), m, docs,
                                     runs.value_or(Tensor()));
      out[0] = g.dq;
      out[1] = g.dk;
      out[2] = g.dv;
    } catch (const PyError& e) {          // runs on an autograd thread: hand the exception over
      pybind11::gil_scoped_acquire gil;
      raise(e);
    }
    if (at::GradMode::is_enabled() && grads[0].requires_grad()) {
      auto twice = std::make_shared<torch::autograd::DelayedError>(
          "trying to differentiate twice a function that is once differentiable", 3);
      auto marked = (*twice)({out[0], out[1], out[2]});
      for (int i = 0; i < 3; ++i) out[i] = marked[i];
    }
    return out;
  }
};

bool needs_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->requires_grad()) return true;
  return false;
}

void forward_only(std::initializer_list<const Tensor*> ts) {
  if (needs_grad(ts))
    fail(PyExc_RuntimeError,
         "this sps_b200 call is forward only: call it under torch.no_grad() / inference_mode(), or detach the inputs "
         "(backward kernels exist for prefill attention with head_dim 64 and 128 only)");
}

MaskArgs mask_args(PyObject* const* a) {     // sm_scale, parity, temporary, persistent or None, flags
  MaskArgs m;
  m.sm_scale = float_arg(a[0]);
  m.parity = int_arg(a[1]);
  m.temporary_window = int_arg(a[2], true);
  m.has_persistent_window = a[3] != Py_None;
  m.persistent_window = m.has_persistent_window ? int_arg(a[3], true) : 0;
  m.flags = int_arg(a[4]);
  return m;
}

// prefill(q, k, v, sm_scale, parity, temporary, persistent, flags, docs, return_lse, out)
PyObject* prefill_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 11) fail(PyExc_TypeError, "prefill takes 11 arguments");
  const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k"), &v = tensor_arg(a[2], "v");
  const MaskArgs m = mask_args(a + 3);
  const optional<Tensor> docs = optional_tensor(a[8], "document ids");
  const bool return_lse = bool_arg(a[9]);
  const optional<Tensor> out = optional_tensor(a[10], "out");
  if (needs_grad({&q, &k, &v})) {
    if (q.dim() != 4 || !backward_head_dim(q.size(3)) || return_lse || out.has_value()) forward_only({&q, &k, &v});
    return THPVariable_Wrap(unlocked([&] { return PrefillAttention::apply(q, k, v, m, docs); }));
  }
  Forward r = unlocked([&] { return prefill_forward(q, k, v, m, docs, return_lse, out); });
  if (!return_lse) return out.has_value() ? Py_NewRef(a[10]) : THPVariable_Wrap(std::move(r.o));
  PyRef o(out.has_value() ? Py_NewRef(a[10]) : THPVariable_Wrap(std::move(r.o)));
  PyRef lse(THPVariable_Wrap(std::move(r.lse)));
  return PyTuple_Pack(2, o.p, lse.p);
}

// prefill_backward(q, k, v, o, lse, d_o, sm_scale, parity, temporary, persistent, flags, docs)
PyObject* prefill_backward_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 12) fail(PyExc_TypeError, "prefill_backward takes 12 arguments");
  const Tensor& q = tensor_arg(a[0], "q");
  if (q.dim() != 4) fail(PyExc_ValueError, "q must be [B, H, N, D]");
  const Tensor &k = tensor_arg(a[1], "k"), &v = tensor_arg(a[2], "v"), &o = tensor_arg(a[3], "o"),
               &lse = tensor_arg(a[4], "lse"), &d_o = tensor_arg(a[5], "d_o");
  const MaskArgs m = mask_args(a + 6);
  const optional<Tensor> docs = optional_tensor(a[11], "document ids");
  Gradients g = unlocked([&] { return prefill_backward(q, k, v, o, lse, d_o, m, docs); });
  PyRef dq(THPVariable_Wrap(std::move(g.dq))), dk(THPVariable_Wrap(std::move(g.dk))), dv(THPVariable_Wrap(std::move(g.dv)));
  return PyTuple_Pack(3, dq.p, dk.p, dv.p);
}

// ------------------------------------------------------------------------------------- decode

// Records and completion tickets of the single-launch decode, kept per (device, stream): calls on
// one stream are ordered, and the kernel leaves its tickets at zero.  Bounded: past kMaxPools
// streams all buffers go back to the allocator, which hands them out again in stream order.
struct DecodePool {
  Tensor records, tickets;
};
constexpr size_t kMaxPools = 32;
std::mutex g_pool_mutex;

DecodePool decode_pool(const Tensor& like, void* stream, size_t record_bytes, size_t ticket_bytes) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(reinterpret_cast<cudaStream_t>(stream), &capturing);
  const auto bytes = like.options().dtype(at::kByte);
  if (capturing != cudaStreamCaptureStatusNone)     // memory of a graph's private pool must not outlive the capture here
    return {empty_bytes(record_bytes, like), at::zeros({(int64_t)ticket_bytes}, bytes)};
  static auto* pools = new std::unordered_map<uint64_t, DecodePool>();
  const uint64_t key = (uint64_t)reinterpret_cast<uintptr_t>(stream) * kMaxDevices + like.get_device();
  const std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (pools->size() >= kMaxPools && !pools->count(key)) pools->clear();
  DecodePool& p = (*pools)[key];
  if (!p.tickets.defined() || (size_t)p.tickets.numel() < ticket_bytes)
    p.tickets = at::zeros({(int64_t)std::max<size_t>(ticket_bytes, 16384)}, bytes);
  if (!p.records.defined() || (size_t)p.records.numel() < record_bytes) p.records = empty_bytes(record_bytes, like);
  return p;
}

struct Interned {
  PyObject *k, *v, *lengths, *max_len_cap, *seq_offset, *head_stride, *row_stride, *max_rows;
};
const Interned& names() {
  static const Interned s = {
      PyUnicode_InternFromString("k"),           PyUnicode_InternFromString("v"),
      PyUnicode_InternFromString("lengths"),     PyUnicode_InternFromString("max_len_cap"),
      PyUnicode_InternFromString("seq_offset"),  PyUnicode_InternFromString("head_stride"),
      PyUnicode_InternFromString("row_stride"),  PyUnicode_InternFromString("max_rows")};
  return s;
}

Tensor attr_tensor(PyObject* o, PyObject* name) {
  const PyRef r(PyObject_GetAttr(o, name));
  return tensor_arg(r.p, PyUnicode_AsUTF8(name));
}

long long attr_int(PyObject* o, PyObject* name) {
  const PyRef r(PyObject_GetAttr(o, name));
  return int_arg(r.p);
}

constexpr int kSegmentLimit = 16, kExtraLimit = 16;    // beyond the library's own limits, which it checks itself

struct DecodeCall {
  Tensor q;
  std::vector<Tensor> keep;
  spsattn_segment segs[kSegmentLimit];
  spsattn_extra extras[kExtraLimit];
  int n_segs = 0, n_extras = 0;
  int64_t s, nq, h, d;

  explicit DecodeCall(const Tensor& q_) : q(q_) {
    if (!q.is_cuda()) fail(PyExc_RuntimeError, "CUDA tensors are required for segmented decode attention");
    if (q.dim() != 4) fail(PyExc_ValueError, "q must be [S, nq, H, D]");
    forward_only({&q});
    s = q.size(0), nq = q.size(1), h = q.size(2), d = q.size(3);
    if (!q.is_contiguous()) q = unlocked([&] { return q.contiguous(); });
    dtype_code(q);
    keep.reserve(16);
  }

  void add_segment(PyObject* seg, unsigned mask) {
    const Interned& nm = names();
    if (n_segs >= kSegmentLimit) fail(PyExc_RuntimeError, "too many segments");
    spsattn_segment& st = segs[n_segs];
    st = spsattn_segment{};
    const Tensor k = attr_tensor(seg, nm.k), v = attr_tensor(seg, nm.v);
    forward_only({&k, &v});
    Tensor lengths = attr_tensor(seg, nm.lengths);
    if (lengths.device() != q.device()) fail(PyExc_RuntimeError, "Segment lengths must live on the same device as query");
    if (lengths.scalar_type() != at::kLong || !lengths.is_contiguous())
      lengths = unlocked([&] { return lengths.to(at::kLong).contiguous(); });
    const int packed = g_packed_type ? PyObject_IsInstance(seg, g_packed_type) : 0;
    if (packed < 0) throw python_error();
    if (packed) {
      Tensor off = attr_tensor(seg, nm.seq_offset);
      if (off.scalar_type() != at::kLong || !off.is_contiguous()) off = unlocked([&] { return off.to(at::kLong).contiguous(); });
      st.seq_offset = off.data_ptr<int64_t>();
      keep.push_back(std::move(off));
      st.head_stride = attr_int(seg, nm.head_stride);
      st.row_stride = attr_int(seg, nm.row_stride);
      st.max_rows = (int)attr_int(seg, nm.max_rows);
    } else {
      if (k.dim() != 4 || v.dim() != 4) fail(PyExc_RuntimeError, "Segment K/V tensors must be rank-4 [B,H,T,D]");
      if (k.sizes() != v.sizes()) fail(PyExc_RuntimeError, "Segment K/V shapes differ");
      if (k.size(0) != s || k.size(1) != h || k.size(3) != d)
        fail(PyExc_RuntimeError, "Segment K/V tensors must match query batch/head/head_dim, got " +
                                     c10::str(k.sizes()) + " for query " + c10::str(q.sizes()));
      if (!k.is_cuda() || !v.is_cuda()) fail(PyExc_RuntimeError, "Segment K/V tensors must be CUDA tensors");
      if (!k.is_contiguous() || !v.is_contiguous()) fail(PyExc_RuntimeError, "Segment K/V tensors must be contiguous");
      const int64_t max_t = k.size(2);
      st.seq_stride = h * max_t * d;
      st.head_stride = max_t * d;
      st.row_stride = d;
      int64_t scan = max_t;                    // decode_attention.py:381-390
      if (max_t > 0) {
        const PyRef cap(PyObject_GetAttr(seg, nm.max_len_cap));
        if (cap.p != Py_None) {
          const long long c = int_arg(cap.p, true);
          if (c < 0) fail(PyExc_ValueError, "KVSegment.max_len_cap must be non-negative, got " + std::to_string(c));
          scan = std::max<int64_t>(1, std::min<int64_t>(max_t, c));
        }
      }
      st.max_rows = (int)scan;
    }
    if (st.max_rows > 0 && k.scalar_type() != q.scalar_type())
      fail(PyExc_RuntimeError, std::string("Segment dtype ") + at::toString(k.scalar_type()) +
                                   " differs from the attention dtype " + at::toString(q.scalar_type()));
    st.k = k.data_ptr();
    st.v = v.data_ptr();
    st.lengths = lengths.data_ptr<int64_t>();
    st.lengths_per_head = lengths.dim() == 2;
    st.query_mask = mask;
    // the caches too: without the lock nothing else holds the segment's attributes to the launch
    keep.push_back(std::move(lengths));
    keep.push_back(k);
    keep.push_back(v);
    ++n_segs;
  }

  void add_extra(Tensor k, Tensor v, unsigned mask) {
    if (n_extras >= kExtraLimit) fail(PyExc_RuntimeError, "too many extra entries");
    if (!k.is_cuda() || !v.is_cuda()) fail(PyExc_RuntimeError, "Current-token K/V tensors must be CUDA tensors");
    forward_only({&k, &v});
    for (Tensor* x : {&k, &v}) {
      if (x->dim() != 3 || x->size(0) != s || x->size(1) != h || x->size(2) != d)
        fail(PyExc_RuntimeError, "Current-token K/V tensors must have shape " + c10::str(at::IntArrayRef({s, h, d})) +
                                     ", got " + c10::str(x->sizes()));
      if (x->scalar_type() != q.scalar_type() || !x->is_contiguous())
        *x = unlocked([&] { return x->to(q.scalar_type()).contiguous(); });
    }
    spsattn_extra& e = extras[n_extras++];
    e = spsattn_extra{};
    e.k = k.data_ptr();
    e.v = v.data_ptr();
    e.query_mask = mask;
    keep.push_back(std::move(k));
    keep.push_back(std::move(v));
  }

  Tensor launch(double scale) {
    const Unlocked u;
    const c10::cuda::CUDAGuard guard(q.device());
    void* stream = stream_of(q);
    Tensor out = at::detail::empty_cuda({s, nq, h, d}, at::kFloat, q.device(), c10::nullopt);
    const size_t records = spsattn_decode_workspace_bytes(s, h, d, nq, segs, n_segs);
    const size_t tickets = ((size_t)s * h + s) * sizeof(int);
    const DecodePool pool = decode_pool(q, stream, records, tickets);
    const int rc = spsattn_decode_step_tickets(
        q.data_ptr(), (int)nq, out.data_ptr(), SPSATTN_DTYPE_FP32, segs, n_segs, extras, n_extras, nullptr, s, h, d,
        dtype_code(q), (float)scale, pool.records.data_ptr(), (size_t)pool.records.numel(),
        reinterpret_cast<int*>(pool.tickets.data_ptr()), (size_t)pool.tickets.numel(), status_ptr(q), stream);
    check_rc(rc, "spsattn_decode_step");
    return out;
  }
};

// a list or tuple as its items (borrowed), without a copy when it is one already
struct Items {
  PyRef seq;
  Py_ssize_t n;
  explicit Items(PyObject* o) : seq(PySequence_Fast(o, "expected a sequence")), n(PySequence_Fast_GET_SIZE(seq.p)) {}
  PyObject* operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(seq.p, i); }
};

// decode(q, segments, extras, segment_query_masks or None, sm_scale or None)
PyObject* decode_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 5) fail(PyExc_TypeError, "decode takes 5 arguments");
  DecodeCall call(tensor_arg(a[0], "q"));
  const Items segs(a[1]), extras(a[2]);
  if (a[3] == Py_None) {
    for (Py_ssize_t i = 0; i < segs.n; ++i) call.add_segment(segs[i], 0xFF);
  } else {
    const Items masks(a[3]);
    if (masks.n < segs.n) fail(PyExc_IndexError, "one query mask per segment is needed");
    for (Py_ssize_t i = 0; i < segs.n; ++i) call.add_segment(segs[i], (unsigned)int_arg(masks[i]));
  }
  for (Py_ssize_t i = 0; i < extras.n; ++i) {
    const Items e(extras[i]);
    if (e.n != 3) fail(PyExc_ValueError, "an extra entry is (k, v, query_mask)");
    call.add_extra(tensor_arg(e[0], "extra k"), tensor_arg(e[1], "extra v"), (unsigned)int_arg(e[2]));
  }
  return THPVariable_Wrap(call.launch(a[4] == Py_None ? 1.0 / std::sqrt((double)call.d) : float_arg(a[4])));
}

// decode_q2(q, segments, normal_k, normal_v, predict_k, predict_v, attn_dtype)
PyObject* decode_q2_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 7) fail(PyExc_TypeError, "decode_q2 takes 7 arguments");
  Tensor q = tensor_arg(a[0], "q");
  if (!q.is_cuda()) fail(PyExc_RuntimeError, "CUDA tensors are required for SPS-family cached generation attention");
  const Items segs(a[1]);
  if (segs.n > 2)
    fail(PyExc_RuntimeError, "SPS-family q2 attention supports at most 2 segments, got " + std::to_string(segs.n));
  if (q.dim() != 4 || q.size(1) != 2)
    fail(PyExc_RuntimeError, "Expected q_Bx2xHxD slot dimension to be 2, got " + c10::str(q.sizes()));
  if (q.size(3) <= 0 || q.size(3) > 256)
    fail(PyExc_RuntimeError, "Unsupported SPS-family q2 attention head_dim=" + std::to_string(q.size(3)));
  const at::ScalarType dt = dtype_arg(a[6]);
  if (q.scalar_type() != dt) q = unlocked([&] { return q.to(dt); });
  DecodeCall call(q);
  for (Py_ssize_t i = 0; i < segs.n; ++i) call.add_segment(segs[i], 0xFF);
  call.add_extra(tensor_arg(a[2], "normal k"), tensor_arg(a[3], "normal v"), 3);
  call.add_extra(tensor_arg(a[4], "predict k"), tensor_arg(a[5], "predict v"), 2);
  return THPVariable_Wrap(call.launch(1.0 / std::sqrt((double)call.d)));
}

// decode_q1(q, segments, extra_kv or None, attn_dtype)
PyObject* decode_q1_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 4) fail(PyExc_TypeError, "decode_q1 takes 4 arguments");
  const Items segs(a[1]);
  if (segs.n > 3) fail(PyExc_RuntimeError, "q1 attention supports at most 3 segments, got " + std::to_string(segs.n));
  Tensor q = tensor_arg(a[0], "q");
  const at::ScalarType dt = dtype_arg(a[3]);
  if (q.scalar_type() != dt) q = unlocked([&] { return q.to(dt); });
  if (q.dim() != 3) fail(PyExc_ValueError, "q must be [B, H, D]");
  DecodeCall call(q.unsqueeze(1));
  for (Py_ssize_t i = 0; i < segs.n; ++i) call.add_segment(segs[i], 0xFF);
  if (a[2] != Py_None) {
    const Items extras(a[2]);
    if (extras.n > 2) fail(PyExc_RuntimeError, "q1 attention supports at most 2 extra entries, got " + std::to_string(extras.n));
    for (Py_ssize_t i = 0; i < extras.n; ++i) {
      const Items e(extras[i]);
      if (e.n != 2) fail(PyExc_ValueError, "an extra entry is (k, v)");
      call.add_extra(tensor_arg(e[0], "extra k"), tensor_arg(e[1], "extra v"), 1);
    }
  }
  return THPVariable_Wrap(call.launch(1.0 / std::sqrt((double)call.d)).squeeze(1));
}

// kv_update(nw_k, nw_v, nw_len, nw_pos, br_k, br_v, br_len, k_window, v_window, k_retained,
//           v_retained, active, window_tokens); the ring arguments are not looked at when window_tokens <= 0
PyObject* kv_update_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 13) fail(PyExc_TypeError, "kv_update takes 13 arguments");
  const Tensor &br_k = tensor_arg(a[4], "br_k"), &br_v = tensor_arg(a[5], "br_v"), &br_len = tensor_arg(a[6], "br_len");
  Tensor kr = tensor_arg(a[9], "k_retained"), vr = tensor_arg(a[10], "v_retained"), active = tensor_arg(a[11], "active_mask");
  const long long window_tokens = int_arg(a[12]);
  if (kr.dim() != 3) fail(PyExc_ValueError, "k_retained must be [B, H, D]");
  const int64_t b = kr.size(0), h = kr.size(1), d = kr.size(2);
  require(br_k.sizes() == br_v.sizes() && br_k.is_cuda() && br_k.is_contiguous() && br_v.is_contiguous(),
          "the retained caches must be contiguous CUDA tensors of one shape");
  require(br_len.dim() == 2 && br_len.size(0) == b && br_len.size(1) == h && br_len.scalar_type() == at::kLong &&
              br_len.is_contiguous(),
          "br_len must be contiguous int64 [B, H]");
  // a bool tensor holds the 0 / 1 bytes that the kernel reads
  if ((active.scalar_type() != at::kChar && active.scalar_type() != at::kBool) || !active.is_contiguous())
    active = unlocked([&] { return active.to(active.scalar_type() == at::kBool ? at::kBool : at::kChar).contiguous(); });
  auto row = [](Tensor& x, const Tensor& like) {
    if (x.scalar_type() != like.scalar_type() || !x.is_contiguous())
      x = unlocked([&] { return x.to(like.scalar_type()).contiguous(); });
  };
  row(kr, br_k);
  row(vr, br_v);
  Tensor kw, vw;
  void *nw_k_ptr = nullptr, *nw_v_ptr = nullptr;
  int64_t *nw_len_ptr = nullptr, *nw_pos_ptr = nullptr, storage = 0;
  if (window_tokens > 0) {
    const Tensor &nw_k = tensor_arg(a[0], "nw_k"), &nw_v = tensor_arg(a[1], "nw_v");
    const Tensor &nw_len = tensor_arg(a[2], "nw_len"), &nw_pos = tensor_arg(a[3], "nw_pos");
    require(nw_k.sizes() == nw_v.sizes(), "nw.k/v shape mismatch");
    require(nw_k.dim() == 4 && nw_k.size(0) == b && nw_k.size(1) == h && nw_k.is_contiguous() && nw_v.is_contiguous(),
            "the ring must be contiguous [B, H, storage, D]");
    require(nw_len.dim() == 1 && nw_len.size(0) == b && nw_pos.dim() == 1 && nw_pos.size(0) == b, "ring counters must be [B]");
    require(nw_len.scalar_type() == at::kLong && nw_pos.scalar_type() == at::kLong, "ring counters must be int64");
    storage = nw_k.size(2);
    kw = tensor_arg(a[7], "k_window");
    vw = tensor_arg(a[8], "v_window");
    row(kw, nw_k);
    row(vw, nw_v);
    nw_k_ptr = nw_k.data_ptr(), nw_v_ptr = nw_v.data_ptr();
    nw_len_ptr = nw_len.data_ptr<int64_t>(), nw_pos_ptr = nw_pos.data_ptr<int64_t>();
  }
  const int rc = unlocked([&] {
    const c10::cuda::CUDAGuard guard(br_k.device());
    return spsattn_kv_update(
        nw_k_ptr, nw_v_ptr, nw_len_ptr, nw_pos_ptr, br_k.data_ptr(), br_v.data_ptr(), br_len.data_ptr<int64_t>(),
        kw.defined() ? kw.data_ptr() : nullptr, vw.defined() ? vw.data_ptr() : nullptr, kr.data_ptr(), vr.data_ptr(),
        reinterpret_cast<const int8_t*>(active.data_ptr()), b, h, d, storage, br_k.size(2), (int)window_tokens,
        (int)br_k.element_size(), stream_of(br_k));
  });
  check_rc(rc, "spsattn_kv_update");
  Py_RETURN_NONE;
}

#include "native_engine.h"

// ------------------------------------------------------------------------------------- module

PyObject* status_word_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 1) fail(PyExc_TypeError, "status_word takes 1 argument");
  const int device = (int)int_arg(a[0]);
  return THPVariable_Wrap(unlocked([&] { return status_word(device); }));
}

// setup(SpsAttnError, PackedKVSegment)
PyObject* setup_impl(PyObject* const* a, Py_ssize_t n) {
  if (n != 2) fail(PyExc_TypeError, "setup takes 2 arguments");
  g_spsattn_error = Py_NewRef(a[0]);
  g_packed_type = Py_NewRef(a[1]);
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS          // torch's errors (out of memory, say) as torch's own functions raise them
  try {
    return F(args, n);
  } catch (const PyError& e) {
    raise(e);
  }
  END_HANDLE_TH_ERRORS
}

#define SPS_ENTRY(name, fn) \
  { name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<fn>)), METH_FASTCALL, nullptr }

PyMethodDef g_methods[] = {
    SPS_ENTRY("prefill", prefill_impl),
    SPS_ENTRY("prefill_backward", prefill_backward_impl),
    SPS_ENTRY("decode", decode_impl),
    SPS_ENTRY("decode_q2", decode_q2_impl),
    SPS_ENTRY("decode_q1", decode_q1_impl),
    SPS_ENTRY("kv_update", kv_update_impl),
    SPS_ENTRY("engine_model", engine_model_impl),
    SPS_ENTRY("engine_scan", engine_scan_impl),
    SPS_ENTRY("engine_prefill", engine_prefill_impl),
    SPS_ENTRY("engine_step", engine_step_impl),
    SPS_ENTRY("status_word", status_word_impl),
    SPS_ENTRY("setup", setup_impl),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&g_module); }
