// The calls of quant.py that a decoder makes per token, with their checks, allocations and launches in
// one native call each.
//
// An eager decode or prompt call launches kernels of 3 to 30 us; made from Python through ctypes a
// launch costs about 18 us of host time (allocations with keyword arguments, stream lookup,
// argument conversion), from here about 5.  A projection of 8 rows 36.3 -> 10.8 us (7.9 as one launch), the
// MLP of one row 51 -> 38 (30 now), a decoder layer of 16 rows 162 -> 73 (55 now); the last two are their kernels' time.
//
// Each function here does what its namesake in quant.py does for the plain case -- ordinary CUDA tensors
// of the current device, no dispatch mode, transform, forward-mode level or tracer, operands the kernels take
// -- and returns None for everything else; quant.py then runs its own code, which decides, converts and raises as it always did.
// Nothing is kept between calls but the scratch slots' counter, which quant.py shares.
//
// The kernels' library is not linked: quant.py hands over the addresses of the functions it has loaded.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <atomic>
#include <cstring>

#include "../../include/braid_b200.h"

// What this file was compiled against: it reads fields of torch's and Python's objects by their layout there.  build.py
// finds the text in the built file and leaves a file of another torch or Python unloaded.
#ifndef BQ_HOST_KEY
#error "compile with braid_b200/build.py"
#endif
extern "C" __attribute__((visibility("default"), used)) const char bq_host_built_for[] =
    "braid_b200 native calls for " BQ_HOST_KEY;

namespace {

struct Lib {
  decltype(&bq_quantize_act) quantize_act;
  decltype(&bq_quantize_weight) quantize_weight;
  decltype(&bq_quantize_weight_workspace_bytes) quantize_weight_workspace;
  decltype(&bq_rmsnorm_quant) rmsnorm_quant;
  decltype(&bq_rmsnorm_quant_rows) rmsnorm_quant_rows;
  decltype(&bq_rmsnorm_scale) rmsnorm_scale;
  decltype(&bq_gated_rmsnorm_quant) gated_rmsnorm_quant;
  decltype(&bq_gated_rmsnorm_scale) gated_rmsnorm_scale;
  decltype(&bq_cast_act) cast_act;
  decltype(&bq_sigmoid_gate_quant) sigmoid_gate_quant;
  decltype(&bq_sigmoid_mul_dense_scale) sigmoid_mul_dense_scale;
  decltype(&bq_gemm_w8a8_grouped) gemm_grouped;
  decltype(&bq_gemm_w8a8_residual) gemm_residual;
  decltype(&bq_linear_w8a8) linear;
  decltype(&bq_project_mixed) project_mixed;
  decltype(&bq_gate_up_silu_quant_next_w8a8) gate_up_silu_quant;
  decltype(&bq_gate_up_silu_w8a8) gate_up_silu;
  decltype(&bq_mlp_w8a8_takes) mlp_takes;
  decltype(&bq_stream_is_captured) stream_is_captured;
  decltype(&bq_mlp_w8a8) mlp;
  decltype(&bq_lm_head_argmax) lm_head_argmax;
  decltype(&bq_lm_head_argmax_workspace_bytes) lm_head_argmax_workspace;
} g_lib;
bool g_ready = false;
int64_t g_two_launch_from = 0;

constexpr int kMaxDevices = 64;
constexpr uint32_t kMaxSlots = 256;
struct Scratch {
  std::atomic<uint64_t> base{0};      // device address of the slots, 0 = none yet
  std::atomic<uint32_t> next{0};
  std::atomic<uint32_t> next_held{0};
  std::atomic<bool> held[kMaxSlots]{};
};
Scratch g_scratch[kMaxDevices];
uint32_t g_slots = 1, g_slot_bytes = 64;
std::atomic<int64_t> g_launches{0};

void* take_slot(int dev) {
  g_launches.fetch_add(1, std::memory_order_relaxed);
  const uint32_t slot = g_scratch[dev].next.fetch_add(1, std::memory_order_relaxed) % g_slots;
  return reinterpret_cast<void*>(g_scratch[dev].base.load(std::memory_order_relaxed) + uint64_t(slot) * g_slot_bytes);
}

// A slot for a call of two launches that leaves something in it between them.  The slots above pass from hand to
// hand by count alone: a thread that is not scheduled between its two launches would find that another one, 256
// calls later, has taken its slot and returned it to zero.  So these are as many slots behind those, nobody else's,
// and each is held until both launches are in the stream.  While a graph is captured it is a common one: the graph puts both
// launches into a stream at once whenever it is replayed, and keeps the slot for longer than it could be held.
struct HeldSlot {
  Scratch& pool;
  void* address;
  int64_t index = -1;       // held; -1: a common one
  HeldSlot(int dev, void* stream) : pool(g_scratch[dev]) {
    if (g_lib.stream_is_captured(stream) != 0) {
      address = take_slot(dev);
      return;
    }
    g_launches.fetch_add(1, std::memory_order_relaxed);
    do index = pool.next_held.fetch_add(1, std::memory_order_relaxed) % g_slots;
    while (pool.held[index].exchange(true, std::memory_order_acquire));
    address = reinterpret_cast<void*>(pool.base.load(std::memory_order_relaxed) + uint64_t(g_slots + index) * g_slot_bytes);
  }
  ~HeldSlot() {
    if (index >= 0) pool.held[index].store(false, std::memory_order_release);
  }
  HeldSlot(const HeldSlot&) = delete;
  HeldSlot& operator=(const HeldSlot&) = delete;
};

// What a call needs of its surroundings; false = leave it to quant.py.  A dual tensor is an ordinary strided
// one with nothing in its keys to tell it by, so an open forward-mode level is asked for by itself, as quant.py does.
struct Here {
  int dev = -1;
  void* stream = nullptr;
  bool ok = false;
  explicit Here(const at::Tensor& t) {
    if (!g_ready || !t.defined() || !t.is_cuda() || c10::impl::TorchDispatchModeTLS::stack_len() > 0 ||
        c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) ||
        at::tracer::impl::is_dispatch_enabled() || torch::autograd::ForwardADLevel::try_get_by_idx(0) != nullptr)
      return;
    dev = t.device().index();
    if (dev < 0 || dev >= kMaxDevices || dev != c10::cuda::current_device() ||
        g_scratch[dev].base.load(std::memory_order_relaxed) == 0)
      return;
    stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    ok = true;
  }
};

// An ordinary tensor of this device: memory of its own, read as it lies there.
bool plain(const Here& h, const at::Tensor& t) {
  return t.defined() && t.is_cuda() && t.device().index() == h.dev && t.layout() == at::kStrided && t.has_storage() &&
         !t.unsafeGetTensorImpl()->is_python_dispatch() && !t.is_neg() && !t._is_zerotensor();
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return BQ_DTYPE_F32;
    case at::kBFloat16: return BQ_DTYPE_BF16;
    case at::kHalf: return BQ_DTYPE_F16;
    default: return -1;
  }
}

bool aligned(const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; }

// `[rows, cols]` with a contiguous last axis and one row stride, without a copy.
struct Rows {
  int64_t rows = 0, ld = 0;
  bool ok = false;
  Rows(const at::Tensor& t, int64_t cols) {
    if (cols <= 0 || t.numel() == 0) return;
    if (t.dim() == 2 && t.stride(1) == 1 && t.size(1) == cols) {
      rows = t.size(0); ld = t.stride(0); ok = true;
    } else if (t.is_contiguous()) {
      rows = t.numel() / cols; ld = cols; ok = true;
    }
  }
};

bool is_codes(const Here& h, const at::Tensor& xq) {
  return plain(h, xq) && xq.scalar_type() == at::kFloat8_e4m3fn && xq.dim() == 2 && xq.is_contiguous() && xq.numel() > 0;
}
bool is_scale(const Here& h, const at::Tensor& s) {
  return plain(h, s) && s.scalar_type() == at::kFloat && s.numel() == 1;
}
bool is_weight(const Here& h, const at::Tensor& w, int64_t K) {
  return plain(h, w) && w.scalar_type() == at::kFloat8_e4m3fn && w.dim() == 2 && w.size(1) == K && w.is_contiguous();
}
// Would torch follow an addition to or a product with this tensor?
bool recorded(const at::Tensor& t) {
  return (t.requires_grad() && c10::GradMode::is_enabled()) || at::autocast::is_autocast_enabled(at::kCUDA);
}

// Memory that is written whole before anybody reads it, from the allocator without the dispatcher (0.5 us of a call's 5):
// the modes that would see a torch.empty are what Here leaves to quant.py.
at::Tensor empty(const Here& h, at::IntArrayRef sizes, at::ScalarType t) {
  return at::Tensor(at::detail::empty_cuda(sizes, t, c10::Device(at::kCUDA, (c10::DeviceIndex)h.dev), std::nullopt));
}

struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

// A positional argument as a tensor; undefined = not a tensor, or a subclass other than Parameter, whose results
// torch would wrap.
at::Tensor arg(PyObject* o) { return THPVariable_CheckExact(o) ? THPVariable_Unpack(o) : at::Tensor(); }
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* pair(const at::Tensor& a, const at::Tensor& b) {
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, wrap(a));
  PyTuple_SET_ITEM(r, 1, wrap(b));
  return r;
}
// A status other than OK: that call launched nothing whose result is kept, and quant.py makes it again and raises.
PyObject* refused() {
  g_launches.fetch_sub(1, std::memory_order_relaxed);
  Py_RETURN_NONE;
}

#define BQ_ARGS(n)                                                         \
  if (nargs != (n)) {                                                      \
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");         \
    return nullptr;                                                        \
  }

// ---- the quantizers -------------------------------------------------------------------------
// (q, scale) of a contiguous activation, undefined tensors where quant.py has to decide.
struct Quantized { at::Tensor q, scale; int rc = BQ_OK; };

Quantized quantize(const Here& h, const at::Tensor& x) {
  Quantized r;
  const int code = dtype_code(x.scalar_type());
  if (!plain(h, x) || code < 0 || x.numel() == 0 || !x.is_contiguous() || !aligned(x.data_ptr(), 16)) return r;
  at::Tensor q = empty(h, x.sizes(), at::kFloat8_e4m3fn), scale = empty(h, {1, 1}, at::kFloat);
  void* slot = take_slot(h.dev);
  {
    NoGil no_gil;
    r.rc = g_lib.quantize_act(x.data_ptr(), code, x.numel(), q.data_ptr(), scale.data_ptr<float>(), slot, 16, h.stream);
  }
  r.q = q; r.scale = scale;
  return r;
}

PyObject* quantize_act(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(1)
  const at::Tensor x = arg(a[0]);
  const Here h(x);
  if (!h.ok) Py_RETURN_NONE;
  const Quantized r = quantize(h, x);
  if (!r.q.defined()) Py_RETURN_NONE;
  if (r.rc != BQ_OK) return refused();
  return pair(r.q, r.scale);
  END_HANDLE_TH_ERRORS
}

// quantize_weight(w) -> (q, scale): a loader's call, 22 us from Python and 9 from here, which is its time for weights of up to
// a few MB
PyObject* quantize_weight(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(1)
  const at::Tensor w = arg(a[0]);
  const Here h(w);
  if (!h.ok || !plain(h, w)) Py_RETURN_NONE;
  const int code = dtype_code(w.scalar_type());
  if (code < 0 || w.dim() != 2 || w.numel() == 0 || !w.is_contiguous() || !aligned(w.data_ptr(), 16) || recorded(w)) Py_RETURN_NONE;
  const at::Tensor q = empty(h, w.sizes(), at::kFloat8_e4m3fn), scale = empty(h, {1, 1}, at::kFloat);
  const size_t bytes = g_lib.quantize_weight_workspace();
  const at::Tensor ws = empty(h, {(int64_t)bytes}, at::kByte);
  int rc;
  {
    NoGil no_gil;
    rc = g_lib.quantize_weight(w.data_ptr(), code, w.numel(), q.data_ptr(), scale.data_ptr<float>(), ws.data_ptr(), bytes,
                               h.stream);
  }
  if (rc != BQ_OK) Py_RETURN_NONE;
  return pair(q, scale);
  END_HANDLE_TH_ERRORS
}

// cast of a dense [rows, cols] under a scale
int cast(const Here& h, const at::Tensor& x, const at::Tensor& scale, at::Tensor& q) {
  q = empty(h, x.sizes(), at::kFloat8_e4m3fn);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  NoGil no_gil;
  return g_lib.cast_act(x.data_ptr(), dtype_code(x.scalar_type()), x.numel(), scale.data_ptr<float>(), q.data_ptr(), h.stream);
}

// rms_norm_quant(x, gamma, eps, keep_dense) -> (q, scale, dense or None)
PyObject* rms_norm_quant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(4)
  const at::Tensor x = arg(a[0]), gamma = arg(a[1]);
  const Here h(x);
  if (!h.ok || !plain(h, x) || !plain(h, gamma) || x.dim() < 1) Py_RETURN_NONE;
  const int code = dtype_code(x.scalar_type());
  const int64_t K = x.size(-1);
  const Rows r(x, K);
  if (code < 0 || !r.ok || K % 4 || gamma.scalar_type() != at::kFloat || gamma.numel() != K || !gamma.is_contiguous())
    Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(a[2]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  const bool keep = PyObject_IsTrue(a[3]) == 1;
  at::Tensor q = empty(h, {r.rows, K}, at::kFloat8_e4m3fn), scale = empty(h, {1, 1}, at::kFloat), dense;
  if (keep) dense = empty(h, x.sizes(), x.scalar_type());
  void* const hp = keep ? dense.data_ptr() : nullptr;
  void* slot = take_slot(h.dev);
  int rc;
  {
    NoGil no_gil;
    rc = g_lib.rmsnorm_quant(x.data_ptr(), code, r.rows, K, r.ld, gamma.data_ptr<float>(), (float)eps, hp, K, q.data_ptr(),
                             scale.data_ptr<float>(), slot, 16, h.stream);
  }
  if (rc == BQ_ERR_TOO_LARGE && !keep) {
    const at::Tensor rstd = empty(h, {r.rows}, at::kFloat);
    NoGil no_gil;
    rc = g_lib.rmsnorm_quant_rows(x.data_ptr(), code, r.rows, K, r.ld, gamma.data_ptr<float>(), (float)eps, q.data_ptr(),
                                  scale.data_ptr<float>(), rstd.data_ptr<float>(), slot, 16, h.stream);
    if (rc == BQ_OK) g_launches.fetch_add(1, std::memory_order_relaxed);
    if (rc == BQ_ERR_UNSUPPORTED) rc = BQ_ERR_TOO_LARGE;
  }
  if (rc == BQ_ERR_TOO_LARGE) {      // h is wanted, or rows are no whole 16-byte pieces: h and its scale, then the cast of h
    at::Tensor norm = keep ? dense : empty(h, {r.rows, K}, x.scalar_type());
    {
      NoGil no_gil;
      rc = g_lib.rmsnorm_scale(x.data_ptr(), code, r.rows, K, r.ld, gamma.data_ptr<float>(), (float)eps, norm.data_ptr(), K,
                               scale.data_ptr<float>(), slot, 16, h.stream);
    }
    if (rc == BQ_OK) {
      g_launches.fetch_add(1, std::memory_order_relaxed);
      NoGil no_gil;
      rc = g_lib.cast_act(norm.data_ptr(), code, norm.numel(), scale.data_ptr<float>(), q.data_ptr(), h.stream);
    }
  }
  if (rc != BQ_OK) return refused();
  PyObject* out = PyTuple_New(3);
  if (out == nullptr) return nullptr;
  PyTuple_SET_ITEM(out, 0, wrap(q));
  PyTuple_SET_ITEM(out, 1, wrap(scale));
  if (keep) PyTuple_SET_ITEM(out, 2, wrap(dense));
  else { Py_INCREF(Py_None); PyTuple_SET_ITEM(out, 2, Py_None); }
  return out;
  END_HANDLE_TH_ERRORS
}

// gated_rms_norm_quant(y, z, gamma, eps, head_dim) -> (q, scale)
PyObject* gated_rms_norm_quant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(5)
  const at::Tensor y = arg(a[0]), z = arg(a[1]), gamma = arg(a[2]);
  const Here h(z);
  if (!h.ok || !plain(h, y) || !plain(h, z) || !plain(h, gamma) || z.dim() < 1) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(a[3]);
  const long head_dim = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  const int code = dtype_code(z.scalar_type()), ycode = dtype_code(y.scalar_type());
  const int64_t width = z.size(-1);
  if (code < 0 || ycode < 0 || (ycode != code && ycode != BQ_DTYPE_F32) || head_dim != 128 || width % head_dim ||
      y.numel() != z.numel() || gamma.scalar_type() != at::kFloat || gamma.numel() != head_dim || !gamma.is_contiguous())
    Py_RETURN_NONE;
  if (y.size(-1) != width && !y.is_contiguous()) Py_RETURN_NONE;
  const Rows ry(y, width), rz(z, width);
  if (!ry.ok || !rz.ok || ry.rows != rz.rows || width / head_dim > 64) Py_RETURN_NONE;
  const int64_t heads = width / head_dim;
  at::Tensor q = empty(h, {rz.rows, width}, at::kFloat8_e4m3fn), scale = empty(h, {1, 1}, at::kFloat);
  void* slot = take_slot(h.dev);
  int rc;
  {
    NoGil no_gil;
    rc = g_lib.gated_rmsnorm_quant(y.data_ptr(), ycode, ry.ld, z.data_ptr(), code, rz.ld, gamma.data_ptr<float>(),
                                   (float)eps, rz.rows, heads, head_dim, q.data_ptr(), scale.data_ptr<float>(), slot, 16,
                                   h.stream);
  }
  if (rc == BQ_ERR_TOO_LARGE) {
    at::Tensor core = empty(h, {rz.rows, width}, z.scalar_type());
    {
      NoGil no_gil;
      rc = g_lib.gated_rmsnorm_scale(y.data_ptr(), ycode, ry.ld, z.data_ptr(), code, rz.ld, gamma.data_ptr<float>(),
                                     (float)eps, rz.rows, heads, head_dim, core.data_ptr(), width,
                                     scale.data_ptr<float>(), slot, 16, h.stream);
    }
    if (rc == BQ_OK) {
      g_launches.fetch_add(1, std::memory_order_relaxed);
      NoGil no_gil;
      rc = g_lib.cast_act(core.data_ptr(), code, core.numel(), scale.data_ptr<float>(), q.data_ptr(), h.stream);
    }
  }
  if (rc != BQ_OK) return refused();
  return pair(q, scale);
  END_HANDLE_TH_ERRORS
}

// sigmoid_gate_quant(o, gate) -> (q, scale); gate dense, or the [rows, H, D] view of a wider row
PyObject* sigmoid_gate_quant(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(2)
  const at::Tensor o = arg(a[0]), gate = arg(a[1]);
  const Here h(o);
  if (!h.ok || !plain(h, o) || !plain(h, gate) || o.dim() != 2) Py_RETURN_NONE;
  const int code = dtype_code(o.scalar_type());
  const int64_t cols = o.size(1);
  const Rows r(o, cols);
  if (code < 0 || gate.scalar_type() != o.scalar_type() || !r.ok) Py_RETURN_NONE;
  int64_t ld_gate, chunk = cols, chunk_stride = 0;
  if (gate.dim() == 3 && gate.size(0) == r.rows && gate.size(1) * gate.size(2) == cols && gate.stride(2) == 1) {
    ld_gate = gate.stride(0); chunk = gate.size(2); chunk_stride = gate.stride(1);
  } else if (gate.dim() == 2 && gate.sizes() == o.sizes() && gate.stride(1) == 1) {
    ld_gate = gate.stride(0);
  } else {
    Py_RETURN_NONE;
  }
  at::Tensor q = empty(h, {r.rows, cols}, at::kFloat8_e4m3fn), scale = empty(h, {1, 1}, at::kFloat);
  int rc;
  if (r.rows * cols >= g_two_launch_from) {
    at::Tensor dense = empty(h, {r.rows, cols}, o.scalar_type());
    if (!aligned(dense.data_ptr(), 16)) Py_RETURN_NONE;
    void* slot = take_slot(h.dev);
    NoGil no_gil;
    rc = g_lib.sigmoid_mul_dense_scale(o.data_ptr(), gate.data_ptr(), code, r.rows, cols, r.ld, ld_gate, chunk,
                                       chunk_stride, dense.data_ptr(), scale.data_ptr<float>(), slot, 16, h.stream);
    if (rc == BQ_OK) {
      g_launches.fetch_add(1, std::memory_order_relaxed);
      rc = g_lib.cast_act(dense.data_ptr(), code, dense.numel(), scale.data_ptr<float>(), q.data_ptr(), h.stream);
    }
  } else {
    void* slot = take_slot(h.dev);
    NoGil no_gil;
    rc = g_lib.sigmoid_gate_quant(o.data_ptr(), gate.data_ptr(), code, r.rows, cols, r.ld, ld_gate, chunk, chunk_stride,
                                  q.data_ptr(), scale.data_ptr<float>(), slot, 16, h.stream);
  }
  if (rc != BQ_OK) return refused();
  return pair(q, scale);
  END_HANDLE_TH_ERRORS
}

// ---- the GEMMs ------------------------------------------------------------------------------
// One weight, with or without the residual added, into `y` if there is one already; undefined where quant.py has
// to decide.
at::Tensor gemm(const Here& h, const at::Tensor& xq, const at::Tensor& sx, const at::Tensor& w, const at::Tensor& sw,
                at::ScalarType out, const at::Tensor& residual, int& rc, at::Tensor y = {}) {
  rc = BQ_OK;
  const int code = dtype_code(out);
  if (code < 0 || !is_codes(h, xq) || !is_scale(h, sx) || !is_scale(h, sw) || !is_weight(h, w, xq.size(1))) return {};
  const int64_t M = xq.size(0), K = xq.size(1), N = w.size(0);
  const bool res = residual.defined();
  if (res && (!plain(h, residual) || residual.dim() != 2 || residual.size(0) != M || residual.size(1) != N ||
              residual.scalar_type() != out || residual.stride(1) != 1 || recorded(residual)))
    return {};
  if (!y.defined()) y = empty(h, {M, N}, out);
  void* slot = take_slot(h.dev);
  const void* wq = w.data_ptr();
  const float* swp = sw.data_ptr<float>();
  void* yp = y.data_ptr();
  NoGil no_gil;
  if (res)
    rc = g_lib.gemm_residual(xq.data_ptr(), wq, sx.data_ptr<float>(), swp, residual.data_ptr(), residual.stride(0), yp, code,
                             M, N, K, N, slot, 16, h.stream);
  else
    rc = g_lib.gemm_grouped(xq.data_ptr(), sx.data_ptr<float>(), M, K, 1, &wq, &swp, &yp, &N, &N, code, slot, 16, h.stream);
  return y;
}

// What a GEMM gives back to Python: the result in `lead`'s shape, None where quant.py has to decide.
PyObject* gemm_result(const at::Tensor& y, int rc) {
  if (!y.defined()) Py_RETURN_NONE;
  if (rc != BQ_OK) return refused();
  return wrap(y);
}

// linear(x, w, sw, residual or None): quantize, multiply, leading dimensions kept.  Few rows: one launch.
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(4)
  const at::Tensor x = arg(a[0]), w = arg(a[1]), sw = arg(a[2]);
  const Here h(x);
  if (!h.ok || !w.defined() || w.dim() != 2 || x.dim() < 1 || x.size(-1) != w.size(1) || x.numel() == 0) Py_RETURN_NONE;
  const bool res = a[3] != Py_None;
  at::Tensor residual = arg(a[3]);
  if (res && !residual.defined()) Py_RETURN_NONE;
  const int64_t K = w.size(1), N = w.size(0);
  // everything the GEMM would refuse is refused before the quantizer runs
  if (!plain(h, x) || !is_weight(h, w, K) || !is_scale(h, sw) || !x.is_contiguous() || K % 16 || N % 16 ||
      !aligned(w.data_ptr(), 16))
    Py_RETURN_NONE;
  if (res) {
    if (!plain(h, residual) || recorded(residual) || residual.numel() != x.numel() / K * N) Py_RETURN_NONE;
    if (residual.dim() != 2) {
      if (!residual.is_contiguous()) Py_RETURN_NONE;
      residual = residual.view({-1, N});
    }
  }
  auto shaped = [&](const at::Tensor& y) {
    if (x.dim() == 2) return y;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    return y.view(shape);
  };
  int rc;
  const int64_t M = x.numel() / K;
  const int code = dtype_code(x.scalar_type());
  at::Tensor y;
  if (M <= BQ_LINEAR_MAX_ROWS && code >= 0 && aligned(x.data_ptr(), 16) &&
      (!res || (residual.scalar_type() == x.scalar_type() && residual.size(0) == M && residual.stride(1) == 1))) {
    y = empty(h, {M, N}, x.scalar_type());
    void* slot = take_slot(h.dev);
    const void* wq = w.data_ptr();
    const float* swp = sw.data_ptr<float>();
    void* yp = y.data_ptr();
    {
      NoGil no_gil;
      rc = g_lib.linear(x.data_ptr(), code, M, K, 1, &wq, &swp, res ? residual.data_ptr() : nullptr,
                        res ? residual.stride(0) : 0, &yp, &N, &N, slot, 16, h.stream);
    }
    if (rc == BQ_OK) return wrap(shaped(y));
    g_launches.fetch_sub(1, std::memory_order_relaxed);
  }
  const Quantized r = quantize(h, x);
  if (!r.q.defined()) Py_RETURN_NONE;
  if (r.rc != BQ_OK) return refused();
  y = gemm(h, x.dim() == 2 ? r.q : r.q.view({-1, K}), r.scale, w, sw, x.scalar_type(), residual, rc, y);
  if (y.defined() && rc == BQ_OK) y = shaped(y);
  return gemm_result(y, rc);
  END_HANDLE_TH_ERRORS
}

bool scalar_type_of(PyObject* o, at::ScalarType& t) {
  if (!THPDtype_Check(o)) return false;
  t = reinterpret_cast<THPDtype*>(o)->scalar_type;
  return true;
}

// matmul(xq, sx, w, sw, dtype, residual or None)
PyObject* matmul(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(6)
  const at::Tensor xq = arg(a[0]), sx = arg(a[1]), w = arg(a[2]), sw = arg(a[3]);
  at::ScalarType out;
  const Here h(xq);
  if (!h.ok || !scalar_type_of(a[4], out)) Py_RETURN_NONE;
  const at::Tensor residual = arg(a[5]);
  if (a[5] != Py_None && !residual.defined()) Py_RETURN_NONE;
  int rc;
  const at::Tensor y = gemm(h, xq, sx, w, sw, out, residual, rc);
  return gemm_result(y, rc);
  END_HANDLE_TH_ERRORS
}

// project(xq, sx, dense or None, dtype, (w...), (sw or None ...)) -> list of [M, N_i]; a weight
// without a scale is a 16-bit one, multiplied with `dense`
PyObject* project(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(6)
  const at::Tensor xq = arg(a[0]), sx = arg(a[1]), dense = arg(a[2]);
  at::ScalarType out;
  const Here h(xq);
  if (!h.ok || !scalar_type_of(a[3], out) || !PyTuple_Check(a[4]) || !PyTuple_Check(a[5])) Py_RETURN_NONE;
  const Py_ssize_t n = PyTuple_GET_SIZE(a[4]);
  const int code = dtype_code(out);
  if (n < 1 || n > BQ_MAX_SEGMENTS || PyTuple_GET_SIZE(a[5]) != n || code < 0 || !is_codes(h, xq) || !is_scale(h, sx))
    Py_RETURN_NONE;
  const int64_t M = xq.size(0), K = xq.size(1);
  std::array<at::Tensor, BQ_MAX_SEGMENTS> y;
  const void* wq[BQ_MAX_SEGMENTS];
  const float* sw[BQ_MAX_SEGMENTS];
  void* yp[BQ_MAX_SEGMENTS];
  int64_t N[BQ_MAX_SEGMENTS];
  int kind[BQ_MAX_SEGMENTS];
  bool mixed = false, ragged = false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    const at::Tensor w = arg(PyTuple_GET_ITEM(a[4], i));
    PyObject* const so = PyTuple_GET_ITEM(a[5], i);
    if (!w.defined()) Py_RETURN_NONE;
    if (so == Py_None) {
      if (!plain(h, w) || w.scalar_type() != out || w.dim() != 2 || w.size(1) != K || w.size(0) % 4 || w.size(0) == 0 ||
          !w.is_contiguous() || !aligned(w.data_ptr(), 16) || (M > 256 && w.size(0) > 256) ||
          ((M > 256 || w.size(0) % 16) && recorded(w)))
        Py_RETURN_NONE;
      ragged = ragged || w.size(0) % 16 != 0;
      kind[i] = 1;
      sw[i] = nullptr;
      mixed = true;
    } else {
      const at::Tensor s = arg(so);
      if (!is_scale(h, s) || !is_weight(h, w, K)) Py_RETURN_NONE;
      kind[i] = 0;
      sw[i] = s.data_ptr<float>();
    }
    wq[i] = w.data_ptr();
    N[i] = w.size(0);
  }
  const void* dp = nullptr;
  if (mixed) {
    if (!dense.defined() || !plain(h, dense) || dense.scalar_type() != out || code == BQ_DTYPE_F32 ||
        !dense.is_contiguous() || dense.numel() != M * K || !aligned(dense.data_ptr(), 16) || ((M > 256 || ragged) && recorded(dense)))
      Py_RETURN_NONE;
    dp = dense.data_ptr();
  }
  for (Py_ssize_t i = 0; i < n; ++i) {
    y[i] = empty(h, {M, N[i]}, out);
    yp[i] = y[i].data_ptr();
  }
  void* slot = take_slot(h.dev);
  int rc;
  {
    NoGil no_gil;
    rc = mixed ? g_lib.project_mixed(xq.data_ptr(), sx.data_ptr<float>(), dp, code, M, K, (int)n, wq, sw, kind, yp, N, N,
                                     code, slot, 16, h.stream)
               : g_lib.gemm_grouped(xq.data_ptr(), sx.data_ptr<float>(), M, K, (int)n, wq, sw, yp, N, N, code, slot, 16,
                                    h.stream);
  }
  if (rc != BQ_OK) return refused();
  PyObject* list = PyList_New(n);
  if (list == nullptr) return nullptr;
  for (Py_ssize_t i = 0; i < n; ++i) PyList_SET_ITEM(list, i, wrap(y[i]));
  return list;
  END_HANDLE_TH_ERRORS
}

// mlp(xq, sx, dtype, gate, s_gate, up, s_up, down, s_down, residual or None) -> [M, H]; with sx None, xq is the [M, K] activation
// itself, and what is quantized here before a refusal comes back as (xq, sx)
PyObject* mlp(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(10)
  at::Tensor xq = arg(a[0]), sx = arg(a[1]);
  const bool quantized = a[1] != Py_None;
  at::ScalarType out;
  const Here h(xq);
  if (!h.ok || !scalar_type_of(a[2], out)) Py_RETURN_NONE;
  const int code = dtype_code(out);
  const at::Tensor wg = arg(a[3]), sg = arg(a[4]), wu = arg(a[5]), su = arg(a[6]), wd = arg(a[7]), sd = arg(a[8]);
  const at::Tensor residual = arg(a[9]);
  if (a[9] != Py_None && !residual.defined()) Py_RETURN_NONE;
  if (code < 0) Py_RETURN_NONE;
  if (quantized ? !is_codes(h, xq) || !is_scale(h, sx)
                : !plain(h, xq) || xq.scalar_type() != out || xq.dim() != 2 || xq.numel() == 0 || xq.size(1) % 16)
    Py_RETURN_NONE;
  const int64_t M = xq.size(0), K = xq.size(1);
  if (!wg.defined() || !wu.defined() || !wd.defined() || !is_weight(h, wg, K) || !is_weight(h, wu, K) ||
      wu.size(0) != wg.size(0) || !is_weight(h, wd, wg.size(0)) || !is_scale(h, sg) || !is_scale(h, su) || !is_scale(h, sd))
    Py_RETURN_NONE;
  const int64_t I = wg.size(0), N = wd.size(0);
  // what the down projection would refuse is refused before anything runs
  if (I % 64 || N % 16 || !aligned(wd.data_ptr(), 16)) Py_RETURN_NONE;
  if (residual.defined() &&
      (!plain(h, residual) || residual.dim() != 2 || residual.size(0) != M || residual.size(1) != N ||
       residual.scalar_type() != out || residual.stride(1) != 1 || residual.stride(0) < N || residual.stride(0) % 4 ||
       !aligned(residual.data_ptr(), out == at::kFloat ? 16 : 8) || recorded(residual)))
    Py_RETURN_NONE;
  int rc;
  if (!quantized) {
    const Quantized r = quantize(h, xq);
    if (!r.q.defined()) Py_RETURN_NONE;
    if (r.rc != BQ_OK) return refused();
    xq = r.q;
    sx = r.scale;
  }
  auto given_back = [&]() -> PyObject* {
    g_launches.fetch_sub(1, std::memory_order_relaxed);
    if (!quantized) return pair(xq, sx);
    Py_RETURN_NONE;
  };
  // both products in one call, where that form takes them: asked before anything is allocated
  if (M <= BQ_MLP_MAX_ROWS && g_lib.mlp_takes(M, I, N, code) != 0) {
    const at::Tensor act = empty(h, {M, I}, out), y = empty(h, {M, N}, out);
    {
      NoGil no_gil;
      const HeldSlot slot(h.dev, h.stream);
      rc = g_lib.mlp(xq.data_ptr(), sx.data_ptr<float>(), wg.data_ptr(), wu.data_ptr(), wd.data_ptr(), sg.data_ptr<float>(),
                     su.data_ptr<float>(), sd.data_ptr<float>(), residual.defined() ? residual.data_ptr() : nullptr,
                     residual.defined() ? residual.stride(0) : 0, M, K, I, N, code, act.data_ptr(), y.data_ptr(), N,
                     slot.address, 16, h.stream);
    }
    if (rc == BQ_OK) {
      g_launches.fetch_add(1, std::memory_order_relaxed);      // the slot counted one of the two
      return wrap(y);
    }
    if (rc != BQ_ERR_UNSUPPORTED) return given_back();
    g_launches.fetch_sub(1, std::memory_order_relaxed);
  }
  at::Tensor hq, sh = empty(h, {1, 1}, at::kFloat), dense;
  if (M <= 256) hq = empty(h, {M, I}, at::kFloat8_e4m3fn);
  else dense = empty(h, {M, I}, out);
  void* slot = take_slot(h.dev);
  {
    NoGil no_gil;
    rc = M <= 256 ? g_lib.gate_up_silu_quant(xq.data_ptr(), sx.data_ptr<float>(), wg.data_ptr(), wu.data_ptr(),
                                             sg.data_ptr<float>(), su.data_ptr<float>(), M, I, K, code, hq.data_ptr(),
                                             sh.data_ptr<float>(), wd.data_ptr(), N * I, slot, 16, h.stream)
                  : g_lib.gate_up_silu(xq.data_ptr(), sx.data_ptr<float>(), wg.data_ptr(), wu.data_ptr(),
                                       sg.data_ptr<float>(), su.data_ptr<float>(), M, I, K, code, dense.data_ptr(), I,
                                       sh.data_ptr<float>(), slot, 16, h.stream);
  }
  if (rc != BQ_OK) return given_back();
  if (M > 256) {
    rc = cast(h, dense, sh, hq);
    if (rc != BQ_OK) return given_back();
  }
  const at::Tensor y = gemm(h, hq, sh, wd, sd, out, residual, rc);
  if (!y.defined() || rc != BQ_OK) return given_back();
  return wrap(y);
  END_HANDLE_TH_ERRORS
}

// lm_head_argmax(xq, sx, w, sw, dtype, want_logits) -> (indices, logits or None); M <= 256
PyObject* lm_head_argmax(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  BQ_ARGS(6)
  const at::Tensor xq = arg(a[0]), sx = arg(a[1]), w = arg(a[2]), sw = arg(a[3]);
  at::ScalarType out;
  const Here h(xq);
  if (!h.ok || !scalar_type_of(a[4], out)) Py_RETURN_NONE;
  const int code = dtype_code(out);
  if (code < 0 || !is_codes(h, xq) || xq.size(0) > 256 || !is_scale(h, sx) || !is_scale(h, sw) ||
      !w.defined() || !is_weight(h, w, xq.size(1)))
    Py_RETURN_NONE;
  const bool want = PyObject_IsTrue(a[5]) == 1;
  const int64_t M = xq.size(0), K = xq.size(1), N = w.size(0);
  const size_t need = g_lib.lm_head_argmax_workspace(M, N);
  at::Tensor partial = empty(h, {(int64_t)(need / 8)}, at::kLong), idx = empty(h, {M}, at::kLong), logits;
  if (want) logits = empty(h, {M, N}, out);
  void* slot = take_slot(h.dev);
  g_launches.fetch_add(1, std::memory_order_relaxed);       // the second-stage reduction
  int rc;
  {
    NoGil no_gil;
    rc = g_lib.lm_head_argmax(xq.data_ptr(), w.data_ptr(), sx.data_ptr<float>(), sw.data_ptr<float>(), code, M, N, K,
                              want ? logits.data_ptr() : nullptr, N, idx.data_ptr<int64_t>(), partial.data_ptr(), need, slot,
                              16, h.stream);
  }
  if (rc != BQ_OK) return refused();
  if (want) return pair(idx, logits);
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) return nullptr;
  PyTuple_SET_ITEM(r, 0, wrap(idx));
  Py_INCREF(Py_None);
  PyTuple_SET_ITEM(r, 1, Py_None);
  return r;
  END_HANDLE_TH_ERRORS
}

// ---- state shared with quant.py -------------------------------------------------------------
// init({name: address}, slots, slot_bytes, two_launch_from)
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  BQ_ARGS(4)
  if (!PyDict_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "init takes a dict of addresses");
    return nullptr;
  }
  auto get = [&](const char* name, auto& fn) {
    PyObject* o = PyDict_GetItemString(a[0], name);
    void* p = o != nullptr ? PyLong_AsVoidPtr(o) : nullptr;
    if (p == nullptr) {
      if (!PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "no address of %s", name);
      return false;
    }
    std::memcpy(&fn, &p, sizeof(p));
    return true;
  };
  if (!get("bq_quantize_act", g_lib.quantize_act) || !get("bq_quantize_weight", g_lib.quantize_weight) ||
      !get("bq_quantize_weight_workspace_bytes", g_lib.quantize_weight_workspace) || !get("bq_rmsnorm_quant", g_lib.rmsnorm_quant) ||
      !get("bq_rmsnorm_quant_rows", g_lib.rmsnorm_quant_rows) || !get("bq_rmsnorm_scale", g_lib.rmsnorm_scale) ||
      !get("bq_gated_rmsnorm_quant", g_lib.gated_rmsnorm_quant) ||
      !get("bq_gated_rmsnorm_scale", g_lib.gated_rmsnorm_scale) || !get("bq_cast_act", g_lib.cast_act) ||
      !get("bq_sigmoid_gate_quant", g_lib.sigmoid_gate_quant) ||
      !get("bq_sigmoid_mul_dense_scale", g_lib.sigmoid_mul_dense_scale) ||
      !get("bq_gemm_w8a8_grouped", g_lib.gemm_grouped) || !get("bq_gemm_w8a8_residual", g_lib.gemm_residual) ||
      !get("bq_linear_w8a8", g_lib.linear) || !get("bq_project_mixed", g_lib.project_mixed) || !get("bq_gate_up_silu_quant_next_w8a8", g_lib.gate_up_silu_quant) || !get("bq_mlp_w8a8", g_lib.mlp) ||
      !get("bq_mlp_w8a8_takes", g_lib.mlp_takes) || !get("bq_stream_is_captured", g_lib.stream_is_captured) ||
      !get("bq_gate_up_silu_w8a8", g_lib.gate_up_silu) || !get("bq_lm_head_argmax", g_lib.lm_head_argmax) ||
      !get("bq_lm_head_argmax_workspace_bytes", g_lib.lm_head_argmax_workspace))
    return nullptr;
  g_slots = (uint32_t)PyLong_AsUnsignedLong(a[1]);
  g_slot_bytes = (uint32_t)PyLong_AsUnsignedLong(a[2]);
  g_two_launch_from = PyLong_AsLongLong(a[3]);
  if (PyErr_Occurred()) return nullptr;
  if (g_slots < 1 || g_slots > kMaxSlots) {
    PyErr_SetString(PyExc_ValueError, "between 1 and 256 slots");
    return nullptr;
  }
  g_ready = true;
  Py_RETURN_NONE;
}

// set_scratch(device, address): the zeroed slots of a device, and as many that calls hold
PyObject* set_scratch(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  BQ_ARGS(2)
  const long dev = PyLong_AsLong(a[0]);
  const unsigned long long base = PyLong_AsUnsignedLongLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  if (dev >= 0 && dev < kMaxDevices) g_scratch[dev].base.store(base);
  Py_RETURN_NONE;
}

// take_slot(device) -> address of the next slot; counts a launch
PyObject* take_slot_py(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  BQ_ARGS(1)
  const long dev = PyLong_AsLong(a[0]);
  if (PyErr_Occurred()) return nullptr;
  if (dev < 0 || dev >= kMaxDevices || g_scratch[dev].base.load() == 0) {
    PyErr_SetString(PyExc_RuntimeError, "no scratch on this device");
    return nullptr;
  }
  return PyLong_FromVoidPtr(take_slot((int)dev));
}

// next_slot(device) -> index of the slot the next call takes
PyObject* next_slot(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  BQ_ARGS(1)
  const long dev = PyLong_AsLong(a[0]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromUnsignedLong(dev >= 0 && dev < kMaxDevices ? g_scratch[dev].next.load() % g_slots : 0);
}

PyObject* launch_count(PyObject*, PyObject* const*, Py_ssize_t nargs) {
  BQ_ARGS(0)
  return PyLong_FromLongLong(g_launches.load());
}

#define BQ_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {BQ_METHOD("init", init),
                          BQ_METHOD("set_scratch", set_scratch),
                          BQ_METHOD("take_slot", take_slot_py),
                          BQ_METHOD("next_slot", next_slot),
                          BQ_METHOD("launch_count", launch_count),
                          BQ_METHOD("quantize_act", quantize_act),
                          BQ_METHOD("quantize_weight", quantize_weight),
                          BQ_METHOD("rms_norm_quant", rms_norm_quant),
                          BQ_METHOD("gated_rms_norm_quant", gated_rms_norm_quant),
                          BQ_METHOD("sigmoid_gate_quant", sigmoid_gate_quant),
                          BQ_METHOD("linear", linear),
                          BQ_METHOD("matmul", matmul),
                          BQ_METHOD("project", project),
                          BQ_METHOD("mlp", mlp),
                          BQ_METHOD("lm_head_argmax", lm_head_argmax),
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&kModule); }
