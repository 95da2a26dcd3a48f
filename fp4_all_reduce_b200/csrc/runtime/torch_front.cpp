// Native front end of the torch ops: argument checks, output allocation and the launch of one call in one C++ function,
// for the Python wrappers (`ops/codec.py`, `ops/gemm.py`, `parallel/context.py`) and for `torch.ops.fp4ar.*`.
//
// Why it exists: with the checks in Python and the C interface reached through ctypes a call cost 13 - 28 us of host time
// (encode 15.6, add_rmsnorm through its custom op 18.2, decode_sum of eight sources 23.7, reduce_reencode 24.6 - 31, a
// fused block 17.4, a GEMM 14.9), which is what every call of fewer than about 2000 rows then takes, several times the
// device time of its kernel.  What is left here is the allocation of the outputs and the launch itself.
//
// Loaded as the extension module `_fp4ar_front` (see `_native.front()`).  The C interface is bound at run time from the
// library that `_native.cuda()` loaded, so there is one copy of its state whatever FP4AR_LIBRARY names.
#include <Python.h>
#include <dlfcn.h>
#include <string>
#include <vector>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/library.h>
#include "../include/fp4ar.h"
#include "../include/fp4ar_gemm.h"

namespace {

using at::Tensor;

constexpr int64_t kHidden = FP4AR_HIDDEN, kQRow = FP4AR_QROW_BYTES, kMxRow = FP4AR_MXROW_BYTES, kRec = FP4AR_REC_STRIDE;
constexpr int64_t kValues = kHidden / 2;

// ---- the C interface ----
struct Api {
  decltype(&fp4ar_launch) launch;
  decltype(&fp4ar_last_cuda_error) last_error;
  decltype(&fp4ar_encode) encode;
  decltype(&fp4ar_encode_static) encode_static;
  decltype(&fp4ar_decode_sum) decode_sum;
  decltype(&fp4ar_reduce_reencode) reduce_reencode;
  decltype(&fp4ar_add_rmsnorm) add_rmsnorm;
  decltype(&fp4ar_gemm_nvfp4) gemm;
};
Api api{};
PyObject* check_rc = nullptr;      // _native.check(rc, what): raises the Python error of a return code

template <class F>
bool bind(void* lib, const char* name, F& f) {
  f = reinterpret_cast<F>(dlsym(lib, name));
  return f != nullptr;
}

// ---- checks, with the messages users of the Python wrappers know ----
std::string dtype_name(at::ScalarType t) { return std::string("torch.") + torch::getTHPDtype(t)->name; }
std::string shape_text(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); i++) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + (t.dim() == 1 ? ",)" : ")");
}
[[noreturn]] void bad_layout(const Tensor& t, at::ScalarType dtype, int64_t cols, const char* name) {
  if (t.scalar_type() != dtype) TORCH_CHECK_VALUE(false, name, " must be ", dtype_name(dtype), ", got ", dtype_name(t.scalar_type()));
  if (cols >= 0 && (t.dim() != 2 || t.size(1) != cols))
    TORCH_CHECK_VALUE(false, name, " must have shape [rows, ", cols, "], got ", shape_text(t));
  if (!t.is_contiguous()) TORCH_CHECK_VALUE(false, name, " must be contiguous");
  TORCH_CHECK_VALUE(false, name, " must be a CUDA tensor");
}
inline bool layout_ok(const Tensor& t, at::ScalarType dtype, int64_t cols) {
  return t.scalar_type() == dtype && (cols < 0 || (t.dim() == 2 && t.size(1) == cols)) && t.is_contiguous();
}
inline void require(const Tensor& t, at::ScalarType dtype, int64_t cols, const char* name) {
  if (!layout_ok(t, dtype, cols) || !t.is_cuda()) bad_layout(t, dtype, cols, name);
}
// The kernels trust their pointers: every tensor of a call lives on the device that it is launched on.
inline void require_on(const Tensor& t, c10::Device dev, const char* name) {
  TORCH_CHECK_VALUE(t.device() == dev, name, " is on ", t.device(), ", the call runs on ", dev);
}

inline Tensor new_empty(at::IntArrayRef size, at::ScalarType dtype, c10::Device dev) {
  return Tensor(at::detail::empty_cuda(size, dtype, dev, std::nullopt));
}
inline fp4ar_stream stream_of(c10::Device dev) { return (fp4ar_stream)c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

void raise_rc(int rc, const char* what) {
  static const char* names[] = {"ok", "bad argument", "unsupported combination", "CUDA error", "context poisoned"};
  std::string msg = std::string(what) + " failed: " + (rc >= 0 && rc <= 4 ? std::string(names[rc]) : std::to_string(rc));
  if (rc == FP4AR_ERR_CUDA) msg += std::string(": ") + api.last_error();
  throw std::runtime_error(msg);
}
inline void ok(int rc, const char* what) {
  if (rc != FP4AR_OK) raise_rc(rc, what);
}

// ---- one function per op: used by the Python entry points (GIL released) and by torch.ops ----
std::tuple<Tensor, Tensor> op_encode(const Tensor& x) {
  require(x, at::kBFloat16, kHidden, "x");
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t rows = x.size(0);
  Tensor q = new_empty({rows, kQRow}, at::kByte, dev), rs = new_empty({rows}, at::kFloat, dev);
  char* qp = (char*)q.mutable_data_ptr();
  ok(api.encode(x.data_ptr(), (int)rows, qp, kQRow, qp + kValues, kQRow, (float*)rs.mutable_data_ptr(), stream_of(dev)), "fp4ar_encode");
  return {std::move(q), std::move(rs)};
}

Tensor op_encode_static(const Tensor& x, double gs) {
  require(x, at::kBFloat16, kHidden, "x");
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t rows = x.size(0);
  Tensor q = new_empty({rows, kQRow}, at::kByte, dev);
  ok(api.encode_static(x.data_ptr(), (int)rows, (float)gs, q.mutable_data_ptr(), stream_of(dev)), "fp4ar_encode_static");
  return q;
}

// Sources of a decode-sum; row_scales[i] undefined: the static scale gs[i].
struct Sources {
  int n = 0;
  int64_t pitch = 0, rows = 0;
  const void* src[FP4AR_MAX_RANKS];
  const float* rs[FP4AR_MAX_RANKS];
  float gs[FP4AR_MAX_RANKS] = {};
};
Sources sources(const std::vector<Tensor>& q, const std::vector<Tensor>& row_scales, const std::vector<double>& gs, bool have_gs) {
  Sources s;
  TORCH_CHECK_VALUE(!q.empty() && q.size() <= FP4AR_MAX_RANKS, "1..8 sources");
  s.n = (int)q.size();
  s.pitch = q[0].dim() == 2 ? q[0].size(1) : -1;
  if (s.pitch < 0) bad_layout(q[0], at::kByte, kQRow, "source");
  for (const Tensor& t : q) {
    require(t, at::kByte, s.pitch, "source");
    require_on(t, q[0].device(), "source");
    TORCH_CHECK_VALUE(t.sizes() == q[0].sizes(), "sources must have one shape");
  }
  TORCH_CHECK_VALUE(s.pitch == kQRow || s.pitch == kRec, "source rows must be 3456 B (NVFP4 rows) or 3584 B (receive records)");
  TORCH_CHECK_INDEX(row_scales.empty() || row_scales.size() >= q.size(), "list index out of range");
  s.rows = q[0].size(0);
  for (int i = 0; i < s.n; i++) {
    s.src[i] = q[i].data_ptr();
    s.rs[i] = nullptr;
    if (!row_scales.empty() && row_scales[i].defined()) {
      require(row_scales[i], at::kFloat, -1, "row_scales");
      require_on(row_scales[i], q[0].device(), "row_scales");
      TORCH_CHECK_VALUE(row_scales[i].numel() >= s.rows, "row_scales must have ", s.rows, " elements, got ", row_scales[i].numel());
      s.rs[i] = (const float*)row_scales[i].data_ptr();
    } else {
      TORCH_CHECK_VALUE(have_gs, "a source without row scales needs a static scale");
      s.gs[i] = (float)gs[i];
    }
  }
  return s;
}

Tensor op_decode_sum(const std::vector<Tensor>& q, const std::vector<Tensor>& row_scales, const std::vector<double>& gs, bool have_gs) {
  const Sources s = sources(q, row_scales, gs, have_gs);
  const c10::Device dev = q[0].device();
  const c10::cuda::CUDAGuard guard(dev);
  Tensor out = new_empty({s.rows, kHidden}, at::kBFloat16, dev);
  ok(api.decode_sum(s.n, s.src, s.pitch, s.rs, s.gs, (int)s.rows, out.mutable_data_ptr(), stream_of(dev)), "fp4ar_decode_sum");
  return out;
}

std::tuple<Tensor, Tensor> op_reduce_reencode(const std::vector<Tensor>& q, const std::vector<Tensor>& row_scales,
                                              const std::vector<double>& gs, bool have_gs) {
  const Sources s = sources(q, row_scales, gs, have_gs);
  const c10::Device dev = q[0].device();
  const c10::cuda::CUDAGuard guard(dev);
  Tensor rec = new_empty({s.rows, kRec}, at::kByte, dev);      // the kernel writes whole records, their zero tail included
  Tensor out = new_empty({s.rows, kHidden}, at::kBFloat16, dev);
  ok(api.reduce_reencode(s.n, s.src, s.pitch, s.rs, s.gs, (int)s.rows, rec.mutable_data_ptr(), out.mutable_data_ptr(), stream_of(dev)),
     "fp4ar_reduce_reencode");
  return {std::move(rec), std::move(out)};
}

// `out` undefined: allocated; given: any contiguous memory of the device that holds the rows.  `inplace`: the updated
// residual replaces `residual`.
std::tuple<Tensor, Tensor> op_norm(const Tensor& x, const Tensor& residual, const Tensor& weight, double eps, double weight_bias,
                                   int64_t epilogue, double qscale, bool inplace, Tensor out) {
  require(x, at::kBFloat16, kHidden, "x");
  require(residual, at::kBFloat16, kHidden, "residual");
  TORCH_CHECK_VALUE(weight.scalar_type() == at::kBFloat16 && weight.numel() == kHidden && weight.is_cuda() && weight.is_contiguous(),
                    "weight must be a contiguous CUDA BF16 tensor of 6144 elements");
  const int64_t rows = x.size(0);
  TORCH_CHECK_VALUE(residual.size(0) >= rows, "residual must have ", rows, " rows, got ", residual.size(0));
  TORCH_CHECK_VALUE(epilogue >= FP4AR_EPI_NORM_BF16 && epilogue <= FP4AR_EPI_NORM_MXFP8, "epilogue must be 1 (BF16), 2 (NVFP4) or 3 (MXFP8)");
  const c10::Device dev = x.device();
  require_on(residual, dev, "residual");
  require_on(weight, dev, "weight");
  const bool bf16 = epilogue == FP4AR_EPI_NORM_BF16;
  const int64_t cols = bf16 ? kHidden : epilogue == FP4AR_EPI_NORM_NVFP4 ? kQRow : kMxRow;
  if (out.defined()) {
    const int64_t bytes = rows * cols * (bf16 ? 2 : 1);
    TORCH_CHECK_VALUE(out.device() == dev && out.is_contiguous() && (int64_t)out.nbytes() >= bytes,
                      "out must be contiguous, on ", dev, " and hold ", bytes, " bytes");
  }
  const c10::cuda::CUDAGuard guard(dev);
  Tensor res_out = inplace ? residual : new_empty(residual.sizes(), at::kBFloat16, dev);
  if (!out.defined()) out = new_empty({rows, cols}, bf16 ? at::kBFloat16 : at::kByte, dev);
  void* op = out.mutable_data_ptr();
  ok(api.add_rmsnorm(x.data_ptr(), residual.data_ptr(), res_out.mutable_data_ptr(), weight.data_ptr(), (float)eps, (float)weight_bias,
                     (int)epilogue, (float)qscale, bf16 ? op : nullptr, bf16 ? nullptr : op, (int)rows, stream_of(dev)),
     "fp4ar_add_rmsnorm");
  return {std::move(out), std::move(res_out)};
}

std::tuple<Tensor, Tensor> op_gemm(const Tensor& x, const Tensor& wt, double gs, bool want_acc, Tensor q) {
  TORCH_CHECK_VALUE(x.is_cuda() && wt.is_cuda() && x.scalar_type() == at::kBFloat16 && wt.scalar_type() == at::kBFloat16,
                    "x and wt must be CUDA BF16 tensors");
  TORCH_CHECK_VALUE(x.dim() == 2 && wt.dim() == 2 && x.size(1) == wt.size(1) && x.is_contiguous() && wt.is_contiguous(),
                    "x [M, K] and wt [N, K] must be contiguous with equal K");
  const int64_t M = x.size(0), K = x.size(1), Nn = wt.size(0);
  TORCH_CHECK_VALUE(K % 64 == 0 && Nn % 256 == 0, "K must be a multiple of 64 and N a multiple of 256");
  const c10::Device dev = x.device();
  require_on(wt, dev, "wt");
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t qb = Nn / 2 + Nn / 16;
  if (!q.defined()) {
    q = new_empty({M, qb}, at::kByte, dev);
  } else {
    TORCH_CHECK_VALUE(layout_ok(q, at::kByte, qb) && q.size(0) == M && q.device() == dev,
                      "out must be a contiguous uint8 [M, N/2 + N/16] tensor on the device of x");
  }
  Tensor acc;
  if (want_acc) acc = new_empty({M, Nn}, at::kFloat, dev);
  ok(api.gemm(nullptr, 0, x.data_ptr(), wt.data_ptr(), (int)M, (int)Nn, (int)K, (float)gs, q.mutable_data_ptr(),
              want_acc ? (float*)acc.mutable_data_ptr() : nullptr, stream_of(dev)), "fp4ar_gemm_nvfp4");
  return {std::move(q), std::move(acc)};
}

// ---- torch.ops.fp4ar.* (the schemas are defined in ops/allreduce.py) ----
Tensor lib_decode_sum(const std::vector<Tensor>& q, const std::vector<Tensor>& rs) { return op_decode_sum(q, rs, {}, false); }
Tensor lib_add_rms_norm(const Tensor& x, Tensor& residual, const Tensor& weight, double eps, double weight_bias) {
  return std::get<0>(op_norm(x, residual, weight, eps, weight_bias, FP4AR_EPI_NORM_BF16, 1.0, true, Tensor()));
}
Tensor lib_linear(const Tensor& x, const Tensor& wt, double gs) { return std::get<0>(op_gemm(x, wt, gs, false, Tensor())); }

// ---- Python entry points: positional arguments only, the wrappers fill in the defaults ----
const Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) throw torch::TypeError(std::string(name) + " must be a tensor, got " + Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
double double_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
int64_t int_arg(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
bool bool_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
void arity(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) throw torch::TypeError("expected " + std::to_string(want) + " arguments, got " + std::to_string(got));
}
PyObject* wrap2(Tensor a, Tensor b) {
  THPObjectPtr t(PyTuple_New(2));
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t.get(), 0, THPVariable_Wrap(std::move(a)));
  PyTuple_SET_ITEM(t.get(), 1, THPVariable_Wrap(std::move(b)));
  return t.release();
}
struct NoGil {
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};

PyObject* py_encode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 1);
  const Tensor& x = tensor_arg(a[0], "x");
  auto r = [&] { NoGil g; return op_encode(x); }();
  return wrap2(std::move(std::get<0>(r)), std::move(std::get<1>(r)));
  END_HANDLE_TH_ERRORS
}
PyObject* py_encode_static(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 2);
  const Tensor& x = tensor_arg(a[0], "x");
  const double gs = double_arg(a[1]);
  return THPVariable_Wrap([&] { NoGil g; return op_encode_static(x, gs); }());
  END_HANDLE_TH_ERRORS
}
template <class F>
void each(PyObject* seq, F&& f) {
  THPObjectPtr fast(PySequence_Fast(seq, "expected a sequence"));
  if (!fast) throw python_error();
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast.get());
  for (Py_ssize_t i = 0; i < n; i++) f(PySequence_Fast_GET_ITEM(fast.get(), i));
}
// (qrows, row_scales or None, gs or None).  Only the static scales of sources without row scales are looked at: the entries
// of the others may be anything, None among them.
struct SourceArgs {
  std::vector<Tensor> q, rs;
  std::vector<double> gs;
  bool have_gs;
  SourceArgs(PyObject* const* a) : have_gs(a[2] != Py_None) {
    q.reserve(FP4AR_MAX_RANKS);
    each(a[0], [&](PyObject* o) { q.push_back(tensor_arg(o, "source")); });
    if (a[1] != Py_None) {
      rs.reserve(FP4AR_MAX_RANKS);
      each(a[1], [&](PyObject* o) { if (o == Py_None) rs.emplace_back(); else rs.push_back(tensor_arg(o, "row_scales")); });
    }
    if (!have_gs) return;
    gs.resize(q.size());
    for (size_t i = 0; i < q.size(); i++) {
      if (a[1] != Py_None && (i >= rs.size() || rs[i].defined())) continue;
      THPObjectPtr key(PyLong_FromSize_t(i)), item(key ? PyObject_GetItem(a[2], key.get()) : nullptr);
      if (!item) throw python_error();
      gs[i] = double_arg(item.get());
    }
  }
};
PyObject* py_decode_sum(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 3);
  const SourceArgs s(a);
  return THPVariable_Wrap([&] { NoGil g; return op_decode_sum(s.q, s.rs, s.gs, s.have_gs); }());
  END_HANDLE_TH_ERRORS
}
PyObject* py_reduce_reencode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 3);
  const SourceArgs s(a);
  auto r = [&] { NoGil g; return op_reduce_reencode(s.q, s.rs, s.gs, s.have_gs); }();
  return wrap2(std::move(std::get<0>(r)), std::move(std::get<1>(r)));
  END_HANDLE_TH_ERRORS
}
// (x, residual, weight, eps, weight_bias, epilogue, qscale, inplace_residual, out or None)
PyObject* py_add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 9);
  const Tensor &x = tensor_arg(a[0], "x"), &res = tensor_arg(a[1], "residual"), &w = tensor_arg(a[2], "weight");
  const double eps = double_arg(a[3]), wb = double_arg(a[4]), qs = double_arg(a[6]);
  const int64_t epi = int_arg(a[5]);
  const bool inplace = bool_arg(a[7]);
  Tensor out = a[8] == Py_None ? Tensor() : tensor_arg(a[8], "out");
  auto r = [&] { NoGil g; return op_norm(x, res, w, eps, wb, epi, qs, inplace, std::move(out)); }();
  return wrap2(std::move(std::get<0>(r)), std::move(std::get<1>(r)));
  END_HANDLE_TH_ERRORS
}
// (x, wt, gs, want_acc, out or None): q, or (q, acc)
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 5);
  const Tensor &x = tensor_arg(a[0], "x"), &wt = tensor_arg(a[1], "wt");
  const double gs = double_arg(a[2]);
  const bool acc = bool_arg(a[3]);
  Tensor out = a[4] == Py_None ? Tensor() : tensor_arg(a[4], "out");
  auto r = [&] { NoGil g; return op_gemm(x, wt, gs, acc, std::move(out)); }();
  if (!acc) return THPVariable_Wrap(std::move(std::get<0>(r)));
  return wrap2(std::move(std::get<0>(r)), std::move(std::get<1>(r)));
  END_HANDLE_TH_ERRORS
}

// ---- fused calls of a context ----
// Holds what a call needs of an Fp4ArContext.  Its methods take the plain, valid call and return None for everything
// else (an argument that does not fit, a tensor subclass): the Python wrapper then goes through its own checks, which
// name what is wrong.
struct FrontContext {
  PyObject_HEAD
  fp4ar_ctx* ctx;
  int nranks, device, compute_only;
  int64_t max_rows;
};

inline const Tensor* plain(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
inline bool on(const Tensor& t, int device) { return t.is_cuda() && t.device().index() == device; }
inline bool rows_ok(const Tensor* t, at::ScalarType dtype, int64_t rows, int64_t cols, int device) {
  return t && layout_ok(*t, dtype, cols) && t->size(0) == rows && on(*t, device);
}
inline bool get_int(PyObject* o, int& v) {
  if (!PyLong_Check(o)) return false;
  int over = 0;
  const long l = PyLong_AsLongAndOverflow(o, &over);
  v = (int)l;
  return !over && l == (long)v;
}
inline bool get_float(PyObject* o, float& v) {
  if (PyFloat_Check(o)) {
    v = (float)PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (!PyLong_CheckExact(o)) return false;
  const double d = PyLong_AsDouble(o);
  v = (float)d;
  if (d != -1.0 || !PyErr_Occurred()) return true;
  PyErr_Clear();                 // beyond a double: the Python wrapper raises it
  return false;
}

// The input (BF16 rows or NVFP4 rows with one positive scale per rank) and the options every call has.
bool call_input(const FrontContext* c, PyObject* x_, PyObject* gs, PyObject* algo, PyObject* mode, PyObject* teams, fp4ar_args& a,
                const Tensor*& x) {
  x = plain(x_);
  if (!x || !on(*x, c->device) || !x->is_contiguous() || x->dim() != 2 || x->size(0) > c->max_rows) return false;
  if (x->scalar_type() == at::kBFloat16 && x->size(1) == kHidden) a.input = FP4AR_IN_BF16;
  else if (x->scalar_type() == at::kByte && x->size(1) == kQRow) a.input = FP4AR_IN_NVFP4;
  else return false;
  for (float& g : a.gs) g = 1.0f;
  if (a.input == FP4AR_IN_NVFP4) {
    if (!PyList_Check(gs) && !PyTuple_Check(gs)) return false;
    if (PySequence_Fast_GET_SIZE(gs) != c->nranks) return false;
    for (int r = 0; r < c->nranks; r++)
      if (!get_float(PySequence_Fast_GET_ITEM(gs, r), a.gs[r]) || !(a.gs[r] > 0.0f)) return false;
  }
  if (!get_int(algo, a.algo) || !get_int(mode, a.mode) || !get_int(teams, a.tune[0])) return false;
  if (c->compute_only && a.mode != FP4AR_MODE_COMPUTE) return false;
  a.x = x->data_ptr();
  a.rows = (int)x->size(0);
  a.hidden = FP4AR_HIDDEN;
  return true;
}
int launch(const FrontContext* c, const fp4ar_args& a) {
  NoGil g;
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)c->device);
  return api.launch(c->ctx, &a, stream_of(c10::Device(c10::kCUDA, (c10::DeviceIndex)c->device)));
}
void launched(int rc) {
  if (rc == FP4AR_OK) return;
  THPObjectPtr r(PyObject_CallFunction(check_rc, "is", rc, "fp4ar_launch"));
  if (!r) throw python_error();
}

// (x, out or None, gs or None, algo, mode, teams)
PyObject* ctx_all_reduce(PyObject* self, PyObject* const* p, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 6);
  const FrontContext* c = (const FrontContext*)self;
  fp4ar_args a{};
  const Tensor* x;
  if (!call_input(c, p[0], p[2], p[3], p[4], p[5], a, x)) Py_RETURN_NONE;
  Tensor out;
  if (p[1] == Py_None) {
    out = new_empty({a.rows, kHidden}, at::kBFloat16, x->device());
  } else {
    if (!rows_ok(plain(p[1]), at::kBFloat16, a.rows, kHidden, c->device)) Py_RETURN_NONE;
    out = THPVariable_Unpack(p[1]);
  }
  a.out = out.mutable_data_ptr();
  launched(launch(c, a));
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}
// (x, residual, weight, eps, weight_bias, epilogue, qscale, gs or None, algo, out or None, residual_out or None, mode, teams)
PyObject* ctx_block(PyObject* self, PyObject* const* p, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 13);
  const FrontContext* c = (const FrontContext*)self;
  fp4ar_args a{};
  const Tensor* x;
  if (!call_input(c, p[0], p[7], p[8], p[11], p[12], a, x)) Py_RETURN_NONE;
  if (!get_float(p[3], a.eps) || !get_float(p[4], a.weight_bias) || !get_int(p[5], a.epilogue) || !get_float(p[6], a.qscale)) Py_RETURN_NONE;
  if (a.epilogue < FP4AR_EPI_NORM_BF16 || a.epilogue > FP4AR_EPI_NORM_MXFP8) Py_RETURN_NONE;
  const Tensor *res = plain(p[1]), *w = plain(p[2]);
  if (!rows_ok(res, at::kBFloat16, a.rows, kHidden, c->device)) Py_RETURN_NONE;
  if (!w || w->scalar_type() != at::kBFloat16 || w->numel() != kHidden || !w->is_contiguous() || !on(*w, c->device)) Py_RETURN_NONE;
  const Tensor* res_out = p[10] == Py_None ? res : plain(p[10]);
  if (res_out != res && !rows_ok(res_out, at::kBFloat16, a.rows, kHidden, c->device)) Py_RETURN_NONE;
  const bool bf16 = a.epilogue == FP4AR_EPI_NORM_BF16;
  const int64_t cols = bf16 ? kHidden : (a.epilogue == FP4AR_EPI_NORM_NVFP4 ? kQRow : kMxRow);
  const at::ScalarType dtype = bf16 ? at::kBFloat16 : at::kByte;
  Tensor out;
  if (p[9] == Py_None) {
    out = new_empty({a.rows, cols}, dtype, x->device());
  } else {
    if (!rows_ok(plain(p[9]), dtype, a.rows, cols, c->device)) Py_RETURN_NONE;
    out = THPVariable_Unpack(p[9]);
  }
  (bf16 ? a.out : a.outq) = out.mutable_data_ptr();
  a.res_in = res->data_ptr();
  a.res_out = res_out->mutable_data_ptr();
  a.weight = w->data_ptr();
  launched(launch(c, a));
  return wrap2(std::move(out), *res_out);
  END_HANDLE_TH_ERRORS
}

PyObject* ctx_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long ptr;
  int nranks, device, compute_only;
  long long max_rows;
  if (!PyArg_ParseTuple(args, "KiLip", &ptr, &nranks, &max_rows, &device, &compute_only)) return nullptr;
  FrontContext* c = (FrontContext*)type->tp_alloc(type, 0);
  if (!c) return nullptr;
  c->ctx = (fp4ar_ctx*)(uintptr_t)ptr;
  c->nranks = nranks; c->device = device; c->compute_only = compute_only; c->max_rows = max_rows;
  return (PyObject*)c;
}
PyMethodDef ctx_methods[] = {
    {"all_reduce", (PyCFunction)(void (*)(void))ctx_all_reduce, METH_FASTCALL, nullptr},
    {"block", (PyCFunction)(void (*)(void))ctx_block, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyTypeObject ctx_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// (library path, _native.check): binds the C interface
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  arity(n, 2);
  const char* path = PyUnicode_AsUTF8(a[0]);
  if (!path) throw python_error();
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!lib) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
  const bool all = bind(lib, "fp4ar_launch", api.launch) && bind(lib, "fp4ar_last_cuda_error", api.last_error) &&
                   bind(lib, "fp4ar_encode", api.encode) && bind(lib, "fp4ar_encode_static", api.encode_static) &&
                   bind(lib, "fp4ar_decode_sum", api.decode_sum) && bind(lib, "fp4ar_reduce_reencode", api.reduce_reencode) &&
                   bind(lib, "fp4ar_add_rmsnorm", api.add_rmsnorm) && bind(lib, "fp4ar_gemm_nvfp4", api.gemm);
  if (!all) throw std::runtime_error(std::string(path) + " lacks a function of the C interface");
  Py_INCREF(a[1]);
  Py_XSETREF(check_rc, a[1]);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

#define FP4AR_METHOD(name) {#name, (PyCFunction)(void (*)(void))py_##name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FP4AR_METHOD(bind), FP4AR_METHOD(encode), FP4AR_METHOD(encode_static), FP4AR_METHOD(decode_sum),
                         FP4AR_METHOD(reduce_reencode), FP4AR_METHOD(add_rmsnorm), FP4AR_METHOD(gemm), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fp4ar_front", nullptr, -1, methods};

}  // namespace

TORCH_LIBRARY_IMPL(fp4ar, CUDA, m) {
  m.impl("encode", op_encode);
  m.impl("encode_static", op_encode_static);
  m.impl("decode_sum", lib_decode_sum);
  m.impl("add_rms_norm", lib_add_rms_norm);
  m.impl("linear_nvfp4", lib_linear);
}

PyMODINIT_FUNC PyInit__fp4ar_front() {
  ctx_type.tp_name = "_fp4ar_front.Context";
  ctx_type.tp_basicsize = sizeof(FrontContext);
  ctx_type.tp_flags = Py_TPFLAGS_DEFAULT;
  ctx_type.tp_methods = ctx_methods;
  ctx_type.tp_new = ctx_new;
  if (PyType_Ready(&ctx_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (!m) return nullptr;
  Py_INCREF(&ctx_type);
  if (PyModule_AddObject(m, "Context", (PyObject*)&ctx_type) < 0) return nullptr;
  return m;
}
