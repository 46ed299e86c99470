// Python boundary of the tensor-level operators (faith_b200/ops.py): argument checks, output allocation, the current
// stream and the C-ABI call in one native function per operator.
//
// What bounds the small calls is the host, not the GPU: an operator of a single sentence is two or three launches of 2 to 10 us,
// and the same steps written in Python over ctypes (attribute checks of every tensor, a device context manager, four
// empty_like calls, the conversion of 10 to 25 arguments) took 25 to 40 us per operator.  The functions here take their
// arguments through the vectorcall protocol (no tuple, no keyword parsing), read the tensors' fields directly and allocate
// from torch's caching allocator without the dispatcher.
//
// No arithmetic happens here and nothing is kept from one call to the next.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cmath>

#include "faith_b200.h"

namespace {

PyObject* g_error = nullptr;   // faith_b200.FaithError
PyObject* g_check = nullptr;   // faith_b200._lib.check(status, what): raises for a status other than FB_OK

[[noreturn]] void fail(const char* msg) {
  PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, msg);
  throw python_error();
}
[[noreturn]] void fail_with(PyObject* type, const char* fmt, PyObject* arg) {
  PyErr_Format(type, fmt, arg);
  throw python_error();
}

// Raises what faith_b200._lib.check raises for this status.
void check_status(int rc, const char* what) {
  if (rc == FB_OK) return;
  PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, what);
  throw python_error();
}

// The arguments of one call, and the device that all of its tensors share.
class Call {
 public:
  Call(PyObject* const* args, Py_ssize_t n, Py_ssize_t want, const char* name) : args_(args) {
    if (n != want) {
      PyErr_Format(PyExc_TypeError, "%s takes %zd positional arguments, got %zd", name, want, n);
      throw python_error();
    }
  }
  bool none(int i) const { return args_[i] == Py_None; }
  // contiguous float32 tensor on the GPU
  const at::Tensor& tensor(int i) { return accept(args_[i]); }
  const at::Tensor& accept(PyObject* o) {
    if (!THPVariable_Check(o)) fail_with(PyExc_TypeError, "expected a torch.Tensor, got %R", (PyObject*)Py_TYPE(o));
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) fail("faith_b200 operators need CUDA tensors (there is no CPU path)");
    if (t.scalar_type() != at::kFloat) {
      PyObject* d = PyObject_GetAttrString(o, "dtype");
      PyErr_Format(g_error, "float32 tensors required, got %S", d);
      Py_XDECREF(d);
      throw python_error();
    }
    if (!t.is_contiguous()) fail("contiguous tensors required");
    const int dev = t.get_device();
    if (dev_ < 0) dev_ = dev;
    else if (dev != dev_) fail("all tensors must live on one device");
    return t;
  }
  // a tuple or list of `n` tensors starting at out[0]
  void tensors(int i, const at::Tensor** out, int n) {
    PyObject* s = args_[i];
    if (!(PyTuple_Check(s) || PyList_Check(s)) || PySequence_Fast_GET_SIZE(s) != n)
      fail_with(PyExc_TypeError, "expected a tuple of tensors, got %R", s);
    for (int k = 0; k < n; ++k) out[k] = &accept(PySequence_Fast_GET_ITEM(s, k));
  }
  int integer(int i) const {
    const long v = PyLong_AsLong(args_[i]);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    if (v < INT_MIN || v > INT_MAX) {
      PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits");
      throw python_error();
    }
    return (int)v;
  }
  float real(int i) const {
    const double v = PyFloat_AsDouble(args_[i]);
    if (v == -1.0 && PyErr_Occurred()) throw python_error();
    return (float)v;
  }
  // perturbation norm (the reference treats p >= 10 as infinity, Verifier.py:17)
  int norm(int i) const {
    const double p = PyFloat_AsDouble(args_[i]);
    if (p == -1.0 && PyErr_Occurred()) throw python_error();
    if (p == 1.0) return FB_P1;
    if (p == 2.0) return FB_P2;
    if (p >= 10.0) return FB_PINF;
    fail_with(PyExc_ValueError, "only p in {1, 2, inf} is supported, got %R", args_[i]);
  }
  // status word of the caller (may be None)
  int* flag(int i) const {
    if (none(i)) return nullptr;
    if (THPVariable_Check(args_[i])) {
      const at::Tensor& t = THPVariable_Unpack(args_[i]);
      if (t.is_cuda() && t.scalar_type() == at::kInt) return static_cast<int*>(t.data_ptr());
    }
    fail("violation flag must be an int32 CUDA tensor");
  }
  int device() const { return dev_; }

 private:
  PyObject* const* args_;
  int dev_ = -1;
};

inline float* ptr(const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); }
inline float* ptr(const at::Tensor* t) { return t != nullptr ? static_cast<float*>(t->data_ptr()) : nullptr; }

inline at::Tensor empty(at::IntArrayRef sizes, int dev) {
  return at::detail::empty_cuda(sizes, at::kFloat, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt);
}
inline at::Tensor empty_like(const at::Tensor& t) { return empty(t.sizes(), t.get_device()); }
// `t`'s shape with its last dimension replaced
inline at::Tensor empty_last(const at::Tensor& t, int64_t last) {
  c10::SmallVector<int64_t, 6> s(t.sizes().begin(), t.sizes().end());
  s.back() = last;
  return empty(s, t.get_device());
}

// The device of the call made current, its current stream, the GIL released while the launches are enqueued.
class Launch {
 public:
  explicit Launch(int dev) : guard_((c10::DeviceIndex)dev), stream_(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream()) {
    state_ = PyEval_SaveThread();
  }
  ~Launch() { PyEval_RestoreThread(state_); }
  void* stream() const { return (void*)stream_; }
  cudaStream_t cuda() const { return stream_; }

 private:
  c10::cuda::CUDAGuard guard_;
  cudaStream_t stream_;
  PyThreadState* state_;
};

template <size_t N>
PyObject* tuple(const std::array<at::Tensor, N>& ts, PyObject* extra = nullptr) {
  PyObject* out = PyTuple_New((Py_ssize_t)N + (extra != nullptr ? 1 : 0));
  if (out == nullptr) throw python_error();
  for (size_t i = 0; i < N; ++i) PyTuple_SET_ITEM(out, (Py_ssize_t)i, THPVariable_Wrap(ts[i]));
  if (extra != nullptr) PyTuple_SET_ITEM(out, (Py_ssize_t)N, extra);
  return out;
}

// lw, uw, lb, ub at positions i .. i+3
struct Four {
  const at::Tensor *lw, *uw, *lb, *ub;
  Four(Call& c, int i) : lw(&c.tensor(i)), uw(&c.tensor(i + 1)), lb(&c.tensor(i + 2)), ub(&c.tensor(i + 3)) {}
  int64_t rows() const { return lb->size(-1) != 0 ? lb->numel() / lb->size(-1) : 0; }
  int Di() const { return (int)lw->size(-2); }
  int Do() const { return (int)lw->size(-1); }
};

#define FB_FN(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t nargs)

FB_FN(concretize) {   // lw, uw, lb, ub, p, eps, words, layout
  HANDLE_TH_ERRORS
  Call c(args, nargs, 8, "concretize");
  const Four x(c, 0);
  const int p = c.norm(4), words = c.integer(6), layout = c.integer(7);
  const float eps = c.real(5);
  const int Do = (int)x.lb->size(-1), Di = (int)(layout == FB_NATIVE ? x.lw->size(-2) : x.lw->size(-1));
  std::array<at::Tensor, 2> z = {empty_like(*x.lb), empty_like(*x.ub)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_concretize_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), x.rows(), Di, Do, words, p, eps,
                           layout, l.stream());
  }
  check_status(rc, "fb_concretize_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(relax) {   // op, lw, uw, lb, ub, p, eps, words, layout, out (None or 4 tensors), violation (None or int32 tensor)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 11, "relax");
  const int op = c.integer(0);
  const Four x(c, 1);
  const int p = c.norm(5), words = c.integer(7), layout = c.integer(8);
  const float eps = c.real(6);
  int* const violation = c.flag(10);
  const int Do = (int)x.lb->size(-1), Di = (int)(layout == FB_NATIVE ? x.lw->size(-2) : x.lw->size(-1));
  std::array<at::Tensor, 4> z;
  if (c.none(9)) {
    z = {empty_like(*x.lw), empty_like(*x.uw), empty_like(*x.lb), empty_like(*x.ub)};
  } else {
    const at::Tensor* o[4];
    c.tensors(9, o, 4);
    for (int i = 0; i < 4; ++i) z[(size_t)i] = *o[i];
  }
  int rc;
  {
    Launch l(c.device());
    rc = fb_relax_f32(op, ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), Di, Do,
                      words, p, eps, layout, violation, l.stream());
  }
  check_status(rc, "fb_relax_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

// The status word of the checked operators: one per host thread, in page-locked memory that the kernels write directly (only
// when something is wrong) and that is read once the stream has been waited for, as the callers that turn the word into an
// exception have to.  A word in device memory took an allocation, a fill and a copy around every such operator: 5 to 8 us of
// the 30 us that the check costs.
class StatusWord {
 public:
  StatusWord() {
    if (cudaHostAlloc(&p_, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) p_ = nullptr;
  }
  ~StatusWord() {
    if (p_ != nullptr) cudaFreeHost(p_);
  }
  StatusWord(const StatusWord&) = delete;
  StatusWord& operator=(const StatusWord&) = delete;
  int* get() const { return static_cast<int*>(p_); }

 private:
  void* p_ = nullptr;
};

template <typename Fn>
int with_status_word(int dev, int* value, const Fn& fn) {
  Launch l(dev);
  static thread_local const StatusWord word;
  int* const w = word.get();
  if (w == nullptr) return FB_ERR_CUDA;
  *static_cast<volatile int*>(w) = 0;   // (no launch that could still write it is left: every call waits for its own)
  const int rc = fn(w, l.stream());
  if (rc != FB_OK) {
    cudaStreamSynchronize(l.cuda());
    return rc;
  }
  if (cudaStreamSynchronize(l.cuda()) != cudaSuccess) return FB_ERR_CUDA;
  *value = *static_cast<volatile int*>(w);
  return FB_OK;
}

FB_FN(relax_checked) {   // op, lw, uw, lb, ub, p, eps, words -> (lw, uw, lb, ub, status word)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 8, "relax_checked");
  const int op = c.integer(0);
  const Four x(c, 1);
  const int p = c.norm(5), words = c.integer(7);
  const float eps = c.real(6);
  const int Do = (int)x.lb->size(-1), Di = x.Di();
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.uw), empty_like(*x.lb), empty_like(*x.ub)};
  int value = 0;
  const int rc = with_status_word(c.device(), &value, [&](int* w, void* st) {
    return fb_relax_f32(op, ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), Di,
                        Do, words, p, eps, FB_NATIVE, w, st);
  });
  check_status(rc, "fb_relax_f32");
  return tuple(z, PyLong_FromLong(value));
  END_HANDLE_TH_ERRORS
}

FB_FN(matmul) {   // lw, uw, lb, ub, W, bias (None or tensor)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 6, "matmul");
  const Four x(c, 0);
  const at::Tensor& W = c.tensor(4);
  const at::Tensor* bias = c.none(5) ? nullptr : &c.tensor(5);
  const int Do = x.Do(), Dy = (int)W.size(0);
  if (W.size(1) != Do) {
    PyErr_Format(g_error, "weight shape (%lld, %lld) does not match feature size %d", (long long)W.size(0), (long long)W.size(1), Do);
    throw python_error();
  }
  std::array<at::Tensor, 4> z = {empty_last(*x.lw, Dy), empty_last(*x.lw, Dy), empty_last(*x.lb, Dy), empty_last(*x.lb, Dy)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_matmul_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(W), ptr(bias), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]),
                       x.rows(), x.Di(), Do, Dy, l.stream());
  }
  check_status(rc, "fb_matmul_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(dot_product) {   // x (4), y (4), p, eps, words, out_scale, layout, scratch (None or 4), out (None or 4)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 15, "dot_product");
  const Four x(c, 0), y(c, 4);
  const int p = c.norm(8), words = c.integer(10), layout = c.integer(12);
  const float eps = c.real(9), scale = c.real(11);
  if (x.lb->dim() != 3 || x.lw->dim() != 4) fail("dot_product: bounds of shape [B, L, Di, K] required");
  const int64_t B = x.lb->size(0), Lx = x.lb->size(1), K = x.lb->size(2), Ly = y.lb->size(1);
  const int64_t Di = layout == FB_NATIVE ? x.lw->size(2) : x.lw->size(3);
  std::array<at::Tensor, 4> z, r;
  const at::Tensor* o[4];
  if (c.none(14)) {
    const std::array<int64_t, 4> zs = layout == FB_NATIVE ? std::array<int64_t, 4>{B, Lx, Di, Ly} : std::array<int64_t, 4>{B, Lx, Ly, Di};
    z = {empty(zs, c.device()), empty(zs, c.device()), empty({B, Lx, Ly}, c.device()), empty({B, Lx, Ly}, c.device())};
  } else {
    c.tensors(14, o, 4);
    for (int i = 0; i < 4; ++i) z[(size_t)i] = *o[i];
  }
  if (c.none(13)) {
    r = {empty_like(*x.lb), empty_like(*x.lb), empty_like(*y.lb), empty_like(*y.lb)};
  } else {
    c.tensors(13, o, 4);
    for (int i = 0; i < 4; ++i) r[(size_t)i] = *o[i];
  }
  int rc;
  {
    Launch l(c.device());
    rc = fb_dot_product_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(y.lw), ptr(y.uw), ptr(y.lb), ptr(y.ub), ptr(z[0]),
                            ptr(z[1]), ptr(z[2]), ptr(z[3]), ptr(r[0]), ptr(r[1]), ptr(r[2]), ptr(r[3]), (int)B, (int)Lx, (int)Ly,
                            (int)Di, (int)K, words, p, eps, scale, layout, l.stream());
  }
  check_status(rc, "fb_dot_product_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

// x (4) [B, Lx, Di, K], v (4) [B, K, Di, Ly], p, eps, words, out_scale, merge_heads; None when the shape is not one of
// fb_context_heads_f32's (the caller transposes v and takes dot_product).
FB_FN(context_kmajor) {
  HANDLE_TH_ERRORS
  Call c(args, nargs, 13, "context_kmajor");
  const Four x(c, 0), v(c, 4);
  const int p = c.norm(8), words = c.integer(10), heads = c.integer(12);
  const float eps = c.real(9), scale = c.real(11);
  if (x.lb->dim() != 3 || x.lw->dim() != 4 || v.lb->dim() != 3 || heads < 1) fail("context: bounds of shape [B, L, Di, K] required");
  const int64_t B = x.lb->size(0), Lx = x.lb->size(1), K = x.lb->size(2), Ly = v.lb->size(2), Di = x.lw->size(2), S = B / heads;
  std::array<at::Tensor, 4> z = {empty({S, Lx, Di, heads * Ly}, c.device()), empty({S, Lx, Di, heads * Ly}, c.device()),
                                 empty({S, Lx, heads * Ly}, c.device()), empty({S, Lx, heads * Ly}, c.device())};
  const std::array<at::Tensor, 4> r = {empty_like(*x.lb), empty_like(*x.lb), empty({B, Ly, K}, c.device()), empty({B, Ly, K}, c.device())};
  int rc;
  {
    Launch l(c.device());
    rc = fb_context_heads_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(v.lw), ptr(v.uw), ptr(v.lb), ptr(v.ub), ptr(z[0]),
                              ptr(z[1]), ptr(z[2]), ptr(z[3]), ptr(r[0]), ptr(r[1]), ptr(r[2]), ptr(r[3]), (int)B, (int)Lx, (int)Ly,
                              (int)Di, (int)K, words, p, eps, scale, heads, l.stream());
  }
  if (rc == FB_ERR_SHAPE) Py_RETURN_NONE;
  check_status(rc, "fb_context_heads_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

// x (4) [B, Lx, Di, K], v (4) [B, K, Di, Ly], p, eps, words; None when the shape is not one of fb_context_f32's
FB_FN(context) {
  HANDLE_TH_ERRORS
  Call c(args, nargs, 11, "context");
  const Four x(c, 0), v(c, 4);
  const int p = c.norm(8), words = c.integer(10);
  const float eps = c.real(9);
  if (x.lb->dim() != 3 || x.lw->dim() != 4 || v.lb->dim() != 3) fail("context: bounds of shape [B, L, Di, K] required");
  const int64_t B = x.lb->size(0), Lx = x.lb->size(1), K = x.lb->size(2), Ly = v.lb->size(2), Di = x.lw->size(2);
  std::array<at::Tensor, 4> z = {empty({B, Lx, Di, Ly}, c.device()), empty({B, Lx, Di, Ly}, c.device()), empty({B, Lx, Ly}, c.device()),
                                 empty({B, Lx, Ly}, c.device())};
  const std::array<at::Tensor, 4> r = {empty_like(*x.lb), empty_like(*x.lb), empty({B, Ly, K}, c.device()), empty({B, Ly, K}, c.device())};
  int rc;
  {
    Launch l(c.device());
    rc = fb_context_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(v.lw), ptr(v.uw), ptr(v.lb), ptr(v.ub), ptr(z[0]), ptr(z[1]),
                        ptr(z[2]), ptr(z[3]), ptr(r[0]), ptr(r[1]), ptr(r[2]), ptr(r[3]), (int)B, (int)Lx, (int)Ly, (int)Di, (int)K,
                        words, p, eps, 1.0f, 1, l.stream());
  }
  if (rc == FB_ERR_SHAPE) Py_RETURN_NONE;
  check_status(rc, "fb_context_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(mul_bounds) {   // x (4), y (4), p, eps, words
  HANDLE_TH_ERRORS
  Call c(args, nargs, 11, "mul_bounds");
  const Four x(c, 0), y(c, 4);
  const int p = c.norm(8), words = c.integer(10);
  const float eps = c.real(9);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_mul_bounds_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(y.lw), ptr(y.uw), ptr(y.lb), ptr(y.ub), ptr(z[0]),
                           ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), x.Di(), x.Do(), words, p, eps, l.stream());
  }
  check_status(rc, "fb_mul_bounds_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(add) {   // x (4), y (4)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 8, "add");
  const Four x(c, 0), y(c, 4);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_add_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(y.lw), ptr(y.uw), ptr(y.lb), ptr(y.ub), ptr(z[0]), ptr(z[1]),
                    ptr(z[2]), ptr(z[3]), x.rows(), x.Di(), x.Do(), l.stream());
  }
  check_status(rc, "fb_add_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(scale) {   // x (4), c
  HANDLE_TH_ERRORS
  Call c(args, nargs, 5, "scale");
  const Four x(c, 0);
  const float f = c.real(4);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_scale_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), x.Di(),
                      x.Do(), f, l.stream());
  }
  check_status(rc, "fb_scale_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(mul_features) {   // x (4), w
  HANDLE_TH_ERRORS
  Call c(args, nargs, 5, "mul_features");
  const Four x(c, 0);
  const at::Tensor& w = c.tensor(4);
  if (w.numel() != x.Do()) {
    PyErr_Format(g_error, "feature vector of %lld elements against %d features", (long long)w.numel(), x.Do());
    throw python_error();
  }
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.uw), empty_like(*x.lb), empty_like(*x.ub)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_mul_features_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(w), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]),
                             x.rows(), x.Di(), x.Do(), l.stream());
  }
  check_status(rc, "fb_mul_features_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(rowsum) {   // x (4)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 4, "rowsum");
  const Four x(c, 0);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_rowsum_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), x.Di(),
                       x.Do(), l.stream());
  }
  check_status(rc, "fb_rowsum_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(layernorm_novar) {   // x (4), gamma, beta, residual (None or 4)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 7, "layernorm_novar");
  const Four x(c, 0);
  const at::Tensor &gamma = c.tensor(4), &beta = c.tensor(5);
  const at::Tensor* r[4] = {nullptr, nullptr, nullptr, nullptr};
  if (!c.none(6)) c.tensors(6, r, 4);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_layernorm_novar_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(r[0]), ptr(r[1]), ptr(r[2]), ptr(r[3]), ptr(gamma),
                                ptr(beta), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), x.Di(), x.Do(), l.stream());
  }
  check_status(rc, "fb_layernorm_novar_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

// x (4), gamma, beta, p, eps, words -> None (not a shape of the fused kernel) or (lw, uw, lb, ub, status word)
FB_FN(layernorm_standard_checked) {
  HANDLE_TH_ERRORS
  Call c(args, nargs, 9, "layernorm_standard_checked");
  const Four x(c, 0);
  const at::Tensor &gamma = c.tensor(4), &beta = c.tensor(5);
  const int p = c.norm(6), words = c.integer(8);
  const float eps = c.real(7);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.lw), empty_like(*x.lb), empty_like(*x.lb)};
  int value = 0;
  const int rc = with_status_word(c.device(), &value, [&](int* w, void* st) {
    return fb_layernorm_standard_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(gamma), ptr(beta), ptr(z[0]), ptr(z[1]),
                                     ptr(z[2]), ptr(z[3]), x.rows(), x.Di(), x.Do(), words, p, eps, w, st);
  });
  if (rc == FB_ERR_SHAPE) Py_RETURN_NONE;
  check_status(rc, "fb_layernorm_standard_f32");
  return tuple(z, PyLong_FromLong(value));
  END_HANDLE_TH_ERRORS
}

FB_FN(split_heads) {   // x (4) [B, L, Di, H * d], heads, transpose_ld
  HANDLE_TH_ERRORS
  Call c(args, nargs, 6, "split_heads");
  const Four x(c, 0);
  const int H = c.integer(4), tr = c.integer(5);
  if (x.lw->dim() != 4 || H < 1) fail("split_heads: bounds of shape [B, L, Di, H * d] required");
  const int64_t B = x.lw->size(0), L = x.lw->size(1), Di = x.lw->size(2), d = x.lw->size(3) / H;
  const std::array<int64_t, 4> ws = tr ? std::array<int64_t, 4>{B * H, d, Di, L} : std::array<int64_t, 4>{B * H, L, Di, d};
  const std::array<int64_t, 3> bs = tr ? std::array<int64_t, 3>{B * H, d, L} : std::array<int64_t, 3>{B * H, L, d};
  std::array<at::Tensor, 4> z = {empty(ws, c.device()), empty(ws, c.device()), empty(bs, c.device()), empty(bs, c.device())};
  int rc;
  {
    Launch l(c.device());
    rc = fb_split_heads_bound_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), (int)B,
                                  (int)L, (int)Di, H, (int)d, tr, l.stream());
  }
  check_status(rc, "fb_split_heads_bound_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(merge_heads) {   // x (4) [B * H, L, Di, d], heads
  HANDLE_TH_ERRORS
  Call c(args, nargs, 5, "merge_heads");
  const Four x(c, 0);
  const int H = c.integer(4);
  if (x.lw->dim() != 4 || H < 1) fail("merge_heads: bounds of shape [B * H, L, Di, d] required");
  const int64_t B = x.lw->size(0) / H, L = x.lw->size(1), Di = x.lw->size(2), d = x.lw->size(3);
  std::array<at::Tensor, 4> z = {empty({B, L, Di, H * d}, c.device()), empty({B, L, Di, H * d}, c.device()),
                                 empty({B, L, H * d}, c.device()), empty({B, L, H * d}, c.device())};
  int rc;
  {
    Launch l(c.device());
    rc = fb_merge_heads_bound_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), (int)B,
                                  (int)L, (int)Di, H, (int)d, l.stream());
  }
  check_status(rc, "fb_merge_heads_bound_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

FB_FN(conv2d) {   // x (4), weight, bias (None or tensor), stride, padding
  HANDLE_TH_ERRORS
  Call c(args, nargs, 8, "conv2d");
  const Four x(c, 0);
  const at::Tensor& w = c.tensor(4);
  const at::Tensor* bias = c.none(5) ? nullptr : &c.tensor(5);
  const int stride = c.integer(6), pad = c.integer(7);
  if (x.lw->dim() != 5 || w.dim() != 4) fail("conv2d: bounds of shape [B, Di, C, H, W] and a weight [Co, Ci, Kh, Kw] required");
  const int64_t B = x.lw->size(0), Di = x.lw->size(1), C = x.lw->size(2), H = x.lw->size(3), W = x.lw->size(4);
  const int64_t Co = w.size(0), Kh = w.size(2), Kw = w.size(3);
  if (w.size(1) != C) {
    PyErr_Format(g_error, "conv weight expects %lld input channels, bounds have %lld", (long long)w.size(1), (long long)C);
    throw python_error();
  }
  if (stride == 0) {
    PyErr_SetString(PyExc_ZeroDivisionError, "integer division or modulo by zero");
    throw python_error();
  }
  auto out_size = [&](int64_t n, int64_t k) {   // rounds down, as Python's //
    const int64_t v = n + 2 * pad - k;
    return (v >= 0 ? v / stride : -((-v + stride - 1) / stride)) + 1;
  };
  const int64_t Ho = out_size(H, Kh), Wo = out_size(W, Kw);
  std::array<at::Tensor, 4> z = {empty({B, Di, Co, Ho, Wo}, c.device()), empty({B, Di, Co, Ho, Wo}, c.device()),
                                 empty({B, Co, Ho, Wo}, c.device()), empty({B, Co, Ho, Wo}, c.device())};
  int rc;
  {
    Launch l(c.device());
    rc = fb_conv2d_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(w), ptr(bias), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]),
                       (int)B, (int)Di, (int)C, (int)H, (int)W, (int)Co, (int)Kh, (int)Kw, stride, pad, l.stream());
  }
  check_status(rc, "fb_conv2d_f32");
  return tuple(z);
  END_HANDLE_TH_ERRORS
}

// x (4), p, eps, words, violation (None or int32 tensor), ranges: None when the shape needs the unfused chain
FB_FN(softmax) {
  HANDLE_TH_ERRORS
  Call c(args, nargs, 9, "softmax");
  const Four x(c, 0);
  const int p = c.norm(4), words = c.integer(6);
  const float eps = c.real(5);
  int* const violation = c.flag(7);
  const bool ranges = PyObject_IsTrue(args[8]) == 1;
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.uw), empty_like(*x.lb), empty_like(*x.ub)};
  std::array<at::Tensor, 2> r;
  if (ranges) r = {empty_like(*x.lb), empty_like(*x.ub)};
  int rc;
  {
    Launch l(c.device());
    rc = fb_softmax_ranges_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]),
                               ranges ? ptr(r[0]) : nullptr, ranges ? ptr(r[1]) : nullptr, x.rows(), x.Di(), x.Do(), words, p, eps,
                               violation, l.stream());
  }
  if (rc == FB_ERR_SHAPE || rc == FB_ERR_ALIGN) Py_RETURN_NONE;
  check_status(rc, "fb_softmax_ranges_f32");
  if (!ranges) return tuple(z);
  return tuple(std::array<at::Tensor, 6>{z[0], z[1], z[2], z[3], r[0], r[1]});
  END_HANDLE_TH_ERRORS
}

FB_FN(softmax_checked) {   // x (4), p, eps, words -> None or (lw, uw, lb, ub, status word)
  HANDLE_TH_ERRORS
  Call c(args, nargs, 7, "softmax_checked");
  const Four x(c, 0);
  const int p = c.norm(4), words = c.integer(6);
  const float eps = c.real(5);
  std::array<at::Tensor, 4> z = {empty_like(*x.lw), empty_like(*x.uw), empty_like(*x.lb), empty_like(*x.ub)};
  int value = 0;
  const int rc = with_status_word(c.device(), &value, [&](int* w, void* st) {
    return fb_softmax_f32(ptr(x.lw), ptr(x.uw), ptr(x.lb), ptr(x.ub), ptr(z[0]), ptr(z[1]), ptr(z[2]), ptr(z[3]), x.rows(), x.Di(),
                          x.Do(), words, p, eps, w, st);
  });
  if (rc == FB_ERR_SHAPE || rc == FB_ERR_ALIGN) Py_RETURN_NONE;
  check_status(rc, "fb_softmax_f32");
  return tuple(z, PyLong_FromLong(value));
  END_HANDLE_TH_ERRORS
}

// net (address of an fb_cnn), image [C, H, W], p, eps, first row, rows, communicator (address or None), all-reduce, compact,
// features of the last layer, arena (uint8 tensor) -> [2, features]: lower and upper ends of the range
FB_FN(cnn_forward) {
  HANDLE_TH_ERRORS
  Call c(args, nargs, 11, "cnn_forward");
  auto address = [&](int i) {
    void* const p = PyLong_AsVoidPtr(args[i]);
    if (p == nullptr && PyErr_Occurred()) throw python_error();
    return p;
  };
  const fb_cnn* const net = static_cast<const fb_cnn*>(address(0));
  const at::Tensor& image = c.tensor(1);
  const int p = c.norm(2), start = c.integer(4), rows = c.integer(5), algo = c.integer(7), compact = c.integer(8), n_out = c.integer(9);
  const float eps = c.real(3);
  fb_comm* const comm = c.none(6) ? nullptr : static_cast<fb_comm*>(address(6));
  if (image.numel() != (int64_t)net->cin * net->h * net->w) fail("cnn_forward: the image is not of the network's input shape");
  if (!THPVariable_Check(args[10])) fail("cnn_forward: arena tensor required");
  const at::Tensor& arena = THPVariable_Unpack(args[10]);
  if (!arena.is_cuda() || arena.scalar_type() != at::kByte || arena.get_device() != c.device()) fail("cnn_forward: arena of the image's device required");
  at::Tensor out = empty({2, n_out}, c.device());
  int rc;
  {
    Launch l(c.device());
    rc = fb_cnn_forward_f32(net, ptr(image), p, eps, start, rows, comm, algo, compact, ptr(out), ptr(out) + n_out, nullptr,
                            arena.data_ptr(), arena.numel(), l.stream());
  }
  check_status(rc, "fb_cnn_forward_f32");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

FB_FN(setup) {   // FaithError, _lib.check
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "setup takes 2 arguments");
    return nullptr;
  }
  Py_INCREF(args[0]);
  Py_INCREF(args[1]);
  Py_XSETREF(g_error, args[0]);
  Py_XSETREF(g_check, args[1]);
  Py_RETURN_NONE;
}

#define FB_DEF(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {FB_DEF(setup), FB_DEF(concretize), FB_DEF(relax), FB_DEF(relax_checked), FB_DEF(matmul), FB_DEF(dot_product),
                          FB_DEF(context_kmajor), FB_DEF(context), FB_DEF(mul_bounds), FB_DEF(add), FB_DEF(scale), FB_DEF(mul_features), FB_DEF(rowsum),
                          FB_DEF(layernorm_novar), FB_DEF(layernorm_standard_checked), FB_DEF(split_heads), FB_DEF(merge_heads), FB_DEF(conv2d), FB_DEF(softmax),
                          FB_DEF(softmax_checked), FB_DEF(cnn_forward), {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_binding", "Native boundary of the tensor-level operators.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding(void) {
  PyObject* const m = PyModule_Create(&kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", FB_BUILT_FOR) != 0) {   // (build.py: binding_target)
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
