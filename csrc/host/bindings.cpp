// Native host path of the ops that run on one GPU alone: argument checks, output allocation, scratch and
// launch without Python in between. A rms_norm call of one row spends 2.3 us in the CUDA launch; the
// same steps in Python and ctypes took 12.5 us, a GEMM call 22 us.
//
// Every function returns None when the arguments are not the plain case it handles (another dtype,
// layout or device, logging of kernel choices switched on): the Python op then takes its general path,
// which also raises the errors. The kernels are reached through the C API of libkraken_b200.so, whose
// addresses bind() receives, so that the debug build of that library serves as well.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <cstdlib>
#include <map>
#include <mutex>
#include <utility>

namespace {

using u64 = unsigned long long;
struct Api {
  const char* (*last_error)();
  int (*rms_norm)(const void*, const void*, void*, int, int, float, void*);
  int (*local_bias_rms_norm)(const void*, int, const void*, u64, const void*, void*, int, int, float, int, void*);
  int (*local_all_reduce)(const void*, void*, const void*, u64, u64, void*);
  int (*gemm_scratch)(int, int, int, long long, long long, int, int, int, int, int, u64*);
  int (*gemm)(const void*, long long, const void*, long long, void*, long long, int, int, int, int, int, int, int, int, int, int,
              uint32_t*, void*, void*);
};
Api api;
PyObject* g_error = nullptr;

PyObject* failed(int rc) {
  PyErr_Format(g_error, "kraken_b200 native call failed (code %d): %s", rc, api.last_error());
  return nullptr;
}

// Kernel choices are logged by the general path.
bool logging() {
  const char* a = getenv("KRAKEN_DUMP_KERNEL");
  if (a && a[0] == '1' && a[1] == 0) return true;
  const char* b = getenv("SYMM_DUMP_KERNEL");
  return b && b[0] == '1' && b[1] == 0;
}

// The tensor behind `o`, if it is an ordinary CUDA tensor on the current device.
const at::Tensor* cuda_tensor(PyObject* o, c10::DeviceIndex dev) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.device().index() != dev || t.layout() != at::kStrided) return nullptr;
  return &t;
}
bool aligned(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
bool plain_bf16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 && t.is_contiguous() && aligned(t); }
bool fits_int(int64_t v) { return v >= 1 && v < (int64_t(1) << 31); }

// ---- counters of GEMMs that draw their tiles ------------------------------------------------------
// They are zero between launches, so one small buffer per stream serves every call on it (calls on one
// stream never overlap). At most kMaxStreams buffers are kept; a dropped one goes back to torch's caching
// allocator, which hands it out again in stream order. Under stream capture the buffer is allocated and
// zeroed inside the graph.
constexpr size_t kMaxStreams = 32;
constexpr int64_t kCounterWords = 32;
std::mutex g_pool_mu;
std::map<std::pair<int, void*>, at::Tensor> g_pool;

// Not through the dispatcher: nobody's dispatch mode may see, replace or delay these words (the lock is held).
at::Tensor zero_words(c10::DeviceIndex dev, c10::cuda::CUDAStream stream, int64_t words) {
  at::Tensor t = at::detail::empty_cuda({words}, at::kInt, at::Device(at::kCUDA, dev), std::nullopt);
  C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, (size_t)words * sizeof(int32_t), stream.stream()));
  return t;
}

at::Tensor counters_for(c10::DeviceIndex dev, c10::cuda::CUDAStream stream, int64_t words) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream.stream(), &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) return zero_words(dev, stream, words);
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto key = std::make_pair((int)dev, (void*)stream.stream());
  auto it = g_pool.find(key);
  if (it != g_pool.end() && it->second.numel() >= words) return it->second;
  if (g_pool.size() >= kMaxStreams) g_pool.clear();
  at::Tensor t = zero_words(dev, stream, std::max(words, kCounterWords));
  g_pool[key] = t;
  return t;
}

// reset(): drops the counters. Every path of the kernels, a wait that ran out included, puts them back to zero; a
// recovery should not have to rely on that.
PyObject* py_reset(PyObject*, PyObject*) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  g_pool.clear();
  Py_RETURN_NONE;
}

// Operands as the kernels take them: a [M, K] with K contiguous, bt [N, K] with K contiguous
// (row stride `ldb`). Whether these are such operands, both bf16 or, with tf32, both fp32.
bool gemm_operands(const at::Tensor& a, const at::Tensor& bt, int64_t N, int64_t Kb, int64_t ldb, int64_t kb_stride, bool tf32) {
  if (a.dim() != 2 || bt.dim() != 2 || a.scalar_type() != bt.scalar_type()) return false;
  const bool fp32 = a.scalar_type() == at::kFloat;
  if (fp32 ? !tf32 : a.scalar_type() != at::kBFloat16) return false;
  const int64_t M = a.size(0), K = a.size(1), unit = fp32 ? 4 : 8, lda = a.stride(0);
  return Kb == K && fits_int(M) && fits_int(N) && fits_int(K) && K % unit == 0 && a.stride(1) == 1 && kb_stride == 1 && lda % unit == 0 &&
         ldb % unit == 0 && lda >= K && ldb >= K && aligned(a) && aligned(bt);
}
int run_gemm(const at::Tensor& a, const at::Tensor& bt, int64_t N, int64_t ldb, bool out_fp32, int act, int swap, int bn, int max_ctas, int pair,
             void* copy_dst, c10::cuda::CUDAStream stream, bool pad_rows, at::Tensor& out) {
  const int64_t M = a.size(0), K = a.size(1);
  const bool fp32 = a.scalar_type() == at::kFloat;
  // pad_rows: rows of whole 128-byte lines, for a result that the next GEMM reads
  const int64_t line = out_fp32 ? 32 : 64, ldo = pad_rows ? (N + line - 1) / line * line : N;
  out = at::detail::empty_cuda({M, ldo}, out_fp32 ? at::kFloat : at::kBFloat16, a.device(), std::nullopt);
  if (ldo != N) out = out.narrow(1, 0, N);
  u64 words = 0;
  int rc = api.gemm_scratch((int)M, (int)N, (int)K, a.stride(0), ldb, fp32, swap, bn, pair, max_ctas, &words);
  if (rc) return rc;
  at::Tensor counters;
  if (words) counters = counters_for(a.device().index(), stream, (int64_t)words);
  return api.gemm(a.data_ptr(), a.stride(0), bt.data_ptr(), ldb, out.data_ptr(), ldo, (int)M, (int)N, (int)K, out_fp32, act, swap, bn, max_ctas,
                  pair, fp32, words ? (uint32_t*)counters.data_ptr() : nullptr, copy_dst, (void*)stream.stream());
}

// gemm(a, b, out_fp32, act, tf32, swap_ab, bn, max_ctas, pair, copy_dst, pad_rows): act(a @ b). a [M, K] with K contiguous, b
// [K, N] stored transposed (N rows of contiguous K), both bf16 or, with tf32, both fp32.
PyObject* py_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 11) {
    PyErr_SetString(PyExc_TypeError, "gemm takes 11 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor *a = cuda_tensor(args[0], dev), *b = cuda_tensor(args[1], dev);
  if (!a || !b || b->dim() != 2 || !gemm_operands(*a, *b, b->size(1), b->size(0), b->stride(1), b->stride(0), args[4] == Py_True)) Py_RETURN_NONE;
  const int act = (int)PyLong_AsLong(args[3]), swap = (int)PyLong_AsLong(args[5]), bn = (int)PyLong_AsLong(args[6]),
            max_ctas = (int)PyLong_AsLong(args[7]), pair = (int)PyLong_AsLong(args[8]);
  if (PyErr_Occurred()) return nullptr;
  void* copy_dst = nullptr;
  if (args[9] != Py_None) {
    const at::Tensor* c = cuda_tensor(args[9], dev);
    if (!c || !plain_bf16(*c) || c->numel() != a->numel() || a->scalar_type() != at::kBFloat16 || !a->is_contiguous()) Py_RETURN_NONE;
    copy_dst = c->data_ptr();
  }
  at::Tensor out;
  const int rc = run_gemm(*a, *b, b->size(1), b->stride(1), args[2] == Py_True, act, swap, bn, max_ctas, pair, copy_dst,
                          c10::cuda::getCurrentCUDAStream(dev), args[10] == Py_True, out);
  if (rc) return failed(rc);
  return THPVariable_Wrap(std::move(out));
}

// decode(h, w_t, bias, norm_w, eps) -> bf16 rms_norm(bf16(bf16(h @ w_t^T) + bias)) * norm_w; w_t [N, K], all bf16
PyObject* py_decode(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 5) {
    PyErr_SetString(PyExc_TypeError, "decode takes 5 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor *h = cuda_tensor(args[0], dev), *wt = cuda_tensor(args[1], dev), *bias = cuda_tensor(args[2], dev),
                   *w = cuda_tensor(args[3], dev);
  if (!h || !wt || !bias || !w || wt->dim() != 2 || !gemm_operands(*h, *wt, wt->size(0), wt->size(1), wt->stride(0), wt->stride(1), false) || logging())
    Py_RETURN_NONE;
  const int64_t N = wt->size(0);
  if (!plain_bf16(*bias) || !plain_bf16(*w) || N % 8 || N > 32768 || bias->numel() != N || w->numel() != N) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[4]);
  if (PyErr_Occurred()) return nullptr;
  auto stream = c10::cuda::getCurrentCUDAStream(dev);
  at::Tensor p;
  int rc = run_gemm(*h, *wt, N, wt->stride(0), false, 0, -1, 0, 0, 1, nullptr, stream, false, p);
  if (rc) return failed(rc);
  at::Tensor y = at::detail::empty_cuda(p.sizes(), at::kBFloat16, p.device(), std::nullopt);
  rc = api.local_bias_rms_norm(p.data_ptr(), 0, bias->data_ptr(), (u64)N, w->data_ptr(), y.data_ptr(), (int)p.size(0), (int)N, (float)eps, 1,
                               (void*)stream.stream());
  if (rc) return failed(rc);
  return THPVariable_Wrap(std::move(y));
}

// rms_norm(x, w, eps) -> y
PyObject* py_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "rms_norm takes 3 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor *x = cuda_tensor(args[0], dev), *w = cuda_tensor(args[1], dev);
  if (!x || !w || !plain_bf16(*x) || !plain_bf16(*w) || x->dim() < 1 || logging()) Py_RETURN_NONE;
  const int64_t D = x->size(-1);
  if (w->numel() != D || D % 8 || !fits_int(D) || !fits_int(x->numel() / std::max<int64_t>(D, 1))) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[2]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor y = at::detail::empty_cuda(x->sizes(), at::kBFloat16, x->device(), std::nullopt);
  int rc = api.rms_norm(x->data_ptr(), w->data_ptr(), y.data_ptr(), (int)(x->numel() / D), (int)D, (float)eps,
                        (void*)c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed(rc);
  return THPVariable_Wrap(std::move(y));
}

// A bias of one row or of the input's size; false: not that.
bool bias_of(PyObject* o, c10::DeviceIndex dev, const at::Tensor& x, const void*& ptr, u64& numel) {
  ptr = nullptr;
  numel = 0;
  if (o == Py_None) return true;
  const at::Tensor* b = cuda_tensor(o, dev);
  if (!b || !plain_bf16(*b) || (b->numel() != x.numel() && (x.dim() == 0 || b->numel() != x.size(-1)))) return false;
  ptr = b->data_ptr();
  numel = (u64)b->numel();
  return true;
}

// bias_rms_norm(scratch, x, bias, w, y, eps): y = rms_norm(x + bias) * w, the sum in fp32; True when done. The
// scratch tensor of the multi-rank form only has to be large enough.
PyObject* py_bias_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "bias_rms_norm takes 6 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor *scratch = cuda_tensor(args[0], dev), *x = cuda_tensor(args[1], dev), *w = cuda_tensor(args[3], dev),
                   *y = cuda_tensor(args[4], dev);
  if (!scratch || !x || !w || !y || scratch->nbytes() < x->nbytes() || !plain_bf16(*x) || !plain_bf16(*w) || !plain_bf16(*y) || x->dim() < 1 || logging()) Py_RETURN_NONE;
  const int64_t D = x->size(-1);
  const void* bias;
  u64 bias_n;
  if (!fits_int(D) || D % 8 || D > 32768 || w->numel() != D || y->numel() != x->numel() || !fits_int(x->numel() / D)) Py_RETURN_NONE;
  if (!bias_of(args[2], dev, *x, bias, bias_n)) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[5]);
  if (PyErr_Occurred()) return nullptr;
  int rc = api.local_bias_rms_norm(x->data_ptr(), 0, bias, bias_n, w->data_ptr(), y->data_ptr(), (int)(x->numel() / D), (int)D, (float)eps, 0,
                                   (void*)c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed(rc);
  Py_RETURN_TRUE;
}

// rounded_bias_rms_norm(p, bias, w, eps) -> bf16 rms_norm(bf16(bf16(p) + bias)) * w; p bf16 or fp32
PyObject* py_rounded_bias_rms_norm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "rounded_bias_rms_norm takes 4 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor *p = cuda_tensor(args[0], dev), *bias = cuda_tensor(args[1], dev), *w = cuda_tensor(args[2], dev);
  if (!p || !bias || !w || !plain_bf16(*bias) || !plain_bf16(*w) || p->dim() < 1 || !p->is_contiguous() || !aligned(*p) || logging()) Py_RETURN_NONE;
  const bool fp32 = p->scalar_type() == at::kFloat;
  const int64_t D = p->size(-1);
  if (!fp32 && p->scalar_type() != at::kBFloat16) Py_RETURN_NONE;
  if (!fits_int(D) || D % 8 || D > 32768 || w->numel() != D || bias->numel() != D || !fits_int(p->numel() / D)) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) return nullptr;
  at::Tensor y = at::detail::empty_cuda(p->sizes(), at::kBFloat16, p->device(), std::nullopt);
  int rc = api.local_bias_rms_norm(p->data_ptr(), fp32, bias->data_ptr(), (u64)D, w->data_ptr(), y.data_ptr(), (int)(p->numel() / D), (int)D,
                                   (float)eps, 1, (void*)c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed(rc);
  return THPVariable_Wrap(std::move(y));
}

// all_reduce(x, bias, out or None) -> out = x (+ bias)
PyObject* py_all_reduce(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "all_reduce takes 3 arguments");
    return nullptr;
  }
  const c10::DeviceIndex dev = c10::cuda::current_device();
  const at::Tensor* x = cuda_tensor(args[0], dev);
  if (!x || !plain_bf16(*x) || x->numel() % 8 || x->numel() < 8 || logging()) Py_RETURN_NONE;
  const void* bias;
  u64 bias_n;
  if (!bias_of(args[1], dev, *x, bias, bias_n) || bias_n % 8) Py_RETURN_NONE;
  at::Tensor fresh;
  void* out;
  if (args[2] == Py_None) {
    fresh = at::detail::empty_cuda(x->sizes(), at::kBFloat16, x->device(), std::nullopt);
    out = fresh.data_ptr();
  } else {
    const at::Tensor* o = cuda_tensor(args[2], dev);
    if (!o || !plain_bf16(*o) || o->numel() != x->numel()) Py_RETURN_NONE;
    out = o->data_ptr();
  }
  int rc = api.local_all_reduce(x->data_ptr(), out, bias, bias_n, (u64)x->numel(), (void*)c10::cuda::getCurrentCUDAStream(dev).stream());
  if (rc) return failed(rc);
  if (args[2] == Py_None) return THPVariable_Wrap(std::move(fresh));
  Py_INCREF(args[2]);
  return args[2];
}

template <class F>
bool address(PyObject* d, const char* name, F& f) {
  PyObject* v = PyDict_GetItemString(d, name);
  void* p = v ? PyLong_AsVoidPtr(v) : nullptr;
  if (!p) {
    PyErr_Format(PyExc_KeyError, "no address of %s", name);
    return false;
  }
  f = reinterpret_cast<F>(p);
  return true;
}

// bind(addresses of the C API by name, exception class)
PyObject* py_bind(PyObject*, PyObject* args) {
  PyObject *d, *err;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &d, &err)) return nullptr;
  if (!address(d, "kr_last_error", api.last_error) || !address(d, "kr_rms_norm", api.rms_norm) ||
      !address(d, "kr_local_bias_rms_norm", api.local_bias_rms_norm) || !address(d, "kr_local_all_reduce", api.local_all_reduce) ||
      !address(d, "kr_gemm_scratch", api.gemm_scratch) || !address(d, "kr_gemm", api.gemm))
    return nullptr;
  Py_XDECREF(g_error);
  Py_INCREF(err);
  g_error = err;
  Py_RETURN_NONE;
}

// C++ exceptions (out of memory above all) as torch would raise them
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return F(self, args, n);
  END_HANDLE_TH_ERRORS
}
#define KR_FAST(NAME) \
  { #NAME, (PyCFunction)(void (*)(void))guarded<py_##NAME>, METH_FASTCALL, nullptr }
PyMethodDef g_methods[] = {KR_FAST(gemm), KR_FAST(decode), KR_FAST(rms_norm), KR_FAST(bias_rms_norm), KR_FAST(rounded_bias_rms_norm), KR_FAST(all_reduce),
                           {"bind", py_bind, METH_VARARGS, nullptr},
                           {"reset", py_reset, METH_NOARGS, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "kraken_b200_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_kraken_b200_host() { return PyModule_Create(&g_module); }
