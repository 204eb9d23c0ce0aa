// Native host path of the layers: takes torch tensors, allocates outputs and scratch from torch's
// caching allocator, and calls the C ABI of libhy3d_int8.so (include/hy3d_int8.h) on the current
// stream.  One call replaces the argument checks, allocations, device guard and 19-argument ctypes
// call of `_binding.py`, which cost 30-35 us of host time per layer -- more than the kernels of every
// layer below about 10 G multiply-adds.
//
// Every function answers Py_None, having done nothing, for arguments outside the plain case (another
// dtype, a non-contiguous or CPU tensor, a tensor subclass, a shape that does not fit); the caller then
// takes the checked path of `_binding.py`, which either handles them or raises with its message.  What only
// the library refuses (an address off a 16-byte boundary, K above a kernel's limit, GEGLU with N % 32 != 0)
// raises here with the library's status, as it does there.  No gradient is recorded, whatever the grad mode.
// Plain CPython calling convention: no argument-conversion layer in between.
#include <Python.h>
#include <dlfcn.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/Context.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include "../../include/hy3d_int8.h"

namespace {

#define HY3D_FN(name) decltype(&::name) name = nullptr
struct Api {
  HY3D_FN(hy3d_linear_w8a8_dense);
  HY3D_FN(hy3d_gemm_w8a8_dense);
  HY3D_FN(hy3d_dense_layer_splitk_plan);
  HY3D_FN(hy3d_gemm_w8a8_dense_splitk);
  HY3D_FN(hy3d_quantize_rows);
  HY3D_FN(hy3d_linear_cluster_plan);
  HY3D_FN(hy3d_linear_w8a8_cluster);
  HY3D_FN(hy3d_linear_w8a8_sparse24);
  HY3D_FN(hy3d_gemm_w8a8_sparse24);
  HY3D_FN(hy3d_layernorm_quantize);
  HY3D_FN(hy3d_groupnorm_nhwc_terms);
  HY3D_FN(hy3d_add_bias_nhwc);
  HY3D_FN(hy3d_concat_nhwc);
  HY3D_FN(hy3d_upsample2x_nhwc);
  HY3D_FN(hy3d_add_quantize_rows);
  HY3D_FN(hy3d_add_layernorm_quantize);
  HY3D_FN(hy3d_quantize_weight);
  HY3D_FN(hy3d_status_string);
} api;
#undef HY3D_FN

// A tensor the kernels can take as it is: plain strided CUDA storage, contiguous.
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;   // torch.Tensor or Parameter, no other subclass
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}

// The same in channels-last memory, f16 / bf16, whole 16-byte vectors of channels.
const at::Tensor* plain_nhwc(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.dim() == 4 && (t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16) &&
                 (t.size(1) & 7) == 0 && t.numel() > 0 && t.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                 (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0
             ? &t
             : nullptr;
}

int half_code(at::ScalarType t) {
  return t == at::kHalf ? HY3D_F16 : t == at::kBFloat16 ? HY3D_BF16 : -1;
}
int param_code(at::ScalarType t) { return t == at::kFloat ? HY3D_F32 : half_code(t); }

// Scratch of one call: taken from the allocator's pool of the stream it is used on and handed back when
// the call has enqueued its kernels, which is when a tensor going out of scope would return it too.
struct Scratch {
  void* p = nullptr;
  Scratch(size_t bytes, cudaStream_t s) : p(c10::cuda::CUDACachingAllocator::raw_alloc_with_stream(bytes, s)) {}
  ~Scratch() { if (p) c10::cuda::CUDACachingAllocator::raw_delete(p); }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  int8_t* at(size_t off) const { return static_cast<int8_t*>(p) + off; }
};

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

PyObject* none() { Py_RETURN_NONE; }

PyObject* failed(const char* what, int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s failed: %s (status %d)", what, api.hy3d_status_string(rc), rc);
  return nullptr;
}

// Weight scales and the optional bias of a layer with N output rows.
struct Params {
  const void* ws = nullptr;
  const void* bias = nullptr;
  int ws_code = 0, bias_code = HY3D_F16;
  bool ok = false;
  // The reduction behind a split K reads scales and bias by 16-byte vectors; the other kernels take any address.
  bool may_split() const { return ((reinterpret_cast<uintptr_t>(ws) | reinterpret_cast<uintptr_t>(bias)) & 15) == 0; }
  Params(PyObject* scale, PyObject* b, int64_t N, c10::Device dev) {
    const at::Tensor* s = plain(scale);
    if (!s || s->dim() != 1 || s->size(0) != N || s->device() != dev) return;
    ws_code = param_code(s->scalar_type());
    ws = s->const_data_ptr();
    if (ws_code < 0) return;
    if (b != Py_None) {
      const at::Tensor* t = plain(b);
      if (!t || t->device() != dev) return;
      if (t->numel() != 0) {
        if (t->dim() != 1 || t->size(0) != N) return;
        bias_code = param_code(t->scalar_type());
        if (bias_code < 0) return;
        bias = t->const_data_ptr();
      }
    }
    ok = true;
  }
};

// The output of a layer: the input's leading dimensions, `cols` columns.
at::Tensor out_like(c10::IntArrayRef lead, int64_t cols, at::ScalarType type, c10::Device dev) {
  c10::SmallVector<int64_t, 6> shape(lead.begin(), lead.end());
  shape.push_back(cols);
  return at::Tensor(at::detail::empty_cuda(shape, type, dev, std::nullopt));
}

bool small_int(PyObject* o, long lo, long hi, long* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongAndOverflow(o, &overflow);
  return !overflow && *v >= lo && *v <= hi;
}

// Small layers in one launch: what a caller waits for there is its own thread's launches, not the device.
// A captured graph replays without those, so capture keeps the two kernels, the faster form on the device.
bool one_launch(int64_t M, int64_t N, int64_t K, int sparse, int* block_t, int* ks) {
  return api.hy3d_linear_cluster_plan(M, N, K, sparse, block_t, ks) &&
         c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
}

// int8 GEMM + epilogue on codes that are already there; follows the library's split-K plan.
int dense_gemm(const int8_t* q, const float* s, const at::Tensor& w, const Params& p, void* out, int out_code,
               int64_t M, int64_t N, int64_t K, int epi, cudaStream_t st) {
  int64_t bytes = 0;
  const int splits = p.may_split() ? api.hy3d_dense_layer_splitk_plan(M, N, K, epi, &bytes) : 1;
  if (splits > 1) {
    Scratch part(static_cast<size_t>(bytes), st);
    return api.hy3d_gemm_w8a8_dense_splitk(q, w.const_data_ptr<int8_t>(), s, p.ws, p.ws_code, p.bias, p.bias_code,
                                           out, out_code, M, N, K, epi, splits, part.p, bytes, st);
  }
  return api.hy3d_gemm_w8a8_dense(q, w.const_data_ptr<int8_t>(), s, p.ws, p.ws_code, p.bias, p.bias_code, out,
                                  out_code, M, N, K, epi, 0, 0, st);
}

// linear_dense(x, w_int8 (N,K), w_scale, bias | None, epilogue) -> y | None
PyObject* linear_dense_impl(PyObject* px, PyObject* pw, PyObject* pscale, PyObject* pbias, long epi) {
  HANDLE_TH_ERRORS
  const at::Tensor *x = plain(px), *w = plain(pw);
  if (!x || !w || x->dim() < 1 || w->dim() != 2 || w->scalar_type() != at::kChar || w->device() != x->device())
    return none();
  const int code = half_code(x->scalar_type());
  const int64_t N = w->size(0), K = w->size(1);
  const int64_t M = K > 0 ? x->numel() / K : 0;
  if (code < 0 || M <= 0 || x->size(-1) != K || (K & 63) || (N & 15)) return none();
  const Params p(pscale, pbias, N, x->device());
  if (!p.ok) return none();
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  at::Tensor y = out_like(x->sizes().slice(0, x->dim() - 1), epi == HY3D_EPI_GEGLU ? N / 2 : N, x->scalar_type(),
                          x->device());
  int rc, block_t = 0, ks = 0;
  if (one_launch(M, N, K, 0, &block_t, &ks)) {
    rc = api.hy3d_linear_w8a8_cluster(x->const_data_ptr(), code, K, w->const_data_ptr<int8_t>(), nullptr, 0, p.ws, p.ws_code,
                                      p.bias, p.bias_code, y.mutable_data_ptr(), M, N, K, static_cast<int>(epi), block_t, ks, st);
    if (rc != HY3D_OK) return failed("hy3d_linear_w8a8_cluster", rc);
    return THPVariable_Wrap(std::move(y));
  }
  const size_t codes = align256(static_cast<size_t>(M) * K);
  Scratch ws(codes + static_cast<size_t>(M) * 4, st);
  int64_t bytes = 0;
  if (p.may_split() && api.hy3d_dense_layer_splitk_plan(M, N, K, static_cast<int>(epi), &bytes) > 1) {
    rc = api.hy3d_quantize_rows(x->const_data_ptr(), code, M, K, K, ws.at(0), reinterpret_cast<float*>(ws.at(codes)), st);
    if (rc == HY3D_OK)
      rc = dense_gemm(ws.at(0), reinterpret_cast<float*>(ws.at(codes)), *w, p, y.mutable_data_ptr(), code, M, N, K,
                      static_cast<int>(epi), st);
  } else {
    rc = api.hy3d_linear_w8a8_dense(x->const_data_ptr(), code, K, ws.at(0), reinterpret_cast<float*>(ws.at(codes)),
                                    w->const_data_ptr<int8_t>(), p.ws, p.ws_code, p.bias, p.bias_code,
                                    y.mutable_data_ptr(), code, M, N, K, static_cast<int>(epi), 0, 0, st);
  }
  if (rc != HY3D_OK) return failed("hy3d_linear_w8a8_dense", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyObject* linear_dense(PyObject*, PyObject* const* a, Py_ssize_t n) {
  long epi = 0;
  if (n != 5 || !small_int(a[4], 0, 2, &epi)) return none();
  return linear_dense_impl(a[0], a[1], a[2], a[3], epi);
}

// linear_sparse(x, w_comp (N,K/2), w_meta, w_scale, bias | None, epilogue) -> y | None
PyObject* linear_sparse_impl(PyObject* px, PyObject* pw, PyObject* pmeta, PyObject* pscale, PyObject* pbias, long epi) {
  HANDLE_TH_ERRORS
  const at::Tensor *x = plain(px), *w = plain(pw), *e = plain(pmeta);
  if (!x || !w || !e || x->dim() < 1 || w->dim() != 2 || e->dim() != 2 || w->scalar_type() != at::kChar ||
      e->scalar_type() != at::kInt || w->device() != x->device() || e->device() != x->device())
    return none();
  const int code = half_code(x->scalar_type());
  const int64_t N = w->size(0), K = 2 * w->size(1);
  const int64_t M = K > 0 ? x->numel() / K : 0;
  if (code < 0 || M <= 0 || x->size(-1) != K || (K & 63) || (N & 15) || e->size(0) != N) return none();
  const Params p(pscale, pbias, N, x->device());
  if (!p.ok) return none();
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  at::Tensor y = out_like(x->sizes().slice(0, x->dim() - 1), epi == HY3D_EPI_GEGLU ? N / 2 : N, x->scalar_type(),
                          x->device());
  int rc, block_t = 0, ks = 0;
  if (one_launch(M, N, K, 1, &block_t, &ks)) {
    rc = api.hy3d_linear_w8a8_cluster(x->const_data_ptr(), code, K, w->const_data_ptr<int8_t>(),
                                      reinterpret_cast<const uint32_t*>(e->const_data_ptr<int32_t>()), e->size(1), p.ws,
                                      p.ws_code, p.bias, p.bias_code, y.mutable_data_ptr(), M, N, K, static_cast<int>(epi),
                                      block_t, ks, st);
    if (rc != HY3D_OK) return failed("hy3d_linear_w8a8_cluster", rc);
    return THPVariable_Wrap(std::move(y));
  }
  const size_t codes = align256(static_cast<size_t>(M) * K);
  Scratch ws(codes + static_cast<size_t>(M) * 4, st);
  rc = api.hy3d_linear_w8a8_sparse24(
      x->const_data_ptr(), code, K, ws.at(0), reinterpret_cast<float*>(ws.at(codes)), w->const_data_ptr<int8_t>(),
      reinterpret_cast<const uint32_t*>(e->const_data_ptr<int32_t>()), e->size(1), p.ws, p.ws_code, p.bias, p.bias_code,
      y.mutable_data_ptr(), code, M, N, K, static_cast<int>(epi), 0, st);
  if (rc != HY3D_OK) return failed("hy3d_linear_w8a8_sparse24", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyObject* linear_sparse(PyObject*, PyObject* const* a, Py_ssize_t n) {
  long epi = 0;
  if (n != 6 || !small_int(a[5], 0, 2, &epi)) return none();
  return linear_sparse_impl(a[0], a[1], a[2], a[3], a[4], epi);
}

// The two forms of a layer whose input arrives as codes and per-row scales: the logical shape is given as a
// tuple, the output type by a code.  The output is allocated from the leading entries and the kernel writes M
// rows, so the tuple has to describe exactly M rows of K.
bool lead_shape(PyObject* o, int64_t M, int64_t K, c10::SmallVector<int64_t, 6>* lead) {
  if (!PyTuple_Check(o)) return false;
  const Py_ssize_t d = PyTuple_GET_SIZE(o);
  int64_t rows = 1;
  for (Py_ssize_t i = 0; i < d; ++i) {
    PyObject* v = PyTuple_GET_ITEM(o, i);
    if (!PyLong_Check(v)) return false;
    int overflow = 0;
    const int64_t n = PyLong_AsLongLongAndOverflow(v, &overflow);      // -1 and no exception where it does not fit
    if (i + 1 == d) return n == K && rows == M;
    if (n < 1 || rows > M / n) return false;
    rows *= n;
    lead->push_back(n);
  }
  return false;
}

// gemm_dense(q (M,K), scale (M), w_int8, w_scale, bias | None, is_bf16, epilogue, shape) -> y | None
PyObject* gemm_dense(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  long epi = 0, bf16 = 0;
  c10::SmallVector<int64_t, 6> lead;
  if (n != 8 || !small_int(a[5], 0, 1, &bf16) || !small_int(a[6], 0, 2, &epi)) return none();
  const at::Tensor *q = plain(a[0]), *s = plain(a[1]), *w = plain(a[2]);
  if (!q || !s || !w || q->dim() != 2 || s->dim() != 1 || w->dim() != 2 || q->scalar_type() != at::kChar ||
      s->scalar_type() != at::kFloat || w->scalar_type() != at::kChar || w->device() != q->device() ||
      s->device() != q->device())
    return none();
  const int64_t M = q->size(0), K = q->size(1), N = w->size(0);
  if (M <= 0 || s->size(0) != M || w->size(1) != K || (K & 63) || (N & 15) || !lead_shape(a[7], M, K, &lead)) return none();
  const Params p(a[3], a[4], N, q->device());
  if (!p.ok) return none();
  c10::cuda::CUDAGuard guard(q->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
  at::Tensor y = out_like(lead, epi == HY3D_EPI_GEGLU ? N / 2 : N, bf16 ? at::kBFloat16 : at::kHalf, q->device());
  const int rc = dense_gemm(q->const_data_ptr<int8_t>(), s->const_data_ptr<float>(), *w, p, y.mutable_data_ptr(),
                            bf16 ? HY3D_BF16 : HY3D_F16, M, N, K, static_cast<int>(epi), st);
  if (rc != HY3D_OK) return failed("hy3d_gemm_w8a8_dense", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// gemm_sparse(q, scale, w_comp, w_meta, w_scale, bias | None, is_bf16, epilogue, shape) -> y | None
PyObject* gemm_sparse(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  long epi = 0, bf16 = 0;
  c10::SmallVector<int64_t, 6> lead;
  if (n != 9 || !small_int(a[6], 0, 1, &bf16) || !small_int(a[7], 0, 2, &epi)) return none();
  const at::Tensor *q = plain(a[0]), *s = plain(a[1]), *w = plain(a[2]), *e = plain(a[3]);
  if (!q || !s || !w || !e || q->dim() != 2 || s->dim() != 1 || w->dim() != 2 || e->dim() != 2 ||
      q->scalar_type() != at::kChar || s->scalar_type() != at::kFloat || w->scalar_type() != at::kChar ||
      e->scalar_type() != at::kInt || w->device() != q->device() || s->device() != q->device() ||
      e->device() != q->device())
    return none();
  const int64_t M = q->size(0), K = q->size(1), N = w->size(0);
  if (M <= 0 || s->size(0) != M || 2 * w->size(1) != K || (K & 63) || (N & 15) || e->size(0) != N ||
      !lead_shape(a[8], M, K, &lead))
    return none();
  const Params p(a[4], a[5], N, q->device());
  if (!p.ok) return none();
  c10::cuda::CUDAGuard guard(q->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(q->device().index()).stream();
  at::Tensor y = out_like(lead, epi == HY3D_EPI_GEGLU ? N / 2 : N, bf16 ? at::kBFloat16 : at::kHalf, q->device());
  const int rc = api.hy3d_gemm_w8a8_sparse24(
      q->const_data_ptr<int8_t>(), s->const_data_ptr<float>(), w->const_data_ptr<int8_t>(),
      reinterpret_cast<const uint32_t*>(e->const_data_ptr<int32_t>()), e->size(1), p.ws, p.ws_code, p.bias, p.bias_code,
      y.mutable_data_ptr(), bf16 ? HY3D_BF16 : HY3D_F16, M, N, K, static_cast<int>(epi), 0, st);
  if (rc != HY3D_OK) return failed("hy3d_gemm_w8a8_sparse24", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// gamma and beta of a normalisation: both of one type (or absent).
struct Affine {
  const void *gamma = nullptr, *beta = nullptr;
  int code = HY3D_F32;
  bool ok = false;
  Affine(PyObject* g, PyObject* b, int64_t C, c10::Device dev) {
    for (int i = 0; i < 2; ++i) {
      PyObject* o = i ? b : g;
      if (o == Py_None) continue;
      const at::Tensor* t = plain(o);
      if (!t || t->numel() != C || t->device() != dev) return;
      const int c = param_code(t->scalar_type());
      if (c < 0 || (i && gamma && c != code)) return;
      code = c;
      (i ? beta : gamma) = t->const_data_ptr();
    }
    ok = true;
  }
};

// layernorm_quantize(x, gamma | None, beta | None, eps) -> (codes (M,K), scale (M)) | None
struct Quantized { at::Tensor q, s, sum; };
// padd: rows to add first; the sum goes to out->sum.
bool layernorm_quantize_impl(PyObject* px, PyObject* padd, PyObject* gamma, PyObject* beta, double eps, Quantized* out,
                             int* status) {
  const at::Tensor* x = plain(px);
  if (!x || x->dim() < 1) return false;
  const int code = half_code(x->scalar_type());
  const int64_t K = x->size(-1), M = K > 0 ? x->numel() / K : 0;
  if (code < 0 || M <= 0) return false;
  const Affine f(gamma, beta, K, x->device());
  if (!f.ok) return false;
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  out->q = at::Tensor(at::detail::empty_cuda({M, K}, at::kChar, x->device(), std::nullopt));
  out->s = at::Tensor(at::detail::empty_cuda({M}, at::kFloat, x->device(), std::nullopt));
  if (padd) {
    const at::Tensor* t = plain(padd);
    if (!t || t->scalar_type() != x->scalar_type() || t->device() != x->device() || t->sizes() != x->sizes()) return false;
    out->sum = at::Tensor(at::detail::empty_cuda(x->sizes(), x->scalar_type(), x->device(), std::nullopt));
    *status = api.hy3d_add_layernorm_quantize(x->const_data_ptr(), t->const_data_ptr(), out->sum.mutable_data_ptr(), code, M, K,
                                              f.gamma, f.beta, f.code, static_cast<float>(eps), out->q.mutable_data_ptr<int8_t>(),
                                              out->s.mutable_data_ptr<float>(), st);
    return true;
  }
  *status = api.hy3d_layernorm_quantize(x->const_data_ptr(), code, M, K, K, f.gamma, f.beta, f.code, static_cast<float>(eps),
                                        out->q.mutable_data_ptr<int8_t>(), out->s.mutable_data_ptr<float>(), nullptr, st);
  return true;
}
PyObject* layernorm_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Quantized z;
  int rc = 0;
  if (n != 4 || !PyFloat_Check(a[3]) || !layernorm_quantize_impl(a[0], nullptr, a[1], a[2], PyFloat_AS_DOUBLE(a[3]), &z, &rc)) return none();
  if (rc != HY3D_OK) return failed("hy3d_layernorm_quantize", rc);
  PyObject* pq = THPVariable_Wrap(std::move(z.q));
  PyObject* ps = pq ? THPVariable_Wrap(std::move(z.s)) : nullptr;
  if (!ps) { Py_XDECREF(pq); return nullptr; }
  PyObject* r = PyTuple_New(2);
  if (!r) { Py_DECREF(pq); Py_DECREF(ps); return nullptr; }
  PyTuple_SET_ITEM(r, 0, pq);
  PyTuple_SET_ITEM(r, 1, ps);
  return r;
  END_HANDLE_TH_ERRORS
}

// groupnorm_nhwc(x channels_last, groups, gamma | None, beta | None, eps, silu, add (B,C) | None) -> y | None
PyObject* groupnorm_impl(PyObject* px, long groups, PyObject* gamma, PyObject* beta, double eps, bool silu, PyObject* padd,
                         PyObject* pbias) {
  HANDLE_TH_ERRORS
  const at::Tensor* px4 = plain_nhwc(px);
  if (!px4) return none();
  const at::Tensor& x = *px4;
  const int code = half_code(x.scalar_type());
  const int64_t B = x.size(0), C = x.size(1), HW = x.size(2) * x.size(3);
  if (code < 0 || B <= 0 || HW <= 0) return none();
  const Affine f(gamma, beta, C, x.device());
  if (!f.ok) return none();
  const void *add = nullptr, *bias = nullptr;
  int64_t add_ld = C;
  if (padd != Py_None) {            // rows may lie apart (a slice of stacked projections)
    if (!THPVariable_CheckExact(padd)) return none();
    const at::Tensor& t = THPVariable_Unpack(padd);
    if (!t.is_cuda() || t.layout() != at::kStrided || t.dim() != 2 || t.size(0) != B || t.size(1) != C ||
        t.scalar_type() != x.scalar_type() || t.device() != x.device() || t.stride(1) != 1)
      return none();
    add = t.const_data_ptr();
    add_ld = B > 1 ? t.stride(0) : C;
    if (add_ld < C || (add_ld & 7) || (reinterpret_cast<uintptr_t>(add) & 15)) return none();
  }
  if (pbias != Py_None) {
    const at::Tensor* t = plain(pbias);
    if (!add || !t || t->numel() != C || t->scalar_type() != x.scalar_type() || t->device() != x.device() ||
        (reinterpret_cast<uintptr_t>(t->const_data_ptr()) & 15))
      return none();
    bias = t->const_data_ptr();
  }
  c10::cuda::CUDAGuard guard(x.device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
  at::Tensor y = at::Tensor(at::detail::empty_cuda(x.sizes(), x.scalar_type(), x.device(), at::MemoryFormat::ChannelsLast));
  const int rc = api.hy3d_groupnorm_nhwc_terms(x.const_data_ptr(), bias, add, add_ld, code, B, HW, C, static_cast<int>(groups),
                                               f.gamma, f.beta, f.code, static_cast<float>(eps), silu ? 1 : 0,
                                               y.mutable_data_ptr(), st);
  if (rc != HY3D_OK) return failed("hy3d_groupnorm_nhwc", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}
PyObject* groupnorm_nhwc(PyObject*, PyObject* const* a, Py_ssize_t n) {
  long groups = 0;
  if (n != 7 || !small_int(a[1], 1, 1 << 20, &groups) || !PyFloat_Check(a[4])) return none();
  return groupnorm_impl(a[0], groups, a[2], a[3], PyFloat_AS_DOUBLE(a[4]), a[5] == Py_True, a[6], Py_None);
}

// quantize_weight(w (N,K), sparse) -> (codes, scale) or (compressed codes, metadata, the layer's empty dense codes, scale) | None
PyObject* quantize_weight(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) return none();
  const at::Tensor* w = plain(a[0]);
  if (!w || w->dim() != 2) return none();
  const int code = param_code(w->scalar_type());
  const int64_t N = w->size(0), K = w->size(1);
  if (code < 0 || N <= 0 || K <= 0 || (K & 31) || (reinterpret_cast<uintptr_t>(w->const_data_ptr()) & 15)) return none();
  const bool sparse = a[1] == Py_True;
  c10::cuda::CUDAGuard guard(w->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(w->device().index()).stream();
  const auto dev = w->device();
  const int64_t ld = 4 * ((K + 127) / 128);
  at::Tensor out[4];
  int count = 0;
  out[count++] = at::Tensor(at::detail::empty_cuda({N, sparse ? K / 2 : K}, at::kChar, dev, std::nullopt));
  if (sparse) {
    out[count++] = at::Tensor(at::detail::empty_cuda({N, ld}, at::kInt, dev, std::nullopt));
    out[count++] = at::Tensor(at::detail::empty_cuda({0}, at::kChar, dev, std::nullopt));
  }
  const at::ScalarType st_type = w->scalar_type() == at::kBFloat16 ? at::kBFloat16 : at::kHalf;
  out[count++] = at::Tensor(at::detail::empty_cuda({N}, st_type, dev, std::nullopt));
  const int rc = api.hy3d_quantize_weight(
      w->const_data_ptr(), code, N, K, out[0].mutable_data_ptr<int8_t>(),
      sparse ? reinterpret_cast<uint32_t*>(out[1].mutable_data_ptr<int32_t>()) : nullptr, sparse ? ld : 0,
      out[count - 1].mutable_data_ptr(), half_code(st_type), st);
  if (rc != HY3D_OK) return failed("hy3d_quantize_weight", rc);
  PyObject* r = PyTuple_New(count);
  if (!r) return nullptr;
  for (int i = 0; i < count; ++i) {
    PyObject* o = THPVariable_Wrap(std::move(out[i]));
    if (!o) { Py_DECREF(r); return nullptr; }
    PyTuple_SET_ITEM(r, i, o);
  }
  return r;
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------
//  Modules
// ---------------------------------------------------------------------------------------
// The functions below are what calling an Int8Linear, Int8LayerNorm or GroupNormNHWC does when nothing
// stands between the call and the kernels: nn.Module's own __call__ and attribute look-ups through Python cost
// 1.5 us, more than half of a launch.  They answer None, having done nothing, for a subclass, a replaced
// `forward`, any hook (of the instance or global), a compiled or traced call, and whatever the functions above
// decline.
struct Names {
  PyObject *dict, *buffers, *parameters, *mode, *epilogue, *bias, *wq, *scale, *comp, *meta, *forward, *compiled, *weight,
      *eps, *fused, *silu, *groups, *shape, *dtype, *q, *act_scale, *conv_groups;
  PyObject* hooks[4];
} names;
struct Registered {
  PyTypeObject* type = nullptr;
  PyObject* forward = nullptr;
} linear_class, layernorm_class, groupnorm_class;
PyTypeObject* quantized_class = nullptr;
PyObject* global_hooks[4] = {};

bool intern_names() {
  struct { PyObject** at; const char* text; } all[] = {
      {&names.dict, "__dict__"}, {&names.buffers, "_buffers"}, {&names.parameters, "_parameters"}, {&names.mode, "mode"},
      {&names.epilogue, "epilogue"}, {&names.bias, "bias"}, {&names.wq, "weight_int8_nk"}, {&names.scale, "weight_scale"},
      {&names.comp, "weight_sparse_comp"}, {&names.meta, "weight_sparse_meta"}, {&names.forward, "forward"},
      {&names.compiled, "_compiled_call_impl"}, {&names.weight, "weight"}, {&names.eps, "eps"}, {&names.fused, "fused"},
      {&names.silu, "silu"}, {&names.groups, "num_groups"}, {&names.shape, "shape"}, {&names.dtype, "dtype"},
      {&names.q, "q"}, {&names.conv_groups, "groups"}, {&names.act_scale, "scale"}, {&names.hooks[0], "_backward_hooks"},
      {&names.hooks[1], "_backward_pre_hooks"}, {&names.hooks[2], "_forward_hooks"}, {&names.hooks[3], "_forward_pre_hooks"}};
  for (auto& n : all)
    if (!(*n.at = PyUnicode_InternFromString(n.text))) return false;
  return true;
}

// register_modules((Int8Linear, Int8LayerNorm, GroupNormNHWC | None), QuantizedActivation, 4 global hook dicts):
// the classes with the `forward` they have now.
PyObject* register_modules(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3 || !PyTuple_Check(a[0]) || !PyType_Check(a[1]) || !PyTuple_Check(a[2]) || PyTuple_GET_SIZE(a[2]) != 4) {
    PyErr_SetString(PyExc_TypeError, "register_modules(classes, quantized class, hook dicts)");
    return nullptr;
  }
  Registered* regs[] = {&linear_class, &layernorm_class, &groupnorm_class};
  for (Py_ssize_t i = 0; i < 3 && i < PyTuple_GET_SIZE(a[0]); ++i) {
    PyObject* c = PyTuple_GET_ITEM(a[0], i);
    if (c == Py_None) continue;
    PyObject* f = PyType_Check(c) ? PyObject_GetAttr(c, names.forward) : nullptr;
    if (!f) return nullptr;
    Py_INCREF(c);
    regs[i]->type = reinterpret_cast<PyTypeObject*>(c);
    regs[i]->forward = f;
  }
  Py_INCREF(a[1]);
  quantized_class = reinterpret_cast<PyTypeObject*>(a[1]);
  for (int i = 0; i < 4; ++i) {
    PyObject* d = PyTuple_GET_ITEM(a[2], i);
    if (!PyDict_Check(d)) { PyErr_SetString(PyExc_TypeError, "hook dicts"); return nullptr; }
    Py_INCREF(d);
    global_hooks[i] = d;
  }
  Py_RETURN_NONE;
}

// The instance dictionary of a module nothing stands before (borrowed), or nullptr.
PyObject* plain_module(PyObject* m, const Registered& reg) {
  if (Py_TYPE(m) != reg.type || torch::jit::tracer::isTracing()) return nullptr;
  if (_PyType_Lookup(reg.type, names.forward) != reg.forward) return nullptr;
  PyObject* dict = PyObject_GetAttr(m, names.dict);
  if (!dict) { PyErr_Clear(); return nullptr; }
  Py_DECREF(dict);                            // the module keeps it
  if (!PyDict_Check(dict) || PyDict_GetItemWithError(dict, names.forward) || PyDict_GetItemWithError(dict, names.compiled))
    return nullptr;
  for (int i = 0; i < 4; ++i) {
    PyObject* h = PyDict_GetItemWithError(dict, names.hooks[i]);
    if (!h || !PyDict_Check(h) || PyDict_GET_SIZE(h) != 0 || PyDict_GET_SIZE(global_hooks[i]) != 0) return nullptr;
  }
  return dict;
}

// The layer of instance dictionary `dict` on a tensor or a QuantizedActivation.
PyObject* linear_of(PyObject* layer, PyObject* dict, PyObject* x) {
  PyObject* buffers = PyDict_GetItemWithError(dict, names.buffers);
  if (!buffers || !PyDict_Check(buffers)) return none();
  PyObject* bias = PyDict_GetItemWithError(buffers, names.bias);
  if (!bias) bias = PyDict_GetItemWithError(dict, names.bias);
  PyObject* scale = PyDict_GetItemWithError(buffers, names.scale);
  if (!bias || !scale) return none();
  // instance or class attributes, compared by text
  auto attribute_is_one_of = [&](PyObject* name, std::initializer_list<const char*> texts) {
    PyObject* v = PyDict_GetItemWithError(dict, name);
    if (!v) v = _PyType_Lookup(Py_TYPE(layer), name);
    int i = 0;
    for (const char* t : texts) {
      if (v && PyUnicode_Check(v) && PyUnicode_CompareWithASCIIString(v, t) == 0) return i;
      ++i;
    }
    return -1;
  };
  const int mode = attribute_is_one_of(names.mode, {"tc", "sparse"});
  const int epi = attribute_is_one_of(names.epilogue, {"linear", "gelu", "geglu"});   // HY3D_EPI_* in order
  if (mode < 0 || epi < 0) return none();
  const bool sparse = mode == 1;
  PyObject* w = PyDict_GetItemWithError(buffers, sparse ? names.comp : names.wq);
  PyObject* meta = sparse ? PyDict_GetItemWithError(buffers, names.meta) : Py_None;
  if (!w || !meta) return none();
  if (THPVariable_CheckExact(x))
    return sparse ? linear_sparse_impl(x, w, meta, scale, bias, epi) : linear_dense_impl(x, w, scale, bias, epi);
  if (Py_TYPE(x) != quantized_class) return none();
  PyObject* part[4] = {PyObject_GetAttr(x, names.q), PyObject_GetAttr(x, names.act_scale), PyObject_GetAttr(x, names.shape),
                       PyObject_GetAttr(x, names.dtype)};
  PyObject* r = nullptr;
  if (part[0] && part[1] && part[2] && part[3]) {
    const at::ScalarType type = THPDtype_Check(part[3]) ? reinterpret_cast<THPDtype*>(part[3])->scalar_type : at::kFloat;
    if (half_code(type) < 0) {
      r = none();
    } else {
      PyObject* bf16 = PyLong_FromLong(type == at::kBFloat16 ? 1 : 0);
      PyObject* code = PyLong_FromLong(epi);
      if (sparse) {
        PyObject* args[] = {part[0], part[1], w, meta, scale, bias, bf16, code, part[2]};
        r = gemm_sparse(nullptr, args, 9);
      } else {
        PyObject* args[] = {part[0], part[1], w, scale, bias, bf16, code, part[2]};
        r = gemm_dense(nullptr, args, 8);
      }
      Py_XDECREF(bf16);
      Py_XDECREF(code);
    }
  }
  for (PyObject* p : part) Py_XDECREF(p);
  return r;
}

// layer_call(layer, x) -> y | None: calling an Int8Linear
PyObject* layer_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PyObject* dict = n == 2 ? plain_module(a[0], linear_class) : nullptr;
  return dict ? linear_of(a[0], dict, a[1]) : none();
}
// layer_forward(layer, x) -> y | None: Int8Linear.forward, also of subclasses
PyObject* layer_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2) return none();
  PyObject* dict = PyObject_GetAttr(a[0], names.dict);
  if (!dict) return nullptr;
  Py_DECREF(dict);
  return PyDict_Check(dict) ? linear_of(a[0], dict, a[1]) : none();
}

// A QuantizedActivation of x's shape and type.
PyObject* quantized_object(PyObject* x, at::Tensor&& q, at::Tensor&& s) {
  PyObject* r = quantized_class->tp_alloc(quantized_class, 0);
  if (!r) return nullptr;
  struct { PyObject *name, *value; } set[] = {{names.q, THPVariable_Wrap(std::move(q))},
                                              {names.act_scale, THPVariable_Wrap(std::move(s))},
                                              {names.shape, PyObject_GetAttr(x, names.shape)},
                                              {names.dtype, PyObject_GetAttr(x, names.dtype)}};
  bool bad = false;
  for (auto& e : set) {
    bad = bad || !e.value || PyObject_SetAttr(r, e.name, e.value) < 0;
    Py_XDECREF(e.value);
  }
  if (bad) { Py_DECREF(r); return nullptr; }
  return r;
}

// norm_call(layer, x) -> QuantizedActivation | None: calling an Int8LayerNorm
// norm_call(layer, x, h) -> (x + h, QuantizedActivation of its LayerNorm) | None
PyObject* norm_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  PyObject* dict = (n == 2 || n == 3) && THPVariable_CheckExact(a[1]) ? plain_module(a[0], layernorm_class) : nullptr;
  PyObject* params = dict ? PyDict_GetItemWithError(dict, names.parameters) : nullptr;
  PyObject* eps = dict ? PyDict_GetItemWithError(dict, names.eps) : nullptr;
  if (!params || !PyDict_Check(params) || !eps || !PyFloat_Check(eps)) return none();
  PyObject* gamma = PyDict_GetItemWithError(params, names.weight);
  PyObject* beta = PyDict_GetItemWithError(params, names.bias);
  Quantized z;
  int rc = 0;
  if (!gamma || !beta || !layernorm_quantize_impl(a[1], n == 3 ? a[2] : nullptr, gamma, beta, PyFloat_AS_DOUBLE(eps), &z, &rc))
    return none();
  if (rc != HY3D_OK) return failed("hy3d_layernorm_quantize", rc);
  PyObject* r = quantized_object(a[1], std::move(z.q), std::move(z.s));
  if (n == 2 || !r) return r;
  PyObject* sum = THPVariable_Wrap(std::move(z.sum));
  PyObject* pair = sum ? PyTuple_New(2) : nullptr;
  if (!pair) { Py_XDECREF(sum); Py_DECREF(r); return nullptr; }
  PyTuple_SET_ITEM(pair, 0, sum);
  PyTuple_SET_ITEM(pair, 1, r);
  return pair;
  END_HANDLE_TH_ERRORS
}

// add_quantize(x, h) -> QuantizedActivation of x + h | None
PyObject* add_quantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* x = n == 2 ? plain(a[0]) : nullptr;
  const at::Tensor* h = x ? plain(a[1]) : nullptr;
  if (!h || !quantized_class || x->dim() < 1 || h->scalar_type() != x->scalar_type() || h->device() != x->device() ||
      h->sizes() != x->sizes())
    return none();
  const int code = half_code(x->scalar_type());
  const int64_t K = x->size(-1), M = K > 0 ? x->numel() / K : 0;
  if (code < 0 || M <= 0 || (K & 7)) return none();
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  at::Tensor q = at::Tensor(at::detail::empty_cuda({M, K}, at::kChar, x->device(), std::nullopt));
  at::Tensor s = at::Tensor(at::detail::empty_cuda({M}, at::kFloat, x->device(), std::nullopt));
  const int rc = api.hy3d_add_quantize_rows(x->const_data_ptr(), h->const_data_ptr(), code, M, K, q.mutable_data_ptr<int8_t>(),
                                            s.mutable_data_ptr<float>(), st);
  if (rc != HY3D_OK) return failed("hy3d_add_quantize_rows", rc);
  return quantized_object(a[0], std::move(q), std::move(s));
  END_HANDLE_TH_ERRORS
}

// add_bias(x, bias_x | None, h | None, bias_h | None) -> round(round(x + bias_x) + round(h + bias_h)) | None
PyObject* add_bias(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* x = n == 4 ? plain_nhwc(a[0]) : nullptr;
  const at::Tensor* h = x && a[2] != Py_None ? plain_nhwc(a[2]) : nullptr;
  if (!x || (a[2] != Py_None && (!h || h->sizes() != x->sizes() || h->scalar_type() != x->scalar_type() || h->device() != x->device())))
    return none();
  const int64_t C = x->size(1);
  const void* bias[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; ++i) {
    PyObject* o = a[i ? 3 : 1];
    if (o == Py_None) continue;
    const at::Tensor* t = plain(o);
    if (!t || t->numel() != C || t->scalar_type() != x->scalar_type() || t->device() != x->device() ||
        (reinterpret_cast<uintptr_t>(t->const_data_ptr()) & 15) || (i && !h))
      return none();
    bias[i] = t->const_data_ptr();
  }
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  at::Tensor y = at::Tensor(at::detail::empty_cuda(x->sizes(), x->scalar_type(), x->device(), at::MemoryFormat::ChannelsLast));
  const int rc = api.hy3d_add_bias_nhwc(x->const_data_ptr(), bias[0], h ? h->const_data_ptr() : nullptr, bias[1],
                                        half_code(x->scalar_type()), y.mutable_data_ptr(), x->numel() / C, C, st);
  if (rc != HY3D_OK) return failed("hy3d_add_bias_nhwc", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// concat_nhwc(a, b) -> torch.cat([a, b], 1) | None
PyObject* concat_nhwc(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* x = n == 2 ? plain_nhwc(a[0]) : nullptr;
  const at::Tensor* h = x ? plain_nhwc(a[1]) : nullptr;
  if (!h || h->scalar_type() != x->scalar_type() || h->device() != x->device() || h->size(0) != x->size(0) ||
      h->size(2) != x->size(2) || h->size(3) != x->size(3))
    return none();
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  const int64_t Ca = x->size(1), Cb = h->size(1);
  at::Tensor y = at::Tensor(at::detail::empty_cuda({x->size(0), Ca + Cb, x->size(2), x->size(3)}, x->scalar_type(), x->device(),
                                                   at::MemoryFormat::ChannelsLast));
  const int rc = api.hy3d_concat_nhwc(x->const_data_ptr(), Ca, h->const_data_ptr(), Cb, y.mutable_data_ptr(), x->numel() / Ca, st);
  if (rc != HY3D_OK) return failed("hy3d_concat_nhwc", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// upsample2x_nhwc(x) -> nearest-neighbour twice the size | None
PyObject* upsample2x_nhwc(PyObject*, PyObject* px) {
  HANDLE_TH_ERRORS
  const at::Tensor* x = plain_nhwc(px);
  if (!x) return none();
  c10::cuda::CUDAGuard guard(x->device());
  cudaStream_t st = c10::cuda::getCurrentCUDAStream(x->device().index()).stream();
  at::Tensor y = at::Tensor(at::detail::empty_cuda({x->size(0), x->size(1), 2 * x->size(2), 2 * x->size(3)}, x->scalar_type(),
                                                   x->device(), at::MemoryFormat::ChannelsLast));
  const int rc = api.hy3d_upsample2x_nhwc(x->const_data_ptr(), y.mutable_data_ptr(), x->size(0), x->size(2), x->size(3), x->size(1), st);
  if (rc != HY3D_OK) return failed("hy3d_upsample2x_nhwc", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// unhooked(module, ...) -> True where calling each module is calling the `forward` of its class, so that a
// caller may do that forward's work itself
PyObject* unhooked(PyObject*, PyObject* const* a, Py_ssize_t n) {
  for (Py_ssize_t i = 0; i < n; ++i) {
    const Registered any{Py_TYPE(a[i]), _PyType_Lookup(Py_TYPE(a[i]), names.forward)};
    if (!global_hooks[0] || !plain_module(a[i], any)) Py_RETURN_FALSE;
  }
  Py_RETURN_TRUE;
}

// bias_apart(x, conv, ...) -> True where running these convolutions on x without their bias and adding it after
// gives the bits of running them whole.  That is how torch itself runs a cuDNN convolution of a 16-bit type; with
// autocast the operands change type on the way, the depthwise and the non-cuDNN kernels add the bias before they
// round, and a hook or a replaced forward has to see the whole call.
PyObject* bias_apart(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 2 || !THPVariable_CheckExact(a[0]) || !global_hooks[0]) Py_RETURN_FALSE;
  const at::Tensor& x = THPVariable_Unpack(a[0]);
  if (!x.is_cuda() || half_code(x.scalar_type()) < 0 || at::autocast::is_autocast_enabled(at::kCUDA) ||
      !at::globalContext().userEnabledCuDNN())
    Py_RETURN_FALSE;
  for (Py_ssize_t i = 1; i < n; ++i) {
    const Registered any{Py_TYPE(a[i]), _PyType_Lookup(Py_TYPE(a[i]), names.forward)};
    PyObject* dict = plain_module(a[i], any);
    PyObject* params = dict ? PyDict_GetItemWithError(dict, names.parameters) : nullptr;
    PyObject* conv_groups = dict ? PyDict_GetItemWithError(dict, names.conv_groups) : nullptr;
    long one = 0;
    if (!params || !PyDict_Check(params) || !conv_groups || !small_int(conv_groups, 1, 1, &one)) Py_RETURN_FALSE;
    for (PyObject* name : {names.weight, names.bias}) {
      PyObject* o = PyDict_GetItemWithError(params, name);
      if (!o || (o == Py_None && name == names.weight)) Py_RETURN_FALSE;
      if (o == Py_None) continue;
      if (!THPVariable_CheckExact(o)) Py_RETURN_FALSE;
      const at::Tensor& t = THPVariable_Unpack(o);
      if (t.scalar_type() != x.scalar_type() || t.device() != x.device()) Py_RETURN_FALSE;
    }
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// groupnorm_call(layer, x, add | None, bias | None) -> y | None: calling a GroupNormNHWC whose kernel path is
// on; `bias` is that of the convolution that made x and is added first
PyObject* groupnorm_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  PyObject* dict = n == 4 ? plain_module(a[0], groupnorm_class) : nullptr;
  if (!dict || PyDict_GetItemWithError(dict, names.fused) != Py_True) return none();
  PyObject* params = PyDict_GetItemWithError(dict, names.parameters);
  PyObject* eps = PyDict_GetItemWithError(dict, names.eps);
  PyObject* silu = PyDict_GetItemWithError(dict, names.silu);
  PyObject* ng = PyDict_GetItemWithError(dict, names.groups);
  long groups = 0;
  if (!params || !PyDict_Check(params) || !eps || !PyFloat_Check(eps) || !silu || !ng || !small_int(ng, 1, 1 << 20, &groups))
    return none();
  PyObject* gamma = PyDict_GetItemWithError(params, names.weight);
  PyObject* beta = PyDict_GetItemWithError(params, names.bias);
  return gamma && beta ? groupnorm_impl(a[1], groups, gamma, beta, PyFloat_AS_DOUBLE(eps), silu == Py_True, a[2], a[3]) : none();
}

// open(path): resolves the C ABI in the library at `path`, which the caller has loaded and checked.
PyObject* open_library(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!h) {
    PyErr_Format(PyExc_RuntimeError, "%s", dlerror());
    return nullptr;
  }
#define HY3D_SYM(name)                                                                       \
  do {                                                                                       \
    api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, #name));                        \
    if (!api.name) {                                                                         \
      PyErr_Format(PyExc_RuntimeError, "%s has no symbol %s", path, #name);                  \
      return nullptr;                                                                        \
    }                                                                                        \
  } while (0)
  HY3D_SYM(hy3d_linear_w8a8_dense);
  HY3D_SYM(hy3d_gemm_w8a8_dense);
  HY3D_SYM(hy3d_dense_layer_splitk_plan);
  HY3D_SYM(hy3d_gemm_w8a8_dense_splitk);
  HY3D_SYM(hy3d_quantize_rows);
  HY3D_SYM(hy3d_linear_cluster_plan);
  HY3D_SYM(hy3d_linear_w8a8_cluster);
  HY3D_SYM(hy3d_linear_w8a8_sparse24);
  HY3D_SYM(hy3d_gemm_w8a8_sparse24);
  HY3D_SYM(hy3d_layernorm_quantize);
  HY3D_SYM(hy3d_groupnorm_nhwc_terms);
  HY3D_SYM(hy3d_add_bias_nhwc);
  HY3D_SYM(hy3d_concat_nhwc);
  HY3D_SYM(hy3d_upsample2x_nhwc);
  HY3D_SYM(hy3d_add_quantize_rows);
  HY3D_SYM(hy3d_add_layernorm_quantize);
  HY3D_SYM(hy3d_quantize_weight);
  HY3D_SYM(hy3d_status_string);
#undef HY3D_SYM
  Py_RETURN_NONE;
}

#define HY3D_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"open", open_library, METH_O, nullptr},
    HY3D_FAST(register_modules),
    HY3D_FAST(layer_call),
    HY3D_FAST(layer_forward),
    HY3D_FAST(norm_call),
    HY3D_FAST(groupnorm_call),
    HY3D_FAST(add_quantize),
    HY3D_FAST(add_bias),
    HY3D_FAST(concat_nhwc),
    {"upsample2x_nhwc", upsample2x_nhwc, METH_O, nullptr},
    HY3D_FAST(unhooked),
    HY3D_FAST(bias_apart),
    HY3D_FAST(linear_dense),
    HY3D_FAST(linear_sparse),
    HY3D_FAST(gemm_dense),
    HY3D_FAST(gemm_sparse),
    HY3D_FAST(layernorm_quantize),
    HY3D_FAST(groupnorm_nhwc),
    HY3D_FAST(quantize_weight),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "hy3d_torch", "Native host path of the INT8 layers.", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_hy3d_torch(void) {
  if (!intern_names()) return nullptr;
  PyObject* m = PyModule_Create(&module_def);
  if (m) PyModule_AddStringConstant(m, "source_digest", HY3D_EXT_DIGEST);
  return m;
}
