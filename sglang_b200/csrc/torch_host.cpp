// Native host path of the torch-facing functions (module sglang_b200._host).
//
// A decode-size linear is 10-20 us of device work; the Python-level sequence in front of it (argument checks, one
// torch.empty per intermediate, a ctypes call with a dozen arguments per kernel) took 60-80 us, a fused expert layer
// 240 us.  Each function here does the allocation and the C-ABI call(s) of one public function in one native call.
//
// Every function looks at its arguments first and returns None when they are not the plain case (CPU or non-contiguous
// tensors, another dtype, a size its caller would reject): the Python function then runs its own checks, which raise
// what they always raised.  Nothing is launched in that case.
#include <Python.h>

#include <ATen/EmptyTensor.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/b200_block_fp8.h"

namespace {

using at::Tensor;

int dt_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return B200_DT_F32;
    case at::kHalf: return B200_DT_F16;
    case at::kBFloat16: return B200_DT_BF16;
    default: return -1;
  }
}
bool is_16bit(at::ScalarType t) { return t == at::kHalf || t == at::kBFloat16; }

// A tensor whose memory this library may use directly: dense CUDA storage, no lazy negation or conjugation.
const Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.is_neg() || t.is_conj()) return nullptr;
  if (t.unsafeGetTensorImpl()->key_set().has(c10::DispatchKey::Python)) return nullptr;
  return &t;
}
const Tensor* cuda_tensor(PyObject* o, at::ScalarType dtype) {
  const Tensor* t = cuda_tensor(o);
  return t && t->scalar_type() == dtype ? t : nullptr;
}

Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& dev) {
  return at::detail::empty_cuda(sizes, dtype, dev, std::nullopt);
}
Tensor empty_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType dtype, const at::Device& dev) {
  return at::detail::empty_strided_cuda(sizes, strides, dtype, dev);
}

void* stream_of(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

PyObject* none() { Py_RETURN_NONE; }

// The interpreter lock is free while this lives.  Allocating may wait for the device and a launch for room in the queue;
// the process's other Python threads go on meanwhile, as they do under a ctypes call.  Everything that is read from a
// Python-owned tensor is read before; tensors held by value are fine.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  NoGil() = default;
  NoGil(const NoGil&) = delete;
  NoGil& operator=(const NoGil&) = delete;
  ~NoGil() { PyEval_RestoreThread(state); }
};

// Raises _lib.B200Error(fn, code, detail), the exception the Python functions raise.
PyObject* raise_status(const char* fn, int code) {
  PyObject* mod = PyImport_ImportModule("sglang_b200._lib");
  if (mod) {
    PyObject* r = PyObject_CallMethod(mod, "check", "si", fn, code);
    Py_XDECREF(r);
    Py_DECREF(mod);
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed (code %d)", fn, code);
  }
  return nullptr;
}

int64_t align4(int64_t v) { return (v + 3) / 4 * 4; }

// Scale tensor of sglang_per_token_group_quant_fp8 for x [..., K] of these sizes seen as [M, K]; `rs` and `gs` are its
// strides.
// Packed words are zero-filled where the quantiser may leave bytes alone (`partial`) or rows are padding.
Tensor scale_tensor(std::vector<int64_t> sizes, int64_t K, int64_t M, int64_t group, bool col_major, bool aligned, bool ue8m0,
                    bool partial, const at::Device& dev, int64_t& rs, int64_t& gs) {
  const int64_t G = K / group;
  if (ue8m0) {
    const int64_t W = (G + 3) / 4, ld = align4(M);
    rs = 1;
    gs = ld;
    Tensor whole = empty({W, ld}, at::kInt, dev);
    if (ld != M || (partial && G % 4 != 0))
      C10_CUDA_CHECK(cudaMemsetAsync(whole.data_ptr(), 0, W * ld * 4, static_cast<cudaStream_t>(stream_of(dev))));
    return whole.transpose(0, 1).narrow(0, 0, M);
  }
  if (col_major) {      // 2-D only (checked by the callers)
    const int64_t ld = aligned ? align4(M) : M;
    rs = 1;
    gs = ld;
    if (ld == M) return empty_strided({M, G}, {1, M}, at::kFloat, dev);
    return empty({G, ld}, at::kFloat, dev).transpose(0, 1).narrow(0, 0, M);
  }
  rs = G;
  gs = 1;
  sizes.back() = G;
  return empty(sizes, at::kFloat, dev);
}

PyObject* pair_of(Tensor a, Tensor b) {
  PyObject* pa = THPVariable_Wrap(std::move(a));
  PyObject* pb = THPVariable_Wrap(std::move(b));
  PyObject* r = PyTuple_Pack(2, pa, pb);
  Py_DECREF(pa);
  Py_DECREF(pb);
  return r;
}

#define HOST_FN(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n) try
#define HOST_END                                        \
  catch (const std::exception& e) {                     \
    PyErr_SetString(PyExc_RuntimeError, e.what());      \
    return nullptr;                                     \
  }

// linear(x, weight, weight_scale, bias | None, out | None, scale_mode)
//   scale_mode 0: fp32 scales; 1: power-of-two activation scales; 2: power-of-two weight scales as well
HOST_FN(linear) {
  if (n != 6) return none();
  const Tensor *x = cuda_tensor(a[0]), *w = cuda_tensor(a[1], at::kFloat8_e4m3fn), *ws = cuda_tensor(a[2], at::kFloat);
  if (!x || !w || !ws || !is_16bit(x->scalar_type()) || x->dim() < 1 || w->dim() != 2 || ws->dim() != 2) return none();
  const int64_t K = w->size(1), N = w->size(0);
  long mode = PyLong_AsLong(a[5]);
  if (K <= 0 || N <= 0 || x->size(-1) != K || K % 128 != 0 || !x->is_contiguous() || !w->is_contiguous()) return none();
  if (ws->size(0) != (N + 127) / 128 || ws->size(1) != K / 128) return none();
  if (N % 128 == 0 && ws->stride(1) != 1) return none();
  if (N % 8 != 0 || w->device() != x->device() || ws->device() != x->device()) return none();
  if (mode != 0 && (x->scalar_type() != at::kBFloat16 || N % 128 != 0)) return none();
  const int64_t M = x->numel() / K;
  if (M == 0) return none();
  const Tensor* bias = nullptr;
  if (a[3] != Py_None) {
    bias = cuda_tensor(a[3], x->scalar_type());
    if (!bias || bias->dim() != 1 || bias->size(0) != N || !bias->is_contiguous() || bias->device() != x->device())
      return none();
  }
  const at::Device dev = x->device();
  const at::ScalarType xt = x->scalar_type();
  Tensor out;
  int64_t ldo = N;
  auto out_sizes = x->sizes().vec();
  out_sizes.back() = N;
  if (a[4] != Py_None) {
    const Tensor* o = cuda_tensor(a[4], xt);
    if (!o || o->dim() != 2 || o->size(0) != M || o->size(1) != N || o->stride(1) != 1 || o->stride(0) < N ||
        o->device() != dev || x->dim() != 2)
      return none();
    ldo = o->stride(0);
    out = *o;
  }
  const void *xp = x->data_ptr(), *wp = w->data_ptr(), *bp = bias ? bias->data_ptr() : nullptr;
  const float* wsp = static_cast<const float*>(ws->data_ptr());
  const int64_t ws_n = ws->stride(0), ws_g = ws->stride(1);
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    if (!out.defined()) out = empty(out_sizes, xt, dev);
    const size_t bytes = b200_fp8_linear_workspace_bytes(M, N, K, static_cast<int>(mode));
    const Tensor work = empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    rc = b200_fp8_linear(xp, dt_of(xt), wp, K, wsp, ws_n, ws_g, bp, out.data_ptr(), ldo, M, N, K, static_cast<int>(mode),
                         work.data_ptr(), bytes, stream_of(dev));
  }
  if (rc != 0) return raise_status("fp8_linear", rc);
  return THPVariable_Wrap(std::move(out));
}
HOST_END

// quant(x, group_size, eps, column_major, aligned, ue8m0) -> (codes, scales)
HOST_FN(quant) {
  if (n != 6) return none();
  const Tensor* x = cuda_tensor(a[0]);
  if (!x || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0) return none();
  const int dt = dt_of(x->scalar_type());
  const int64_t group = PyLong_AsLong(a[1]), K = x->size(-1);
  if (dt < 0 || (group != 64 && group != 128 && group != 256 && group != 512) || K % group != 0) return none();
  const double eps = PyFloat_AsDouble(a[2]);
  const bool col = PyObject_IsTrue(a[3]), aligned = PyObject_IsTrue(a[4]), ue8m0 = PyObject_IsTrue(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if ((col || ue8m0) && x->dim() != 2) return none();
  if (ue8m0 && !(col && aligned && group == 128)) return none();
  const at::Device dev = x->device();
  const int64_t M = x->numel() / K;
  const auto sizes = x->sizes().vec();
  const void* xp = x->data_ptr();
  Tensor q, s;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    q = empty(sizes, at::kFloat8_e4m3fn, dev);
    int64_t rs, gs;
    s = scale_tensor(sizes, K, M, group, col, aligned, ue8m0, false, dev, rs, gs);
    void* st = stream_of(dev);
    rc = ue8m0 ? b200_per_token_group_quant_fp8_ue8m0(xp, dt, q.data_ptr(), static_cast<uint32_t*>(s.data_ptr()), M, K, gs,
                                                      static_cast<float>(eps), -448.0f, 448.0f, st)
               : b200_per_token_group_quant_fp8(xp, dt, q.data_ptr(), static_cast<float*>(s.data_ptr()), M, K, group, rs, gs,
                                                static_cast<float>(eps), -448.0f, 448.0f, st);
  }
  if (rc != 0) return raise_status("sgl_per_token_group_quant_fp8", rc);
  return pair_of(std::move(q), std::move(s));
}
HOST_END

// norm_quant(x, weight, norm_eps, residual | None, eps, column_major, aligned, ue8m0) -> (codes, scales)
HOST_FN(norm_quant) {
  if (n != 8) return none();
  const Tensor* x = cuda_tensor(a[0]);
  if (!x || !is_16bit(x->scalar_type()) || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0) return none();
  const Tensor* w = cuda_tensor(a[1], x->scalar_type());
  const int64_t K = x->size(-1), M = x->numel() / K;
  if (!w || w->dim() != 1 || w->size(0) != K || !w->is_contiguous() || K % 128 != 0 || K > 16384) return none();
  const double norm_eps = PyFloat_AsDouble(a[2]), eps = PyFloat_AsDouble(a[4]);
  const Tensor* r = nullptr;
  if (a[3] != Py_None) {
    r = cuda_tensor(a[3], x->scalar_type());
    if (!r || r->sizes() != x->sizes() || !r->is_contiguous() || r->device() != x->device()) return none();
  }
  const bool col = PyObject_IsTrue(a[5]), aligned = PyObject_IsTrue(a[6]), ue8m0 = PyObject_IsTrue(a[7]);
  if (PyErr_Occurred()) return nullptr;
  if (x->dim() != 2 || (ue8m0 && !(col && aligned)) || w->device() != x->device()) return none();
  const at::Device dev = x->device();
  const auto sizes = x->sizes().vec();
  const int dt = dt_of(x->scalar_type());
  const void *xp = x->data_ptr(), *wp = w->data_ptr();
  void* rp = r ? r->data_ptr() : nullptr;
  Tensor q, s;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    q = empty(sizes, at::kFloat8_e4m3fn, dev);
    int64_t rs, gs;
    s = scale_tensor(sizes, K, M, 128, col, aligned, ue8m0, true, dev, rs, gs);
    rc = b200_rmsnorm_per_token_group_quant_fp8(xp, dt, rp, wp, static_cast<float>(norm_eps), nullptr, q.data_ptr(),
                                                s.data_ptr(), M, K, rs, gs, ue8m0 ? 1 : 0, static_cast<float>(eps), -448.0f,
                                                448.0f, stream_of(dev));
  }
  if (rc != 0) return raise_status("rmsnorm_per_token_group_quant_fp8", rc);
  return pair_of(std::move(q), std::move(s));
}
HOST_END

// silu_and_mul(x) -> out
HOST_FN(silu_and_mul) {
  if (n != 1) return none();
  const Tensor* x = cuda_tensor(a[0]);
  if (!x || !is_16bit(x->scalar_type()) || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0) return none();
  const int64_t d2 = x->size(-1), d = d2 / 2;
  if (d2 % 16 != 0) return none();
  const at::Device dev = x->device();
  const at::ScalarType xt = x->scalar_type();
  auto sizes = x->sizes().vec();
  sizes.back() = d;
  const int64_t rows = x->numel() / d2;
  const void* xp = x->data_ptr();
  Tensor out;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    out = empty(sizes, xt, dev);
    rc = b200_silu_and_mul(xp, out.data_ptr(), rows, d, dt_of(xt), stream_of(dev));
  }
  if (rc != 0) return raise_status("silu_and_mul", rc);
  return THPVariable_Wrap(std::move(out));
}
HOST_END

// matmul(a [M, K], b [N, K], a_scale [M, K/128], b_scale [N/128, K/128], out_dtype) -> [M, N]: fp32 scales, any strides
HOST_FN(matmul) {
  if (n != 5) return none();
  const Tensor *x = cuda_tensor(a[0], at::kFloat8_e4m3fn), *w = cuda_tensor(a[1], at::kFloat8_e4m3fn),
               *xs = cuda_tensor(a[2], at::kFloat), *ws = cuda_tensor(a[3], at::kFloat);
  if (!x || !w || !xs || !ws || !THPDtype_Check(a[4])) return none();
  if (x->dim() != 2 || w->dim() != 2 || xs->dim() != 2 || ws->dim() != 2 || !x->is_contiguous() || !w->is_contiguous())
    return none();
  const at::ScalarType ot = reinterpret_cast<THPDtype*>(a[4])->scalar_type;
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  if (dt_of(ot) < 0 || M == 0 || N == 0 || w->size(1) != K || K % 128 != 0 || N % 8 != 0) return none();
  if (xs->size(0) != M || xs->size(1) != K / 128 || ws->size(0) != (N + 127) / 128 || ws->size(1) != K / 128) return none();
  const at::Device dev = x->device();
  if (w->device() != dev || xs->device() != dev || ws->device() != dev) return none();
  const void *xp = x->data_ptr(), *wp = w->data_ptr();
  const float *xsp = static_cast<const float*>(xs->data_ptr()), *wsp = static_cast<const float*>(ws->data_ptr());
  const int64_t xs_m = xs->stride(0), xs_g = xs->stride(1), ws_n = ws->stride(0), ws_g = ws->stride(1);
  Tensor out;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    out = empty({M, N}, ot, dev);
    const size_t bytes = b200_fp8_blockwise_scaled_mm_workspace_bytes(M, N, K);
    Tensor work;
    if (bytes) work = empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    rc = b200_fp8_blockwise_scaled_mm_splitk(xp, K, wp, K, xsp, xs_m, xs_g, wsp, ws_n, ws_g, out.data_ptr(), N, dt_of(ot), M,
                                             N, K, 0, bytes ? work.data_ptr() : nullptr, bytes, stream_of(dev));
  }
  if (rc != 0) return raise_status("w8a8_block_fp8_matmul", rc);
  return THPVariable_Wrap(std::move(out));
}
HOST_END

// matmul_packed(a [M, K], b [N, K], a_words int32 [M, K/512], b_scale [N/128, K/128], weights_pow2) -> bf16 [M, N]
HOST_FN(matmul_packed) {
  if (n != 5) return none();
  const Tensor *x = cuda_tensor(a[0], at::kFloat8_e4m3fn), *w = cuda_tensor(a[1], at::kFloat8_e4m3fn),
               *xs = cuda_tensor(a[2], at::kInt), *ws = cuda_tensor(a[3], at::kFloat);
  if (!x || !w || !xs || !ws) return none();
  if (x->dim() != 2 || w->dim() != 2 || xs->dim() != 2 || ws->dim() != 2 || !x->is_contiguous() || !w->is_contiguous())
    return none();
  const int64_t M = x->size(0), K = x->size(1), N = w->size(0);
  if (M == 0 || N == 0 || w->size(1) != K || K % 128 != 0 || N % 128 != 0) return none();
  if (xs->size(0) != M || xs->size(1) != (K / 128 + 3) / 4 || (xs->stride(0) != 1 && M != 1)) return none();
  if (ws->size(0) != N / 128 || ws->size(1) != K / 128) return none();
  const at::Device dev = x->device();
  if (w->device() != dev || xs->device() != dev || ws->device() != dev) return none();
  const bool pow2 = PyObject_IsTrue(a[4]);
  const void *xp = x->data_ptr(), *wp = w->data_ptr();
  const uint32_t* xsp = static_cast<const uint32_t*>(xs->data_ptr());
  const float* wsp = static_cast<const float*>(ws->data_ptr());
  const int64_t xs_m = xs->stride(0), xs_g = xs->stride(1), ws_n = ws->stride(0), ws_g = ws->stride(1);
  Tensor out;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    out = empty({M, N}, at::kBFloat16, dev);
    rc = (pow2 ? b200_fp8_blockwise_scaled_mm_pow2 : b200_fp8_blockwise_scaled_mm_ue8m0)(
        xp, K, wp, K, xsp, xs_m, xs_g, wsp, ws_n, ws_g, out.data_ptr(), N, B200_DT_BF16, M, N, K, stream_of(dev));
  }
  if (rc != 0) return raise_status("w8a8_block_fp8_matmul_deepgemm", rc);
  return THPVariable_Wrap(std::move(out));
}
HOST_END

// gate_up_silu_quant(a [M, K], a_words, w [2n, K], w_scale [2n/128, K/128], mid_dtype) -> (codes [M, n], words)
HOST_FN(gate_up_silu_quant) {
  if (n != 5) return none();
  const Tensor *x = cuda_tensor(a[0], at::kFloat8_e4m3fn), *xs = cuda_tensor(a[1], at::kInt),
               *w = cuda_tensor(a[2], at::kFloat8_e4m3fn), *ws = cuda_tensor(a[3], at::kFloat);
  if (!x || !w || !xs || !ws || !THPDtype_Check(a[4])) return none();
  const at::ScalarType mid = reinterpret_cast<THPDtype*>(a[4])->scalar_type;
  if (!is_16bit(mid) || x->dim() != 2 || w->dim() != 2 || xs->dim() != 2 || ws->dim() != 2 || !x->is_contiguous() ||
      !w->is_contiguous())
    return none();
  const int64_t M = x->size(0), K = x->size(1), n2 = w->size(0), N = n2 / 2;
  if (M == 0 || w->size(1) != K || K % 128 != 0 || n2 % 256 != 0 || n2 == 0) return none();
  if (xs->size(0) != M || xs->size(1) < (K / 128 + 3) / 4 || ws->size(0) != n2 / 128 || ws->size(1) != K / 128) return none();
  const at::Device dev = x->device();
  if (w->device() != dev || xs->device() != dev || ws->device() != dev) return none();
  const auto sizes = x->sizes().vec();
  const void *xp = x->data_ptr(), *wp = w->data_ptr();
  const uint32_t* xsp = static_cast<const uint32_t*>(xs->data_ptr());
  const float* wsp = static_cast<const float*>(ws->data_ptr());
  const int64_t xs_m = xs->stride(0), xs_g = xs->stride(1), ws_n = ws->stride(0), ws_g = ws->stride(1);
  Tensor q, s;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    q = empty({M, N}, at::kFloat8_e4m3fn, dev);
    int64_t rs, gs;
    s = scale_tensor(sizes, N, M, 128, true, true, true, true, dev, rs, gs);
    rc = b200_fp8_gate_up_silu_quant_pow2(xp, K, wp, K, xsp, xs_m, xs_g, wsp, ws_n, ws_g, q.data_ptr(), N,
                                          static_cast<uint32_t*>(s.data_ptr()), gs, dt_of(mid), M, N, K, stream_of(dev));
  }
  if (rc != 0) return raise_status("gate_up_silu_quant_pow2", rc);
  return pair_of(std::move(q), std::move(s));
}
HOST_END

// topk_softmax(logits [m, E], topk, renormalize) -> (weights fp32 [m, topk], ids int32 [m, topk])
HOST_FN(topk_softmax) {
  if (n != 3) return none();
  const Tensor* x = cuda_tensor(a[0]);
  if (!x || x->dim() != 2 || dt_of(x->scalar_type()) < 0 || x->stride(1) != 1) return none();
  const int64_t m = x->size(0), E = x->size(1), topk = PyLong_AsLong(a[1]);
  if (m == 0 || topk <= 0 || topk > E || topk > 32 || E > 1024 || x->stride(0) < E) return none();
  const at::Device dev = x->device();
  const int dt = dt_of(x->scalar_type()), renormalize = PyObject_IsTrue(a[2]) ? 1 : 0;
  const int64_t ld = x->stride(0);
  const void* xp = x->data_ptr();
  Tensor w, ids;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    w = empty({m, topk}, at::kFloat, dev);
    ids = empty({m, topk}, at::kInt, dev);
    rc = b200_topk_softmax(xp, dt, ld, static_cast<float*>(w.data_ptr()), static_cast<int32_t*>(ids.data_ptr()), m,
                           static_cast<int>(E), static_cast<int>(topk), renormalize, stream_of(dev));
  }
  if (rc != 0) return raise_status("topk_softmax", rc);
  return pair_of(std::move(w), std::move(ids));
}
HOST_END

// fused_gate(logits, bias, num_expert_group, topk_group, topk, num_fused_shared_experts, routed_scaling_factor)
HOST_FN(fused_gate) {
  if (n != 7) return none();
  const Tensor *x = cuda_tensor(a[0], at::kFloat), *b = cuda_tensor(a[1], at::kFloat);
  if (!x || !b || x->dim() != 2 || b->dim() != 1 || b->numel() != x->size(1) || x->stride(1) != 1 || !b->is_contiguous())
    return none();
  const int64_t m = x->size(0), E = x->size(1);
  const long groups = PyLong_AsLong(a[2]), tg = PyLong_AsLong(a[3]), topk = PyLong_AsLong(a[4]), shared = PyLong_AsLong(a[5]);
  const double factor = PyFloat_AsDouble(a[6]);
  if (PyErr_Occurred()) return nullptr;
  if (m == 0 || b->device() != x->device() || groups <= 0 || groups > 32 || E % groups != 0 || E / groups < 2 || E > 1024)
    return none();
  if (tg <= 0 || tg > groups || topk > 32 || shared < 0 || topk - shared <= 0 || topk - shared > tg * (E / groups) ||
      (shared > 0 && factor == 0.0) || x->stride(0) < E)
    return none();
  const at::Device dev = x->device();
  const int64_t ld = x->stride(0);
  const float *xp = static_cast<const float*>(x->data_ptr()), *bp = static_cast<const float*>(b->data_ptr());
  Tensor w, ids;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    w = empty({m, topk}, at::kFloat, dev);
    ids = empty({m, topk}, at::kInt, dev);
    rc = b200_moe_fused_gate_shared_experts(xp, ld, bp, static_cast<float*>(w.data_ptr()),
                                            static_cast<int32_t*>(ids.data_ptr()), m, static_cast<int>(E),
                                            static_cast<int>(groups), static_cast<int>(tg), static_cast<int>(topk),
                                            static_cast<int>(shared), shared ? factor : 1.0, stream_of(dev));
  }
  if (rc != 0) return raise_status("moe_fused_gate", rc);
  return pair_of(std::move(w), std::move(ids));
}
HOST_END

// experts(x [m, k], w13 [E, 2n, k], w2 [E, k, n], w13_scale, w2_scale, topk_weights, topk_ids, expert_offsets | None,
//         problem_sizes1 | None, problem_sizes2 | None, ue8m0) -> [m, k]
HOST_FN(experts) {
  if (n != 11) return none();
  const Tensor *x = cuda_tensor(a[0]), *w13 = cuda_tensor(a[1], at::kFloat8_e4m3fn), *w2 = cuda_tensor(a[2], at::kFloat8_e4m3fn),
               *s13 = cuda_tensor(a[3], at::kFloat), *s2 = cuda_tensor(a[4], at::kFloat), *tw = cuda_tensor(a[5], at::kFloat),
               *ti = cuda_tensor(a[6], at::kInt);
  if (!x || !w13 || !w2 || !s13 || !s2 || !tw || !ti || !is_16bit(x->scalar_type())) return none();
  if (x->dim() != 2 || w13->dim() != 3 || w2->dim() != 3 || s13->dim() != 3 || s2->dim() != 3 || tw->dim() != 2 || ti->dim() != 2)
    return none();
  const at::Device dev = x->device();
  for (const Tensor* t : {x, w13, w2, s13, s2, tw, ti})
    if (!t->is_contiguous() || t->device() != dev) return none();
  const int64_t m = x->size(0), k = x->size(1), E = w13->size(0), N = w2->size(2), topk = ti->size(1);
  if (m == 0 || E == 0 || topk == 0 || N == 0 || k == 0 || N % 128 != 0 || k % 128 != 0) return none();
  if (w13->size(1) != 2 * N || w13->size(2) != k || w2->size(0) != E || w2->size(1) != k || ti->size(0) != m ||
      tw->sizes() != ti->sizes())
    return none();
  if (s13->size(0) != E || s13->size(1) != 2 * N / 128 || s13->size(2) != k / 128 || s2->size(0) != E ||
      s2->size(1) != k / 128 || s2->size(2) != N / 128)
    return none();
  int32_t* tables[3] = {nullptr, nullptr, nullptr};
  for (int i = 0; i < 3; ++i) {
    if (a[7 + i] == Py_None) continue;
    const Tensor* t = cuda_tensor(a[7 + i], at::kInt);
    if (!t || !t->is_contiguous() || t->device() != dev || t->numel() != (i == 0 ? E + 1 : 3 * E)) return none();
    tables[i] = static_cast<int32_t*>(t->data_ptr());
  }
  const int ue8m0 = PyObject_IsTrue(a[10]) ? 1 : 0;
  const at::ScalarType xt = x->scalar_type();
  const void *xp = x->data_ptr(), *w13p = w13->data_ptr(), *w2p = w2->data_ptr();
  const float *s13p = static_cast<const float*>(s13->data_ptr()), *s2p = static_cast<const float*>(s2->data_ptr()),
              *twp = static_cast<const float*>(tw->data_ptr());
  const int32_t* tip = static_cast<const int32_t*>(ti->data_ptr());
  Tensor out;
  int rc;
  {
    const NoGil no_gil;
    const c10::cuda::OptionalCUDAGuard guard(dev);
    out = empty({m, k}, xt, dev);
    const size_t bytes = b200_fused_experts_fp8_workspace_bytes(m, k, N, static_cast<int>(topk), static_cast<int>(E), ue8m0);
    const Tensor work = empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    rc = b200_fused_experts_fp8(xp, dt_of(xt), w13p, w2p, s13p, s2p, twp, tip, m, k, N, static_cast<int>(topk),
                                static_cast<int>(E), tables[0], tables[1], tables[2], out.data_ptr(), ue8m0,
                                work.data_ptr(), bytes, stream_of(dev));
  }
  if (rc != 0) return raise_status("fused_experts_fp8", rc);
  return THPVariable_Wrap(std::move(out));
}
HOST_END

#define ENTRY(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(linear),        ENTRY(quant),         ENTRY(norm_quant),         ENTRY(silu_and_mul),
                         ENTRY(matmul),        ENTRY(matmul_packed), ENTRY(gate_up_silu_quant), ENTRY(topk_softmax),
                         ENTRY(fused_gate),    ENTRY(experts),       {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }
