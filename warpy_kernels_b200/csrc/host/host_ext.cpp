// The host side of the entry points' common case, as a CPython module (warpy_kernels_b200/_host.so).
//
// A call of attn_fwd, attn_bwd, gemm or quantize_mx costs 20-70 us of interpreter time when its checks, its output
// tensors and its argument block are made in Python, which is more than the kernels of a small problem take.  Here
// the same work takes 3-6 us: arguments are read from the vectorcall array, outputs come from the caching allocator
// without going through the dispatcher, and the C ABI entry point is called with the GIL released.
//
// Every function returns None for anything but the plain, valid case (a wrong shape or dtype, a tensor that needs a
// copy, an unknown option): the Python function of the same name then does the call, copies and raises as documented.
// So this file repeats conditions, never messages.  The kernels are reached through the C ABI of libwarpy_b200.so,
// whose addresses _lib.py hands over (bind()), so that another build of that library can be used.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cmath>
#include <cstring>
#include <exception>
#include <map>
#include <string>
#include <unordered_map>
#include <utility>

#include "../../../include/warpy_b200.h"

namespace {

// ---- the C ABI --------------------------------------------------------------------------------------------------
struct Abi {
  int (*device_arch)(int);
  const char* (*error_string)(int);
  int (*attn_fwd_fp8)(const wk_attn_fwd_args*, void*);
  int (*attn_fwd_bf16)(const wk_attn_fwd_args*, void*);
  int64_t (*attn_fwd_workspace_bytes)(int, int, int);
  int (*attn_bwd_fp8)(const wk_attn_bwd_args*, void*);
  int (*attn_bwd_bf16)(const wk_attn_bwd_args*, void*);
  int64_t (*attn_bwd_fp8_workspace_bytes)(int, int, int);
  int64_t (*attn_bwd_bf16_workspace_bytes)(int, int, int);
  int (*gemm_16bit)(const wk_gemm16_args*, void*);
  int (*gemm_mxfp8)(const wk_gemm_mx_args*, void*);
  int64_t (*gemm_mxfp8_workspace_bytes)(int, int, int);
  int (*quantize_mx)(const void*, int, int64_t, int64_t, int64_t, void*, void*, void*);
} abi;
bool bound = false;

const struct {
  const char* name;
  void** slot;
} kSymbols[] = {
    {"wk_device_arch", reinterpret_cast<void**>(&abi.device_arch)},
    {"wk_error_string", reinterpret_cast<void**>(&abi.error_string)},
    {"wk_attn_fwd_fp8", reinterpret_cast<void**>(&abi.attn_fwd_fp8)},
    {"wk_attn_fwd_bf16", reinterpret_cast<void**>(&abi.attn_fwd_bf16)},
    {"wk_attn_fwd_workspace_bytes", reinterpret_cast<void**>(&abi.attn_fwd_workspace_bytes)},
    {"wk_attn_bwd_fp8", reinterpret_cast<void**>(&abi.attn_bwd_fp8)},
    {"wk_attn_bwd_bf16", reinterpret_cast<void**>(&abi.attn_bwd_bf16)},
    {"wk_attn_bwd_fp8_workspace_bytes", reinterpret_cast<void**>(&abi.attn_bwd_fp8_workspace_bytes)},
    {"wk_attn_bwd_bf16_workspace_bytes", reinterpret_cast<void**>(&abi.attn_bwd_bf16_workspace_bytes)},
    {"wk_gemm_16bit", reinterpret_cast<void**>(&abi.gemm_16bit)},
    {"wk_gemm_mxfp8", reinterpret_cast<void**>(&abi.gemm_mxfp8)},
    {"wk_gemm_mxfp8_workspace_bytes", reinterpret_cast<void**>(&abi.gemm_mxfp8_workspace_bytes)},
    {"wk_quantize_mx", reinterpret_cast<void**>(&abi.quantize_mx)},
};

constexpr int kMaxDevices = 64;
constexpr int kArch = 100;

// Whether the library has kernels for CUDA device `dev` (asked once per device).
bool device_ok(int dev) {
  static signed char known[kMaxDevices] = {};  // 0 not asked, 1 yes; guarded by the GIL
  if (dev < 0 || dev >= kMaxDevices) return false;
  if (!known[dev] && abi.device_arch(dev) == kArch) known[dev] = 1;
  return known[dev] == 1;
}

// ---- arguments --------------------------------------------------------------------------------------------------
// The values of a fixed list of parameter names, from the positional and keyword arguments of a vectorcall.
template <int N>
struct Params {
  std::array<PyObject*, N> v{};

  // False if an argument is not in the list (the Python function decides what that means).
  bool read(const std::array<PyObject*, N>& names, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
    if (nargs > N) return false;
    for (Py_ssize_t i = 0; i < nargs; ++i) v[i] = args[i];
    const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
    for (Py_ssize_t j = 0; j < nkw; ++j) {
      PyObject* key = PyTuple_GET_ITEM(kwnames, j);
      int at = -1;
      for (int i = 0; i < N && at < 0; ++i)  // keyword names of a call site are interned: the pointers are equal
        if (names[i] == key) at = i;
      for (int i = 0; i < N && at < 0; ++i)
        if (PyUnicode_Compare(names[i], key) == 0) at = i;
      if (at < 0 || v[at]) return false;
      v[at] = args[nargs + j];
    }
    return true;
  }
  bool given(int i) const { return v[i] && v[i] != Py_None; }
  // A truth value, `fallback` where the argument is absent. False if the argument has none (a tensor of several
  // elements): the Python function asks it again and raises.
  bool flag(int i, bool fallback, bool& out) const {
    const int t = v[i] ? PyObject_IsTrue(v[i]) : fallback;
    if (t < 0) PyErr_Clear();
    out = t > 0;
    return t >= 0;
  }
};

template <int N>
std::array<PyObject*, N> interned(const std::array<const char*, N>& names) {
  std::array<PyObject*, N> out{};
  for (int i = 0; i < N; ++i) out[i] = PyUnicode_InternFromString(names[i]);
  return out;
}

const at::Tensor* tensor_of(PyObject* o) {
  return o && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}

PyObject* declined() { Py_RETURN_NONE; }

PyObject* failed(int code, const char* what) {
  PyErr_Format(code == WK_E_ARG ? PyExc_ValueError : PyExc_RuntimeError,
               code == WK_E_ARG ? "%s: %s" : "%s: %s (code %d)", what, abi.error_string(code), code);
  return nullptr;
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, const at::Device& dev) {
  return at::Tensor(at::detail::empty_cuda(sizes, dtype, dev, std::nullopt));
}
at::Tensor empty_strided(at::IntArrayRef sizes, at::IntArrayRef strides, at::ScalarType dtype, const at::Device& dev) {
  return at::Tensor(at::detail::empty_strided_cuda(sizes, strides, dtype, dev));
}

bool aligned(const void* p, uintptr_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

// Gives up the GIL for as long as it lives; an exception on the way out takes it back too.
struct GilReleased {
  PyThreadState* state = PyEval_SaveThread();
  ~GilReleased() { PyEval_RestoreThread(state); }
};

// Calls fn(stream) on the current stream of `dev` with that device current and the GIL released.
template <class F>
int on_device(int dev, F fn) {
  const GilReleased gil;
  const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(dev)));
  return fn(static_cast<void*>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream()));
}

// ---- attention --------------------------------------------------------------------------------------------------
// Zeroed scratch for the forward's block flags, one per (device, stream): the kernels hand it back zeroed, so the
// calls that follow one another on a stream share it.  Torch has a fixed number of streams per device, which bounds
// the table; a buffer only ever grows.  Guarded by the GIL.
at::Tensor& block_flags(int dev, void* stream, int64_t nbytes) {
  static auto* table = new std::map<std::pair<int, void*>, at::Tensor>();  // outlives the interpreter's teardown
  at::Tensor& buf = (*table)[{dev, stream}];
  if (!buf.defined() || buf.numel() < nbytes)
    buf = at::zeros({std::max<int64_t>(nbytes, 1 << 16)},
                    at::TensorOptions().dtype(at::kByte).device(at::kCUDA, static_cast<c10::DeviceIndex>(dev)));
  return buf;
}

struct AttnShape {
  int64_t B, Hq, Hkv, Nq, Nk, d;
  bool fp8;
  at::Device dev{at::kCPU};
};

// TMA reads a tensor where it is: last stride 1, the others multiples of 16 elements, 16-byte aligned base.
bool tma_direct(const at::Tensor& t) {
  return t.stride(3) == 1 && t.stride(0) % 16 == 0 && t.stride(1) % 16 == 0 && t.stride(2) % 16 == 0 &&
         aligned(t.data_ptr(), 16);
}

bool attn_shape(const at::Tensor* q, const at::Tensor* k, const at::Tensor* v, AttnShape& s) {
  if (!q || !k || !v || q->dim() != 4 || k->dim() != 4 || v->dim() != 4) return false;
  const at::ScalarType t = q->scalar_type();
  s.fp8 = t == at::kFloat8_e4m3fn;
  if ((!s.fp8 && t != at::kBFloat16) || k->scalar_type() != t || v->scalar_type() != t) return false;
  s.dev = q->device();
  if (!s.dev.is_cuda() || k->device() != s.dev || v->device() != s.dev || !device_ok(s.dev.index())) return false;
  s.B = q->size(0), s.Hq = q->size(1), s.Nq = q->size(2), s.d = q->size(3);
  s.Hkv = k->size(1), s.Nk = k->size(2);
  if (k->sizes() != v->sizes() || k->size(0) != s.B || k->size(3) != s.d || (s.d != 64 && s.d != 128)) return false;
  if (s.B < 1 || s.Hkv < 1 || s.Nq < 1 || s.Nk < 1 || s.Hq % s.Hkv || s.Nq > INT32_MAX / 2 || s.Nk > INT32_MAX / 2)
    return false;
  return tma_direct(*q) && tma_direct(*k) && tma_direct(*v);
}

// A [B, Hkv] contiguous float32 descale on the inputs' device.
bool descale(PyObject* o, const AttnShape& s, const float*& out) {
  const at::Tensor* t = tensor_of(o);
  if (!t || t->dim() != 2 || t->size(0) != s.B || t->size(1) != s.Hkv || t->scalar_type() != at::kFloat ||
      t->device() != s.dev || !t->is_contiguous())
    return false;
  out = t->const_data_ptr<float>();
  return true;
}

bool softmax_scale_of(PyObject* o, int64_t d, float& out) {
  if (!o || o == Py_None) {
    out = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d)));
    return true;
  }
  if (!PyFloat_Check(o) && !PyLong_Check(o)) return false;
  const double x = PyFloat_AsDouble(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  out = static_cast<float>(x);
  return x > 0.0;
}

void put_strides(int64_t (&dst)[3], const at::Tensor& t) {
  for (int i = 0; i < 3; ++i) dst[i] = t.stride(i);
}

PyObject* attn_fwd(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  enum { Q, K, V, QD, KD, VD, CAUSAL, SCALE, STAGES, PIPE, BLOCK_N, BLOCK_M, WARP_ROWS, CTAS, LOCAL, LPT, TMA, OUT,
         LSE, USED, NATURAL, SPEC, SPLIT, COUNT };
  static const auto names = interned<COUNT>(
      {"q", "k", "v", "q_descale", "k_descale", "v_descale", "causal", "softmax_scale", "num_stages", "pipelined",
       "block_n", "block_m", "warp_rows", "ctas_per_sm", "tile_local", "lpt", "tma", "out", "return_lse", "seqused_k",
       "lse_natural", "warp_spec", "split_kv"});
  Params<COUNT> p;
  AttnShape s;
  if (!bound || !p.read(names, args, nargs, kwnames)) return declined();
  const at::Tensor *q = tensor_of(p.v[Q]), *k = tensor_of(p.v[K]), *v = tensor_of(p.v[V]);
  if (!attn_shape(q, k, v, s)) return declined();
  wk_attn_fwd_args a = {};
  if (s.fp8) {
    if (!descale(p.v[QD], s, a.q_descale) || !descale(p.v[KD], s, a.k_descale) || !descale(p.v[VD], s, a.v_descale))
      return declined();
  } else if (p.given(QD) || p.given(KD) || p.given(VD)) {
    return declined();
  }
  if (!softmax_scale_of(p.v[SCALE], s.d, a.softmax_scale)) return declined();
  bool with_lse, causal, natural;
  if (!p.flag(LSE, true, with_lse) || !p.flag(CAUSAL, false, causal) || !p.flag(NATURAL, false, natural))
    return declined();
  if (p.given(CTAS)) {
    const long n = PyLong_Check(p.v[CTAS]) ? PyLong_AsLong(p.v[CTAS]) : 0;
    if (n == -1) PyErr_Clear();  // beyond a long
    if (n != 1 && n != 2) return declined();
    a.ctas_per_sm = static_cast<int32_t>(n);
  }
  if (p.given(USED)) {
    const at::Tensor* used = tensor_of(p.v[USED]);
    if (!used || used->dim() != 1 || used->size(0) != s.B || used->scalar_type() != at::kInt ||
        used->device() != s.dev || !used->is_contiguous())
      return declined();
    a.seqused_k = used->const_data_ptr<int32_t>();
  }
  at::Tensor out;
  if (p.given(OUT)) {
    const at::Tensor* o = tensor_of(p.v[OUT]);
    if (!o || o->dim() != 4 || o->sizes() != q->sizes() || o->scalar_type() != at::kBFloat16 || o->device() != s.dev ||
        o->stride(3) != 1 || o->stride(0) % 8 || o->stride(1) % 8 || o->stride(2) % 8 || !aligned(o->data_ptr(), 16))
      return declined();
    out = *o;
  } else if (q->is_non_overlapping_and_dense()) {
    out = empty_strided(q->sizes(), q->strides(), at::kBFloat16, s.dev);  // the memory layout of q
  } else {
    out = at::empty_like(*q, q->options().dtype(at::kBFloat16));
  }
  a.q = q->data_ptr(), a.k = k->data_ptr(), a.v = v->data_ptr(), a.out = out.data_ptr();
  put_strides(a.q_strides, *q), put_strides(a.k_strides, *k), put_strides(a.v_strides, *v);
  put_strides(a.out_strides, out);
  at::Tensor lse, pmax;
  if (with_lse) {
    const int64_t nq_pad = (s.Nq + 127) / 128 * 128;  // rows of lse and pmax start every nq_pad entries
    const std::array<int64_t, 3> sizes = {s.B, s.Hq, s.Nq}, strides = {s.Hq * nq_pad, nq_pad, 1};
    lse = empty_strided(sizes, strides, at::kFloat, s.dev);
    pmax = empty_strided(sizes, strides, at::kFloat, s.dev);
    a.lse = lse.mutable_data_ptr<float>(), a.pmax = pmax.mutable_data_ptr<float>();
    a.lse_strides[0] = strides[0], a.lse_strides[1] = strides[1];
    a.write_lse = 1;
  }
  a.B = s.B, a.Hq = s.Hq, a.Hkv = s.Hkv, a.Nq = s.Nq, a.Nk = s.Nk, a.d = s.d;
  a.causal = causal, a.lse_natural = natural;
  a.workspace_bytes = abi.attn_fwd_workspace_bytes(a.B, a.Hq, a.Nq);
  void* stream = c10::cuda::getCurrentCUDAStream(s.dev.index()).stream();
  a.workspace = block_flags(s.dev.index(), stream, a.workspace_bytes).data_ptr();
  const int code = on_device(s.dev.index(), [&](void* st) { return (s.fp8 ? abi.attn_fwd_fp8 : abi.attn_fwd_bf16)(&a, st); });
  if (code) return failed(code, "attn_fwd");
  PyObject* o = p.given(OUT) ? Py_NewRef(p.v[OUT]) : THPVariable_Wrap(std::move(out));
  PyObject* l = with_lse ? THPVariable_Wrap(std::move(lse)) : Py_NewRef(Py_None);
  PyObject* m = with_lse ? THPVariable_Wrap(std::move(pmax)) : Py_NewRef(Py_None);
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, o), PyTuple_SET_ITEM(r, 1, l), PyTuple_SET_ITEM(r, 2, m);
  return r;
}

// bf16 with last stride 1: out and dout of the FP8 backward go through 8-byte loads, dout of the BF16 one through TMA.
bool bf16_rows(const at::Tensor* t, const at::Tensor& q, int64_t stride_unit, uintptr_t base_unit) {
  return t && t->dim() == 4 && t->sizes() == q.sizes() && t->scalar_type() == at::kBFloat16 &&
         t->device() == q.device() && t->stride(3) == 1 && t->stride(0) % stride_unit == 0 &&
         t->stride(1) % stride_unit == 0 && t->stride(2) % stride_unit == 0 && aligned(t->data_ptr(), base_unit);
}

PyObject* attn_bwd(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  enum { Q, K, V, OUT, LSE, PMAX, DOUT, QD, KD, VD, CAUSAL, SCALE, STAGES, BULK, INTER, DET, BLOCK_M, MAJOR, USED, ONE,
         COUNT };
  static const auto names = interned<COUNT>(
      {"q", "k", "v", "out", "lse", "pmax", "dout", "q_descale", "k_descale", "v_descale", "causal", "softmax_scale",
       "num_stages", "dq_bulk", "dq_interleave", "deterministic", "block_m", "kb_major", "seqused_k", "one_barrier"});
  Params<COUNT> p;
  AttnShape s;
  if (!bound || !p.read(names, args, nargs, kwnames) || p.given(USED)) return declined();
  const at::Tensor *q = tensor_of(p.v[Q]), *k = tensor_of(p.v[K]), *v = tensor_of(p.v[V]);
  const at::Tensor *out = tensor_of(p.v[OUT]), *dout = tensor_of(p.v[DOUT]);
  const at::Tensor *lse = tensor_of(p.v[LSE]), *pmax = tensor_of(p.v[PMAX]);
  if (!attn_shape(q, k, v, s)) return declined();
  wk_attn_bwd_args a = {};
  if (s.fp8) {
    if (!descale(p.v[QD], s, a.q_descale) || !descale(p.v[KD], s, a.k_descale) || !descale(p.v[VD], s, a.v_descale))
      return declined();
  } else if (p.given(QD) || p.given(KD) || p.given(VD)) {
    return declined();
  }
  if (!bf16_rows(out, *q, 4, 8) || !bf16_rows(dout, *q, s.fp8 ? 4 : 16, s.fp8 ? 8 : 16)) return declined();
  const std::array<int64_t, 3> rows = {s.B, s.Hq, s.Nq};
  if (!lse || !pmax || lse->sizes() != at::IntArrayRef(rows) || pmax->sizes() != at::IntArrayRef(rows) ||
      lse->scalar_type() != at::kFloat || lse->device() != s.dev || lse->stride(2) != 1)
    return declined();
  bool causal;
  if (!softmax_scale_of(p.v[SCALE], s.d, a.softmax_scale) || !p.flag(CAUSAL, false, causal)) return declined();
  at::Tensor dq = empty({s.B, s.Hq, s.Nq, s.d}, at::kBFloat16, s.dev);
  at::Tensor dk = empty({s.B, s.Hkv, s.Nk, s.d}, at::kBFloat16, s.dev);
  at::Tensor dv = empty({s.B, s.Hkv, s.Nk, s.d}, at::kBFloat16, s.dev);
  a.workspace_bytes = (s.fp8 ? abi.attn_bwd_fp8_workspace_bytes : abi.attn_bwd_bf16_workspace_bytes)(s.B, s.Hq, s.Nq);
  at::Tensor workspace = empty({a.workspace_bytes}, at::kByte, s.dev);
  a.q = q->data_ptr(), a.k = k->data_ptr(), a.v = v->data_ptr(), a.out = out->data_ptr(), a.dout = dout->data_ptr();
  a.lse = lse->const_data_ptr<float>();
  a.dq = dq.data_ptr(), a.dk = dk.data_ptr(), a.dv = dv.data_ptr(), a.workspace = workspace.data_ptr();
  put_strides(a.q_strides, *q), put_strides(a.k_strides, *k), put_strides(a.v_strides, *v);
  put_strides(a.out_strides, *out), put_strides(a.dout_strides, *dout);
  a.lse_strides[0] = lse->stride(0), a.lse_strides[1] = lse->stride(1);
  a.B = s.B, a.Hq = s.Hq, a.Hkv = s.Hkv, a.Nq = s.Nq, a.Nk = s.Nk, a.d = s.d;
  a.causal = causal;
  const int code = on_device(s.dev.index(), [&](void* st) { return (s.fp8 ? abi.attn_bwd_fp8 : abi.attn_bwd_bf16)(&a, st); });
  if (code) return failed(code, "attn_bwd");
  PyObject* r = PyTuple_New(3);
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(dq)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(dk)));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(std::move(dv)));
  return r;
}

// ---- GEMM -------------------------------------------------------------------------------------------------------
bool small_int(PyObject* o, long& out) {
  if (!PyLong_CheckExact(o)) return false;  // no bool
  out = PyLong_AsLong(o);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return out >= 1 && out <= (1 << 20);
}

// A float32 scale of one element or of `size` (then contiguous, aligned for the kernels' vector loads).
bool gemm_scale(PyObject* o, int64_t size, const at::Device& dev, uintptr_t unit, const float*& ptr, int32_t& vec) {
  const at::Tensor* t = tensor_of(o);
  if (!t || t->scalar_type() != at::kFloat || t->device() != dev) return false;
  const int64_t n = t->numel();
  if (n != 1 && n != size) return false;
  vec = n > 1 && size > 1;
  if (n > 1 && (!t->is_contiguous() || !aligned(t->data_ptr(), unit))) return false;
  ptr = t->const_data_ptr<float>();
  return true;
}

bool mx_scale(PyObject* o, int64_t rows, int64_t k, const at::Device& dev, const void*& ptr) {
  const at::Tensor* t = tensor_of(o);
  if (!t || t->scalar_type() != at::kByte || t->dim() != 2 || t->size(0) != rows || t->size(1) != k / 32 ||
      t->device() != dev || !t->is_contiguous() || !aligned(t->data_ptr(), 4))
    return false;
  ptr = t->data_ptr();
  return true;
}

PyObject* gemm(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  enum { A, B, OUT, BK, STAGES, GROUP_M, MIN_BLOCKS, BN, FRAG, TMA, SPEC, PERSIST, MAXNREG, SA, SB, OUT_DTYPE, ACT,
         STORE_PRE, PRE, A_TRANS, B_TRANS, ACCUM, SA_MX, OUT_MX, SB_MX, PAIR, COUNT };
  static const auto names = interned<COUNT>(
      {"a", "b", "out", "bk", "stages", "group_m", "min_blocks", "bn", "frag_pipe", "tma", "warp_spec", "persistent",
       "setmaxnreg", "scale_a", "scale_b", "out_dtype", "act", "store_pre", "pre", "a_trans", "b_trans", "accum",
       "a_scale_mx", "out_mx", "b_scale_mx", "cta_pair"});
  Params<COUNT> p;
  if (!bound || !p.read(names, args, nargs, kwnames)) return declined();
  const at::Tensor *a = tensor_of(p.v[A]), *b = tensor_of(p.v[B]);
  if (!a || !b || a->dim() != 2 || b->dim() != 2) return declined();
  const at::ScalarType dt = a->scalar_type();
  const bool fp8 = dt == at::kFloat8_e4m3fn;
  if ((!fp8 && dt != at::kBFloat16 && dt != at::kHalf) || b->scalar_type() != dt) return declined();
  const at::Device dev = a->device();
  if (!dev.is_cuda() || b->device() != dev || !device_ok(dev.index())) return declined();
  if (!a->is_contiguous() || !b->is_contiguous() || !aligned(a->data_ptr(), 16) || !aligned(b->data_ptr(), 16))
    return declined();
  bool a_trans, b_trans, store_pre, accum, out_mx, pair;
  if (!p.flag(A_TRANS, false, a_trans) || !p.flag(B_TRANS, false, b_trans) || !p.flag(STORE_PRE, false, store_pre) ||
      !p.flag(ACCUM, false, accum) || !p.flag(OUT_MX, false, out_mx) || !p.flag(PAIR, false, pair))
    return declined();
  const int64_t m = a->size(a_trans ? 1 : 0), k = a->size(a_trans ? 0 : 1);
  const int64_t n = b->size(b_trans ? 1 : 0), kb = b->size(b_trans ? 0 : 1);
  if (kb != k || ((a_trans || b_trans) && fp8) || m < 1 || n < 1 || k < 1) return declined();
  if (m > INT32_MAX / 2 || n > INT32_MAX / 2 || k > INT32_MAX / 2) return declined();
  long bk = fp8 ? 128 : 64, bn = 128, group_m = 0;
  if (p.given(BK) && !small_int(p.v[BK], bk)) return declined();
  if (p.v[BN] && (!small_int(p.v[BN], bn) || (bn != 128 && bn != 256))) return declined();
  if (p.given(GROUP_M) && !small_int(p.v[GROUP_M], group_m)) return declined();
  if (m % 128 || n % bn || k % bk || k % (fp8 ? 128 : 64)) return declined();
  int act = 0;
  if (p.v[ACT]) {
    if (!PyUnicode_Check(p.v[ACT])) return declined();
    if (PyUnicode_CompareWithASCIIString(p.v[ACT], "gelu") == 0)
      act = 1;
    else if (PyUnicode_CompareWithASCIIString(p.v[ACT], "dgelu") == 0)
      act = 2;
    else if (PyUnicode_GET_LENGTH(p.v[ACT]) != 0)
      return declined();
  }
  if ((store_pre && act != 1) || (accum && !p.given(OUT))) return declined();
  at::ScalarType odt = dt;
  at::Tensor out;
  if (p.given(OUT)) {
    const at::Tensor* o = tensor_of(p.v[OUT]);
    if (!o || o->dim() != 2 || o->size(0) != m || o->size(1) != n || !o->is_contiguous() || o->device() != dev ||
        !aligned(o->data_ptr(), 16))
      return declined();
    odt = o->scalar_type();
    out = *o;
  } else if (fp8) {
    odt = at::kBFloat16;
    if (p.v[OUT_DTYPE]) {
      if (!THPDtype_Check(p.v[OUT_DTYPE])) return declined();
      odt = reinterpret_cast<THPDtype*>(p.v[OUT_DTYPE])->scalar_type;
    }
  }
  if ((odt != at::kBFloat16 && odt != at::kHalf) || (!fp8 && odt != dt)) return declined();
  const float *scale_a = nullptr, *scale_b = nullptr;
  int32_t row_scale = 0, col_scale = 0;
  if (p.given(SA) && !gemm_scale(p.v[SA], m, dev, 8, scale_a, row_scale)) return declined();
  if (p.given(SB) && !gemm_scale(p.v[SB], n, dev, 16, scale_b, col_scale)) return declined();
  if (!fp8) {  // one-element scales apply to fp8 inputs only
    if (!row_scale) scale_a = nullptr;
    if (!col_scale) scale_b = nullptr;
  }
  const void *sa_mx = nullptr, *sb_mx = nullptr, *pre_in = nullptr;
  if ((p.given(SA_MX) || p.given(SB_MX)) && !fp8) return declined();
  if (p.given(SA_MX) && !mx_scale(p.v[SA_MX], m, k, dev, sa_mx)) return declined();
  if (p.given(SB_MX) && !mx_scale(p.v[SB_MX], n, k, dev, sb_mx)) return declined();
  if (act == 2) {
    const at::Tensor* pre = tensor_of(p.v[PRE]);
    if (!pre || pre->dim() != 2 || pre->size(0) != m || pre->size(1) != n || pre->scalar_type() != odt ||
        pre->device() != dev || !pre->is_contiguous() || !aligned(pre->data_ptr(), 16))
      return declined();
    pre_in = pre->data_ptr();
  }
  int cta_pair = 0;
  if (p.given(PAIR)) cta_pair = pair ? 1 : 2;

  if (!out.defined()) out = empty({m, n}, odt, dev);
  at::Tensor pre_out, q_mx, s_mx, workspace;
  if (store_pre) pre_out = empty({m, n}, odt, dev);
  if (out_mx) {
    q_mx = empty({m, n}, at::kFloat8_e4m3fn, dev);
    s_mx = empty({m, n / 32}, at::kByte, dev);
  }
  auto fill = [&](auto& g) {
    g.a = a->data_ptr(), g.b = b->data_ptr(), g.out = out.data_ptr();
    g.m = m, g.n = n, g.k = k;
    g.scale_a = scale_a, g.scale_b = scale_b, g.scale_a_rows = row_scale, g.scale_b_cols = col_scale;
    g.accum = accum, g.act = act;
    g.pre_out = store_pre ? pre_out.data_ptr() : nullptr, g.pre_in = pre_in;
    g.q_mx = out_mx ? q_mx.data_ptr() : nullptr, g.s_mx = out_mx ? s_mx.data_ptr() : nullptr;
    g.cta_pair = cta_pair, g.group_m = static_cast<int32_t>(group_m);
  };
  int code;
  if (fp8) {
    wk_gemm_mx_args g = {};
    fill(g);
    g.a_scale_mx = sa_mx, g.b_scale_mx = sb_mx;
    g.out_f16 = odt == at::kHalf;
    g.workspace_bytes = abi.gemm_mxfp8_workspace_bytes(g.m, g.n, g.k);
    workspace = empty({g.workspace_bytes}, at::kByte, dev);
    g.workspace = workspace.data_ptr();
    code = on_device(dev.index(), [&](void* st) { return abi.gemm_mxfp8(&g, st); });
  } else {
    wk_gemm16_args g = {};
    fill(g);
    g.f16 = dt == at::kHalf, g.a_trans = a_trans, g.b_trans = b_trans;
    code = on_device(dev.index(), [&](void* st) { return abi.gemm_16bit(&g, st); });
  }
  if (code) return failed(code, fp8 ? "gemm (fp8)" : "gemm (16-bit)");
  PyObject* o = p.given(OUT) ? Py_NewRef(p.v[OUT]) : THPVariable_Wrap(std::move(out));
  if (act != 1 && !out_mx) return o;
  PyObject* r = PyTuple_New(1 + (act == 1) + 2 * out_mx);
  Py_ssize_t at = 0;
  PyTuple_SET_ITEM(r, at++, o);
  if (act == 1) PyTuple_SET_ITEM(r, at++, store_pre ? THPVariable_Wrap(std::move(pre_out)) : Py_NewRef(Py_None));
  if (out_mx) {
    PyTuple_SET_ITEM(r, at++, THPVariable_Wrap(std::move(q_mx)));
    PyTuple_SET_ITEM(r, at++, THPVariable_Wrap(std::move(s_mx)));
  }
  return r;
}

PyObject* quantize_mx(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  enum { X, Q, S, COUNT };
  static const auto names = interned<COUNT>({"x", "q", "s"});
  Params<COUNT> p;
  if (!bound || !p.read(names, args, nargs, kwnames)) return declined();
  const at::Tensor* x = tensor_of(p.v[X]);
  if (!x || x->dim() != 2 || (x->scalar_type() != at::kBFloat16 && x->scalar_type() != at::kFloat)) return declined();
  const at::Device dev = x->device();
  const int64_t m = x->size(0), k = x->size(1);
  if (!dev.is_cuda() || !device_ok(dev.index()) || m < 1 || k < 32 || k % 32 || x->stride(1) != 1 ||
      (m > 1 && x->stride(0) % 8))
    return declined();
  at::Tensor q, s;
  if (p.given(Q)) {
    const at::Tensor* t = tensor_of(p.v[Q]);
    if (!t || t->sizes() != x->sizes() || t->scalar_type() != at::kFloat8_e4m3fn || !t->is_contiguous() ||
        t->device() != dev)
      return declined();
    q = *t;
  }
  if (p.given(S)) {
    const at::Tensor* t = tensor_of(p.v[S]);
    if (!t || t->dim() != 2 || t->size(0) != m || t->size(1) != k / 32 || t->scalar_type() != at::kByte ||
        !t->is_contiguous() || t->device() != dev)
      return declined();
    s = *t;
  }
  if (!q.defined()) q = empty({m, k}, at::kFloat8_e4m3fn, dev);
  if (!s.defined()) s = empty({m, k / 32}, at::kByte, dev);
  const int dtype = x->scalar_type() == at::kBFloat16 ? WK_BF16 : WK_F32;
  const int64_t ld = m > 1 ? x->stride(0) : std::max<int64_t>(k, 8);
  const int code = on_device(dev.index(), [&](void* st) {
    return abi.quantize_mx(x->data_ptr(), dtype, m, k, ld, q.data_ptr(), s.data_ptr(), st);
  });
  if (code) return failed(code, "quantize_mx");
  PyObject* r = PyTuple_New(2);
  PyTuple_SET_ITEM(r, 0, p.given(Q) ? Py_NewRef(p.v[Q]) : THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(r, 1, p.given(S) ? Py_NewRef(p.v[S]) : THPVariable_Wrap(std::move(s)));
  return r;
}

// ---- prepared launches --------------------------------------------------------------------------------------------
// launch(entry, args, device) -> code: calls the C ABI function at address `entry` with the argument block at address
// `args` on the current stream of the device.
PyObject* launch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "launch(entry, args, device)");
    return nullptr;
  }
  void* entry = PyLong_AsVoidPtr(args[0]);
  void* block = PyLong_AsVoidPtr(args[1]);
  const long dev = PyLong_AsLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromLong(on_device(static_cast<int>(dev), [&](void* st) {
    return reinterpret_cast<int (*)(const void*, void*)>(entry)(block, st);
  }));
}

// block_flags(device, nbytes) -> tensor: the forward's flag scratch of the device's current stream.
PyObject* py_block_flags(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "block_flags(device, nbytes)");
    return nullptr;
  }
  const long dev = PyLong_AsLong(args[0]);
  const long long nbytes = PyLong_AsLongLong(args[1]);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(
      block_flags(static_cast<int>(dev), c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream(), nbytes));
}

// bind({name: address}): the C ABI functions of the loaded library.
PyObject* bind(PyObject*, PyObject* table) {
  if (!PyDict_Check(table)) {
    PyErr_SetString(PyExc_TypeError, "bind() takes a dict of addresses");
    return nullptr;
  }
  for (const auto& sym : kSymbols) {
    PyObject* o = PyDict_GetItemString(table, sym.name);
    void* ptr = o ? PyLong_AsVoidPtr(o) : nullptr;
    if (!ptr) {
      if (!PyErr_Occurred()) PyErr_Format(PyExc_KeyError, "%s is missing", sym.name);
      return nullptr;
    }
    *sym.slot = ptr;
  }
  bound = true;
  Py_RETURN_NONE;
}

// A C++ exception (an allocation that failed, a CUDA error) becomes the Python exception torch raises for it.
template <class F>
PyObject* guard(F call) {
  try {
    return call();
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    PyErr_Clear();
    PyErr_SetString(type ? type : PyExc_MemoryError, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t, PyObject*)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return guard([&] { return F(self, args, nargs, kwnames); });
}
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded_plain(PyObject* self, PyObject* const* args, Py_ssize_t nargs) {
  return guard([&] { return F(self, args, nargs); });
}

template <auto F>
PyCFunction as_method() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F));
}

PyMethodDef methods[] = {
    {"attn_fwd", as_method<guarded<attn_fwd>>(), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"attn_bwd", as_method<guarded<attn_bwd>>(), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"gemm", as_method<guarded<gemm>>(), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"quantize_mx", as_method<guarded<quantize_mx>>(), METH_FASTCALL | METH_KEYWORDS, nullptr},
    {"launch", as_method<guarded_plain<launch>>(), METH_FASTCALL, nullptr},
    {"block_flags", as_method<guarded_plain<py_block_flags>>(), METH_FASTCALL, nullptr},
    {"bind", bind, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
