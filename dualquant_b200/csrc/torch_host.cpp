// Native half of the tensor-level wrappers (ops.py) and of PermLinear.forward: takes torch tensors,
// checks them, allocates results and calls the C ABI.
//
// Why it exists: a decode-size call is two kernels of a few microseconds, and the same sequence spelled
// in Python (attribute look-ups, ctypes conversions, torch.empty through the dispatcher) kept the host
// busy for 28-43 us per call while the GPU needed 9-20 - the GPU waited for the host in every linear of
// a small batch.  Here a PermLinear call takes 8.2 to 8.6 us of the host, two launches, a tensor map, output and
// scratch included; that still bounds the smallest one (one token, 4096 -> 4096 with the Hadamard across heads: 8.4 us
// called in a loop, 7.2 replayed from a graph).
//
// Loaded by _lib.py after torch; compiled by g++ against torch's headers.  The C ABI is not linked: its
// functions are looked up in the library that _lib.py has opened (same file, so one copy of its state).
// Every function runs under the GIL and launches on torch's current stream of the tensors' device.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/add.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include <algorithm>
#include <string>

#include "../../include/dualquant_b200.h"

namespace {

// ------------------------------------------------------------------------------------ the C ABI
#define DQ_FUNCTIONS(X)                                                                              \
  X(dq_quant_act_int4) X(dq_quant_act_int4_f32) X(dq_quant_act_int4_gated) X(dq_quant_act_int4_rmsnorm) \
  X(dq_gemm_w4a4_int4_ex) X(dq_gemm_w4a4_int4_residual) X(dq_gemm_w4a4_int4_e4m3)                      \
  X(dq_linear_w4a4_int4) X(dq_linear_w4a4_int4_bias) X(dq_linear_w4a4_int4_scratch_bytes)             \
  X(dq_linear_w4a4_int4_prefill_scratch_bytes) X(dq_linear_a16w4) X(dq_linear_a16w4_scratch_bytes)     \
  X(dq_linear_w4a4_fp4) X(dq_linear_w4a4_fp4_scratch_bytes)
#define DQ_DECLARE(name) decltype(&::name) name = nullptr;
struct Abi {
  DQ_FUNCTIONS(DQ_DECLARE)
} abi;
#undef DQ_DECLARE

PyObject* g_check = nullptr;        // _lib.check(rc, what): raises for a non-zero status
PyObject* g_ensure_init = nullptr;  // _lib.ensure_init(index)
uint64_t g_inited = 0;              // devices ensure_init has been called for

// attribute names, interned once
#define DQ_NAMES(X)                                                                                   \
  X(kind) X(had_k) X(had_dim) X(scale) X(had_mat) X(w_packed) X(sw_t) X(N) X(K) X(group) X(codes)       \
  X(sf_atoms) X(tensor_scale) X(fmt) X(_plan) X(act_quant_enabled) X(online_full_had)                  \
  X(online_partial_had) X(had_K) X(act_fmt) X(quantize_bmm_input) X(dtype) X(_buffers) X(act_scale)    \
  X(_modules) X(layer) X(_parameters) X(bias) X(_packed) X(_packed_fp4) X(name) X(block_size)
#define DQ_DECLARE(n) PyObject* n = nullptr;
struct Names {
  DQ_NAMES(DQ_DECLARE)
} names;
#undef DQ_DECLARE

// Thrown once a Python exception has been set.
struct PyError {};
[[noreturn]] void fail(PyObject* type, const char* msg) {
  PyErr_SetString(type, msg);
  throw PyError();
}

// owned reference
struct Ref {
  PyObject* p = nullptr;
  explicit Ref(PyObject* o) : p(o) {
    if (o == nullptr) throw PyError();
  }
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
};

void check(int rc, const char* what) {
  if (rc == DQ_OK) return;
  PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
  Py_XDECREF(r);
  if (PyErr_Occurred() == nullptr) PyErr_SetString(PyExc_RuntimeError, what);
  throw PyError();
}

const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor", what);
    throw PyError();
  }
  return THPVariable_Unpack(o);
}
const void* ptr_or_null(PyObject* o, const char* what) {
  return o == Py_None ? nullptr : tensor(o, what).data_ptr();
}

// Makes the tensor's device current and the library ready on it; returns the device index.
int prep(const at::Tensor& t) {
  if (!t.is_cuda()) fail(PyExc_RuntimeError, "dualquant_b200 runs on CUDA (sm_100a) tensors only; got a CPU tensor");
  const int idx = t.get_device();
  if (c10::cuda::current_device() != idx) c10::cuda::set_device(static_cast<c10::DeviceIndex>(idx));
  if (idx > 63 || ((g_inited >> idx) & 1u) == 0) {
    Ref r(PyObject_CallFunction(g_ensure_init, "i", idx));
    if (idx <= 63) g_inited |= 1ull << idx;
  }
  return idx;
}
void* stream_of(int idx) {
  return static_cast<void*>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(idx)).stream());
}
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, int idx) {
  return at::detail::empty_cuda(sizes, dtype, at::Device(at::kCUDA, static_cast<c10::DeviceIndex>(idx)), std::nullopt);
}

// Scratch of one call, from torch's allocator for the current stream: calls of one module on several streams, and graphs
// captured through it, keep theirs apart.
struct Scratch {
  c10::DataPtr mem;
  size_t bytes = 0;
  Scratch() = default;
  explicit Scratch(int64_t n)
      : mem(c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(n))), bytes(static_cast<size_t>(n)) {}
};

long as_long(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyError();
  return v;
}
long attr_long(PyObject* o, PyObject* name) {
  Ref r(PyObject_GetAttr(o, name));
  return as_long(r.p);
}
const void* attr_ptr(PyObject* o, PyObject* name, int* device = nullptr) {
  Ref r(PyObject_GetAttr(o, name));
  if (device != nullptr) *device = static_cast<int>(tensor(r.p, "packed weight field").get_device());
  return ptr_or_null(r.p, "packed weight field");
}

// ops.Hadamard -> the ABI's description (kind 0: none)
dq_hadamard_desc hadamard(PyObject* o) {
  dq_hadamard_desc d = {};
  if (o == Py_None) return d;
  d.kind = static_cast<int32_t>(attr_long(o, names.kind));
  if (d.kind == DQ_HAD_NONE) return d;
  d.had_k = static_cast<int32_t>(attr_long(o, names.had_k));
  d.had_dim = static_cast<int32_t>(attr_long(o, names.had_dim));
  Ref s(PyObject_GetAttr(o, names.scale));
  d.scale = static_cast<float>(PyFloat_AsDouble(s.p));
  if (PyErr_Occurred()) throw PyError();
  d.had_mat = static_cast<const float*>(attr_ptr(o, names.had_mat));
  return d;
}
const dq_hadamard_desc* desc(const dq_hadamard_desc& d) { return d.kind == DQ_HAD_NONE ? nullptr : &d; }

// ops.PackedInt4Weight
struct PackedInt4 {
  const uint8_t* w_packed;
  const void* sw_t;
  int N, K, group, device;
};
PackedInt4 packed_int4(PyObject* o) {
  PackedInt4 w;
  w.w_packed = static_cast<const uint8_t*>(attr_ptr(o, names.w_packed, &w.device));
  w.sw_t = attr_ptr(o, names.sw_t);
  w.N = static_cast<int>(attr_long(o, names.N));
  w.K = static_cast<int>(attr_long(o, names.K));
  w.group = static_cast<int>(attr_long(o, names.group));
  return w;
}

// ops.PackedFp4Weight
struct PackedFp4 {
  const uint8_t *codes, *sf_atoms;
  const float* tensor_scale;
  int N, K, fmt, device;
};
PackedFp4 packed_fp4(PyObject* o) {
  PackedFp4 w;
  w.codes = static_cast<const uint8_t*>(attr_ptr(o, names.codes, &w.device));
  w.sf_atoms = static_cast<const uint8_t*>(attr_ptr(o, names.sf_atoms));
  w.tensor_scale = static_cast<const float*>(attr_ptr(o, names.tensor_scale));
  w.N = static_cast<int>(attr_long(o, names.N));
  w.K = static_cast<int>(attr_long(o, names.K));
  w.fmt = static_cast<int>(attr_long(o, names.fmt));
  return w;
}

int y_dtype_of(const at::Tensor& out) { return out.scalar_type() == at::kBFloat16 ? DQ_DTYPE_BF16 : DQ_DTYPE_F32; }
at::ScalarType dtype_arg(PyObject* o) {
  if (!THPDtype_Check(o)) fail(PyExc_TypeError, "out_dtype must be a torch.dtype");
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

// rows with unit inner stride, as the kernels read them (a copy is made only where that does not hold)
at::Tensor unit_rows(const at::Tensor& x) { return x.stride(-1) == 1 ? x : x.contiguous(); }
void need_2d(const at::Tensor& x) {
  if (x.dim() != 2) fail(PyExc_ValueError, "expected a 2-D tensor of token rows");
}
int64_t row_stride(const at::Tensor& x) { return x.size(0) > 1 ? x.stride(0) : x.size(1); }

PyObject* wrap(at::Tensor t) {
  PyObject* o = THPVariable_Wrap(std::move(t));
  if (o == nullptr) throw PyError();
  return o;
}
PyObject* pair(at::Tensor a, at::Tensor b) {
  Ref x(wrap(std::move(a))), y(wrap(std::move(b)));
  return PyTuple_Pack(2, x.p, y.p);
}

// Runs a wrapper body: C++ exceptions become Python exceptions.
template <typename F>
PyObject* guarded(F&& body) {
  try {
    return body();
  } catch (const PyError&) {
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}
#define DQ_ARGS(count, name)                                                             \
  if (n != (count)) {                                                                    \
    PyErr_Format(PyExc_TypeError, name " takes %d arguments, got %zd", (count), n);      \
    return nullptr;                                                                      \
  }

// ------------------------------------------------------------------------------------ wrappers of ops.py
// (argument meaning and checks: the Python functions of the same names)

// quant_act_int4(x, a, had, scale_mode, e4m3) -> (codes, sx)
PyObject* quant_act_int4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(5, "quant_act_int4");
  return guarded([&]() {
    const at::Tensor& xin = tensor(v[0], "x");
    const int idx = prep(xin);
    const bool bf16 = xin.scalar_type() == at::kBFloat16;
    if (!bf16 && xin.scalar_type() != at::kFloat)
      fail(PyExc_ValueError, "quant_act_int4 expects bf16 or fp32 activations");
    need_2d(xin);
    const at::Tensor x = unit_rows(xin);
    const int M = static_cast<int>(x.size(0)), K = static_cast<int>(x.size(1));
    const bool e4m3 = v[4] == Py_True;
    const int mode = static_cast<int>(as_long(v[3])) | (e4m3 ? DQ_CODES_E4M3 : 0);
    const dq_hadamard_desc d = hadamard(v[2]);
    const float* a = static_cast<const float*>(ptr_or_null(v[1], "a"));
    at::Tensor codes = empty({M, K}, e4m3 ? at::kByte : at::kChar, idx), sx = empty({M}, at::kFloat, idx);
    int8_t* cp = static_cast<int8_t*>(codes.data_ptr());
    float* sp = static_cast<float*>(sx.data_ptr());
    if (bf16)
      check(abi.dq_quant_act_int4(x.data_ptr(), row_stride(x), a, desc(d), M, K, cp, sp, mode, stream_of(idx)),
            "dq_quant_act_int4");
    else
      check(abi.dq_quant_act_int4_f32(static_cast<const float*>(x.data_ptr()), row_stride(x), a, desc(d), M, K, cp, sp,
                                      mode, stream_of(idx)),
            "dq_quant_act_int4_f32");
    return pair(std::move(codes), std::move(sx));
  });
}

// quant_act_int4_gated(gate, up, a, had, scale_mode, e4m3) -> (codes, sx)
PyObject* quant_act_int4_gated(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(6, "quant_act_int4_gated");
  return guarded([&]() {
    const at::Tensor &gate = tensor(v[0], "gate"), &up = tensor(v[1], "up");
    const int idx = prep(gate);
    if (gate.scalar_type() != at::kBFloat16 || up.scalar_type() != at::kBFloat16)
      fail(PyExc_ValueError, "quant_act_int4_gated expects bf16 inputs");
    need_2d(gate);
    if (gate.sizes() != up.sizes() || gate.strides() != up.strides() || gate.stride(-1) != 1)
      fail(PyExc_ValueError, "gate and up must have the same shape and strides (unit inner stride)");
    const int M = static_cast<int>(gate.size(0)), K = static_cast<int>(gate.size(1));
    const bool e4m3 = v[5] == Py_True;
    const int mode = static_cast<int>(as_long(v[4])) | (e4m3 ? DQ_CODES_E4M3 : 0);
    const dq_hadamard_desc d = hadamard(v[3]);
    at::Tensor codes = empty({M, K}, e4m3 ? at::kByte : at::kChar, idx), sx = empty({M}, at::kFloat, idx);
    check(abi.dq_quant_act_int4_gated(gate.data_ptr(), up.data_ptr(), row_stride(gate),
                                      static_cast<const float*>(ptr_or_null(v[2], "a")), desc(d), M, K,
                                      static_cast<int8_t*>(codes.data_ptr()), static_cast<float*>(sx.data_ptr()), mode,
                                      stream_of(idx)),
          "dq_quant_act_int4_gated");
    return pair(std::move(codes), std::move(sx));
  });
}

// quant_act_int4_rmsnorm(x, norm_weight, eps, a, scale_mode, e4m3) -> (codes, sx)
PyObject* quant_act_int4_rmsnorm(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(6, "quant_act_int4_rmsnorm");
  return guarded([&]() {
    const at::Tensor& x = tensor(v[0], "x");
    const int idx = prep(x);
    if (x.scalar_type() != at::kBFloat16 || x.stride(-1) != 1)
      fail(PyExc_ValueError, "quant_act_int4_rmsnorm expects bf16 rows with unit inner stride");
    need_2d(x);
    const int M = static_cast<int>(x.size(0)), K = static_cast<int>(x.size(1));
    const void* w = nullptr;
    if (v[1] != Py_None) {
      const at::Tensor& nw = tensor(v[1], "norm_weight");
      if (nw.scalar_type() != at::kBFloat16 || nw.numel() != K)
        fail(PyExc_ValueError, "norm_weight must be bf16 with one entry per input channel");
      w = nw.data_ptr();
    }
    const double eps = PyFloat_AsDouble(v[2]);
    if (PyErr_Occurred()) throw PyError();
    const bool e4m3 = v[5] == Py_True;
    const int mode = static_cast<int>(as_long(v[4])) | (e4m3 ? DQ_CODES_E4M3 : 0);
    at::Tensor codes = empty({M, K}, e4m3 ? at::kByte : at::kChar, idx), sx = empty({M}, at::kFloat, idx);
    check(abi.dq_quant_act_int4_rmsnorm(x.data_ptr(), row_stride(x), w, static_cast<float>(eps),
                                        static_cast<const float*>(ptr_or_null(v[3], "a")), M, K,
                                        static_cast<int8_t*>(codes.data_ptr()), static_cast<float*>(sx.data_ptr()), mode,
                                        stream_of(idx)),
          "dq_quant_act_int4_rmsnorm");
    return pair(std::move(codes), std::move(sx));
  });
}

// the output tensor of a linear: the caller's, or a new one of the residual's / the asked-for type
at::Tensor output(PyObject* out, PyObject* residual, PyObject* out_dtype, int64_t M, int64_t N, int idx) {
  if (out != Py_None) return tensor(out, "out");
  const at::ScalarType t = residual != Py_None ? tensor(residual, "residual").scalar_type() : dtype_arg(out_dtype);
  return empty({M, N}, t, idx);
}
const void* residual_ptr(PyObject* residual, const at::Tensor& out, int64_t M, int64_t N) {
  if (residual == Py_None) return nullptr;
  const at::Tensor& r = tensor(residual, "residual");
  if (r.scalar_type() != out.scalar_type() || r.dim() != 2 || r.size(0) != M || r.size(1) != N || !r.is_contiguous())
    fail(PyExc_ValueError, "residual must be a contiguous [M, N] tensor of the output's dtype");
  return r.data_ptr();
}

// gemm_w4a4_int4(codes, sx, pw, r, out_dtype, token_tile, split_k, out, residual) -> out
PyObject* gemm_w4a4_int4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(9, "gemm_w4a4_int4");
  return guarded([&]() {
    const at::Tensor &codes = tensor(v[0], "codes"), &sx = tensor(v[1], "sx");
    const int idx = prep(codes);
    need_2d(codes);
    const PackedInt4 w = packed_int4(v[2]);
    const int M = static_cast<int>(codes.size(0)), K = static_cast<int>(codes.size(1));
    if (K != w.K) {
      PyErr_Format(PyExc_ValueError, "K mismatch: activations %d, weight %d", K, w.K);
      throw PyError();
    }
    const float* r = static_cast<const float*>(ptr_or_null(v[3], "r"));
    at::Tensor out = output(v[7], v[8], v[4], M, w.N, idx);
    const void* res = residual_ptr(v[8], out, M, w.N);
    const int8_t* cp = static_cast<const int8_t*>(codes.data_ptr());
    const float* sp = static_cast<const float*>(sx.data_ptr());
    if (res != nullptr)
      check(abi.dq_gemm_w4a4_int4_residual(cp, sp, w.w_packed, w.sw_t, r, res, M, w.N, K, w.group, out.data_ptr(),
                                           y_dtype_of(out), stream_of(idx)),
            "dq_gemm_w4a4_int4_residual");
    else
      check(abi.dq_gemm_w4a4_int4_ex(cp, sp, w.w_packed, w.sw_t, r, M, w.N, K, w.group, out.data_ptr(), y_dtype_of(out),
                                     nullptr, 0, stream_of(idx), static_cast<int>(as_long(v[5])),
                                     static_cast<int>(as_long(v[6]))),
            "dq_gemm_w4a4_int4");
    return wrap(std::move(out));
  });
}

// gemm_w4a4_int4_e4m3(x8, sx, w8, pw, r, out_dtype, out, residual) -> out
PyObject* gemm_w4a4_int4_e4m3(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(8, "gemm_w4a4_int4_e4m3");
  return guarded([&]() {
    const at::Tensor &x8 = tensor(v[0], "x8"), &sx = tensor(v[1], "sx"), &w8 = tensor(v[2], "w8");
    const int idx = prep(x8);
    need_2d(x8);
    const PackedInt4 w = packed_int4(v[3]);
    const int M = static_cast<int>(x8.size(0)), K = static_cast<int>(x8.size(1));
    if (K != w.K || w8.dim() != 2 || w8.size(0) != w.N || w8.size(1) != w.K || !x8.is_contiguous() || !w8.is_contiguous())
      fail(PyExc_ValueError, "x8 [M, K] and w8 [N, K] must be contiguous and match the packed weight");
    at::Tensor out = output(v[6], v[7], v[5], M, w.N, idx);
    const void* res = residual_ptr(v[7], out, M, w.N);
    check(abi.dq_gemm_w4a4_int4_e4m3(static_cast<const uint8_t*>(x8.data_ptr()), static_cast<const float*>(sx.data_ptr()),
                                     static_cast<const uint8_t*>(w8.data_ptr()), w.sw_t,
                                     static_cast<const float*>(ptr_or_null(v[4], "r")), M, w.N, K, w.group, out.data_ptr(),
                                     y_dtype_of(out), res, stream_of(idx)),
          "dq_gemm_w4a4_int4_e4m3");
    return wrap(std::move(out));
  });
}

// Scratch of linear_int4: for prefill batches with room for the weight's byte form, which every call expands anew.  (Kept
// with the packed weight it would save 5 to 18 us a call, but nothing tells when those bytes are written again, or
// whether another stream's expansion has finished.  A caller who knows keeps it: ops.PackedInt4Weight.bytes_e4m3.)
int64_t int4_scratch_bytes(int M, int N, int K) {
  return std::max<int64_t>(static_cast<int64_t>(abi.dq_linear_w4a4_int4_prefill_scratch_bytes(M, N, K)), 256);
}
// Activation quantiser + GEMM of one linear.
void linear_int4(const void* x, int64_t ldx, const float* a, const dq_hadamard_desc* had, const PackedInt4& w,
                 const float* r, const void* bias, int M, const at::Tensor& out, int mode, void* scratch, size_t bytes,
                 int idx) {
  void* stream = stream_of(idx);
  if (bias == nullptr)
    check(abi.dq_linear_w4a4_int4(x, ldx, a, had, w.w_packed, w.sw_t, r, M, w.N, w.K, w.group, out.data_ptr(),
                                  y_dtype_of(out), mode, scratch, bytes, stream),
          "dq_linear_w4a4_int4");
  else
    check(abi.dq_linear_w4a4_int4_bias(x, ldx, a, had, w.w_packed, nullptr, w.sw_t, r, bias, M, w.N, w.K, w.group,
                                       out.data_ptr(), y_dtype_of(out), mode, scratch, bytes, stream),
          "dq_linear_w4a4_int4_bias");
}

// linear_w4a4_int4(x, a, had, pw, r, out_dtype, scale_mode, scratch, out) -> out
PyObject* linear_w4a4_int4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(9, "linear_w4a4_int4");
  return guarded([&]() {
    const at::Tensor& xin = tensor(v[0], "x");
    const int idx = prep(xin);
    if (xin.scalar_type() != at::kBFloat16)
      fail(PyExc_ValueError, "linear_w4a4_int4 expects bf16 activations (quantise fp32 rows with "
                             "quant_act_int4 and call gemm_w4a4_int4)");
    need_2d(xin);
    const at::Tensor x = unit_rows(xin);
    const PackedInt4 w = packed_int4(v[3]);
    const int M = static_cast<int>(x.size(0)), K = static_cast<int>(x.size(1));
    if (K != w.K) {
      PyErr_Format(PyExc_ValueError, "K mismatch: activations %d, weight %d", K, w.K);
      throw PyError();
    }
    // a caller's scratch is used as it is when it covers the plain path; the library takes the FP8-path GEMM for
    // prefill batches only where it also has room for the weight's byte form
    Scratch own;
    void* scratch = nullptr;
    size_t bytes = 0;
    if (v[7] != Py_None && tensor(v[7], "scratch").numel() >=
                               static_cast<int64_t>(abi.dq_linear_w4a4_int4_scratch_bytes(M, w.N, K))) {
      scratch = tensor(v[7], "scratch").data_ptr();
      bytes = static_cast<size_t>(tensor(v[7], "scratch").numel());
    } else {
      own = Scratch(int4_scratch_bytes(M, w.N, K));
      scratch = own.mem.get();
      bytes = own.bytes;
    }
    at::Tensor out = output(v[8], Py_None, v[5], M, w.N, idx);
    const dq_hadamard_desc d = hadamard(v[2]);
    linear_int4(x.data_ptr(), row_stride(x), static_cast<const float*>(ptr_or_null(v[1], "a")), desc(d), w,
                static_cast<const float*>(ptr_or_null(v[4], "r")), nullptr, M, out, static_cast<int>(as_long(v[6])),
                scratch, bytes, idx);
    return wrap(std::move(out));
  });
}

// linear_a16w4(x, a, pw, r, out_dtype, scratch, out) -> out
PyObject* linear_a16w4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(7, "linear_a16w4");
  return guarded([&]() {
    const at::Tensor& xin = tensor(v[0], "x");
    const int idx = prep(xin);
    if (xin.scalar_type() != at::kBFloat16) fail(PyExc_ValueError, "linear_a16w4 expects bf16 activations");
    need_2d(xin);
    const at::Tensor x = unit_rows(xin);
    const PackedInt4 w = packed_int4(v[2]);
    const int M = static_cast<int>(x.size(0)), K = static_cast<int>(x.size(1));
    if (K != w.K) {
      PyErr_Format(PyExc_ValueError, "K mismatch: activations %d, weight %d", K, w.K);
      throw PyError();
    }
    const int64_t need = static_cast<int64_t>(abi.dq_linear_a16w4_scratch_bytes(M, w.N, K));
    at::Tensor scratch = (v[5] != Py_None && tensor(v[5], "scratch").numel() >= need)
                             ? tensor(v[5], "scratch")
                             : empty({std::max<int64_t>(need, 256)}, at::kByte, idx);
    at::Tensor out = output(v[6], Py_None, v[4], M, w.N, idx);
    check(abi.dq_linear_a16w4(x.data_ptr(), row_stride(x), static_cast<const float*>(ptr_or_null(v[1], "a")), w.w_packed,
                              static_cast<const float*>(ptr_or_null(v[3], "r")), M, w.N, K, w.group, out.data_ptr(),
                              y_dtype_of(out), scratch.data_ptr(), static_cast<size_t>(scratch.numel()), stream_of(idx)),
          "dq_linear_a16w4");
    return wrap(std::move(out));
  });
}

int64_t fp4_scratch_bytes(int M, int K, int fmt) {
  return std::max<int64_t>(static_cast<int64_t>(abi.dq_linear_w4a4_fp4_scratch_bytes(M, K, fmt)), 256);
}
void linear_fp4(const void* x, bool f32, int64_t ldx, int M, const float* a, const PackedFp4& w, const float* r,
                const void* bias, const at::Tensor& out, const Scratch& scratch, int idx) {
  check(abi.dq_linear_w4a4_fp4(x, f32 ? 1 : 0, ldx, a, w.codes, w.sf_atoms, w.tensor_scale, r, bias, M, w.N, w.K, w.fmt,
                               out.data_ptr(), y_dtype_of(out), scratch.mem.get(), scratch.bytes, stream_of(idx)),
        "dq_linear_w4a4_fp4");
}

// linear_w4a4_fp4(x, a, pw, r, out_dtype) -> out
PyObject* linear_w4a4_fp4(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(5, "linear_w4a4_fp4");
  return guarded([&]() {
    const at::Tensor& xin = tensor(v[0], "x");
    const int idx = prep(xin);
    const bool f32 = xin.scalar_type() == at::kFloat;
    if (!f32 && xin.scalar_type() != at::kBFloat16) fail(PyExc_ValueError, "quant_fp4 expects bf16 or fp32");
    need_2d(xin);
    const at::Tensor x = xin.contiguous();
    const PackedFp4 w = packed_fp4(v[2]);
    const int M = static_cast<int>(x.size(0));
    if (x.size(1) != w.K) {
      PyErr_Format(PyExc_ValueError, "K mismatch: activations %d, weight %d", static_cast<int>(x.size(1)), w.K);
      throw PyError();
    }
    const Scratch scratch(fp4_scratch_bytes(M, w.K, w.fmt));
    at::Tensor out = empty({M, w.N}, dtype_arg(v[4]), idx);
    linear_fp4(x.data_ptr(), f32, w.K, M, static_cast<const float*>(ptr_or_null(v[1], "a")), w,
               static_cast<const float*>(ptr_or_null(v[3], "r")), nullptr, out, scratch, idx);
    return wrap(std::move(out));
  });
}

// ------------------------------------------------------------------------------------ PermLinear.forward
// A Plan is what PermLinear._make_plan found out about a module: which of the packed paths its forward takes
// and the objects of that path.  perm_forward uses it as long as nothing it was derived from has been
// replaced since - it compares the objects themselves - and answers None otherwise; the Python forward then
// does the work and makes a new plan.  No pointer and no value of a tensor is kept: the packed weight's fields,
// act_scale, bias and the Hadamard factor are read by every call.
enum PlanKind { PLAN_INT4 = 0, PLAN_FP4 = 1, PLAN_A16 = 2 };

struct Plan {
  PyObject_HEAD
  int kind, scale_mode;
  PyObject *act_quant_enabled, *online_full_had, *online_partial_had, *had_K, *K, *had_dim, *act_fmt, *quantize_bmm_input,
      *dtype, *act_scale, *layer, *packed;  // owned; compared by identity
  PyObject *fmt_name, *fmt_block;           // owned: act_fmt's, which may be changed in place
  PyObject* had_mat;                        // owned: the device copy of the factor (None: no factor)
  dq_hadamard_desc had;                     // had_mat is filled in by each call
  at::ScalarType out_dtype;
};

#define DQ_PLAN_OBJECTS(X)                                                                                      \
  X(act_quant_enabled) X(online_full_had) X(online_partial_had) X(had_K) X(K) X(had_dim) X(act_fmt)              \
  X(quantize_bmm_input) X(dtype)

int plan_traverse(PyObject* self, visitproc visit, void* arg) {
  Plan* p = reinterpret_cast<Plan*>(self);
#define DQ_VISIT(f) Py_VISIT(p->f);
  DQ_PLAN_OBJECTS(DQ_VISIT) DQ_VISIT(act_scale) DQ_VISIT(layer) DQ_VISIT(packed) DQ_VISIT(had_mat)
  DQ_VISIT(fmt_name) DQ_VISIT(fmt_block)
#undef DQ_VISIT
  return 0;
}
int plan_clear(PyObject* self) {
  Plan* p = reinterpret_cast<Plan*>(self);
#define DQ_CLEAR(f) Py_CLEAR(p->f);
  DQ_PLAN_OBJECTS(DQ_CLEAR) DQ_CLEAR(act_scale) DQ_CLEAR(layer) DQ_CLEAR(packed) DQ_CLEAR(had_mat)
  DQ_CLEAR(fmt_name) DQ_CLEAR(fmt_block)
#undef DQ_CLEAR
  return 0;
}
void plan_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  plan_clear(self);
  Py_TYPE(self)->tp_free(self);
}
// copies and pickles of a module carry no plan: they make their own
PyObject* plan_reduce(PyObject*, PyObject*) {
  return Py_BuildValue("(O())", reinterpret_cast<PyObject*>(Py_TYPE(Py_None)));
}
PyMethodDef plan_methods[] = {{"__reduce__", plan_reduce, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyTypeObject plan_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// the module's attributes that live in its own __dict__ (borrowed references)
struct ModuleDict {
  PyObject* d;
  explicit ModuleDict(PyObject* self) : d(PyObject_GenericGetDict(self, nullptr)) {
    if (d == nullptr) throw PyError();
  }
  ModuleDict(const ModuleDict&) = delete;
  ~ModuleDict() { Py_DECREF(d); }
  PyObject* get(PyObject* name) const { return PyDict_GetItemWithError(d, name); }
  PyObject* in(PyObject* table, PyObject* name) const {  // self.<table>[name]
    PyObject* t = get(table);
    return (t != nullptr && PyDict_Check(t)) ? PyDict_GetItemWithError(t, name) : nullptr;
  }
};

// make_plan(module, kind, hadamard or None, scale_mode, out_dtype) -> Plan
PyObject* make_plan(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(5, "make_plan");
  return guarded([&]() {
    const ModuleDict m(v[0]);
    Ref obj(plan_type.tp_alloc(&plan_type, 0));
    Plan* p = reinterpret_cast<Plan*>(obj.p);
    p->kind = static_cast<int>(as_long(v[1]));
    p->scale_mode = static_cast<int>(as_long(v[3]));
    p->out_dtype = dtype_arg(v[4]);
    p->had = hadamard(v[2]);
    auto keep = [](PyObject* o) {
      if (o == nullptr) fail(PyExc_AttributeError, "incomplete PermLinear");
      Py_INCREF(o);
      return o;
    };
#define DQ_KEEP(f) p->f = keep(m.get(names.f));
    DQ_PLAN_OBJECTS(DQ_KEEP)
#undef DQ_KEEP
    p->fmt_name = Py_NewRef(Ref(PyObject_GetAttr(p->act_fmt, names.name)).p);
    p->fmt_block = Py_NewRef(Ref(PyObject_GetAttr(p->act_fmt, names.block_size)).p);
    p->act_scale = keep(m.in(names._buffers, names.act_scale));
    p->layer = keep(m.in(names._modules, names.layer));
    p->packed = keep(m.get(p->kind == PLAN_FP4 ? names._packed_fp4 : names._packed));
    if (p->had.had_mat != nullptr) {
      p->had.had_mat = nullptr;
      p->had_mat = PyObject_GetAttr(v[2], names.had_mat);
      if (p->had_mat == nullptr) throw PyError();
    } else {
      Py_INCREF(Py_None);
      p->had_mat = Py_None;
    }
    Py_INCREF(obj.p);
    return obj.p;
  });
}

// perm_forward(module, x) -> output tensor, or None when the Python forward has to take the call
PyObject* perm_forward(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(2, "perm_forward");
  return guarded([&]() -> PyObject* {
    if (!THPVariable_Check(v[1])) Py_RETURN_NONE;
    const ModuleDict m(v[0]);
    PyObject* po = m.get(names._plan);
    if (po == nullptr || Py_TYPE(po) != &plan_type) Py_RETURN_NONE;
    const Ref hold(Py_NewRef(po));  // another thread may replace the module's plan meanwhile
    Plan* p = reinterpret_cast<Plan*>(po);
#define DQ_SAME(f) if (m.get(names.f) != p->f) Py_RETURN_NONE;
    DQ_PLAN_OBJECTS(DQ_SAME)
#undef DQ_SAME
    if (Ref(PyObject_GetAttr(p->act_fmt, names.name)).p != p->fmt_name ||
        Ref(PyObject_GetAttr(p->act_fmt, names.block_size)).p != p->fmt_block)
      Py_RETURN_NONE;
    if (m.in(names._buffers, names.act_scale) != p->act_scale || m.in(names._modules, names.layer) != p->layer ||
        m.get(p->kind == PLAN_FP4 ? names._packed_fp4 : names._packed) != p->packed)
      Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(v[1]);
    PackedInt4 w4 = {};
    PackedFp4 w_fp4 = {};
    if (p->kind == PLAN_FP4) w_fp4 = packed_fp4(p->packed);
    else w4 = packed_int4(p->packed);
    const int K = p->kind == PLAN_FP4 ? w_fp4.K : w4.K, N = p->kind == PLAN_FP4 ? w_fp4.N : w4.N;
    const int device = p->kind == PLAN_FP4 ? w_fp4.device : w4.device;
    if (!x.is_cuda() || x.get_device() != device || x.scalar_type() != at::kBFloat16 || x.dim() < 1 ||
        x.size(-1) != K || x.numel() == 0)
      Py_RETURN_NONE;
    int64_t ldx = K;
    if (!x.is_contiguous()) {  // token rows with gaps between them; anything else is left to the Python forward
      if (x.dim() != 2 || x.stride(1) != 1 || p->kind == PLAN_FP4) Py_RETURN_NONE;
      ldx = row_stride(x);
    }
    const float* a = nullptr;
    if (p->act_scale != Py_None) {
      const at::Tensor& s = tensor(p->act_scale, "act_scale");
      if (!s.is_cuda() || s.get_device() != device) Py_RETURN_NONE;
      a = static_cast<const float*>(s.data_ptr());
    }
    const ModuleDict layer(p->layer);
    PyObject* bias = layer.in(names._parameters, names.bias);
    if (bias == nullptr) Py_RETURN_NONE;
    const int idx = prep(x);
    const int M = static_cast<int>(x.numel() / K);
    int64_t need;
    if (p->kind == PLAN_INT4) need = int4_scratch_bytes(M, N, K);
    else if (p->kind == PLAN_FP4) need = fp4_scratch_bytes(M, K, w_fp4.fmt);
    else need = static_cast<int64_t>(abi.dq_linear_a16w4_scratch_bytes(M, N, K));
    const Scratch scratch(std::max<int64_t>(need, 256));
    c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
    sizes.back() = N;
    at::Tensor out = empty(sizes, p->out_dtype, idx);
    // a bias of the output's type and width is added in the GEMM's epilogue, any other (or one that wants a gradient)
    // by torch, which broadcasts it or says what is wrong with it
    const void* bias_ptr = nullptr;
    if (p->kind != PLAN_A16 && bias != Py_None) {
      const at::Tensor& b = tensor(bias, "bias");
      if (b.scalar_type() == p->out_dtype && b.dim() == 1 && b.size(0) == N && b.is_contiguous() && b.is_cuda() &&
          b.get_device() == device && !(b.requires_grad() && at::GradMode::is_enabled())) {
        bias_ptr = b.data_ptr();
        bias = Py_None;
      }
    }
    if (p->kind == PLAN_INT4) {
      dq_hadamard_desc had = p->had;
      had.had_mat = static_cast<const float*>(ptr_or_null(p->had_mat, "had_mat"));
      linear_int4(x.data_ptr(), ldx, a, desc(had), w4, nullptr, bias_ptr, M, out, p->scale_mode,
                  scratch.mem.get(), scratch.bytes, idx);
    } else if (p->kind == PLAN_FP4) {
      linear_fp4(x.data_ptr(), false, K, M, a, w_fp4, nullptr, bias_ptr, out, scratch, idx);
    } else {
      check(abi.dq_linear_a16w4(x.data_ptr(), ldx, a, w4.w_packed, nullptr, M, N, K, w4.group, out.data_ptr(),
                                y_dtype_of(out), scratch.mem.get(), scratch.bytes, stream_of(idx)),
            "dq_linear_a16w4");
    }
    if (bias != Py_None) return wrap(at::add(out, tensor(bias, "bias")));
    return wrap(std::move(out));
  });
}

// ------------------------------------------------------------------------------------ module
// setup(library path, check, ensure_init)
PyObject* setup(PyObject*, PyObject* const* v, Py_ssize_t n) {
  DQ_ARGS(3, "setup");
  return guarded([&]() -> PyObject* {
    const char* path = PyUnicode_AsUTF8(v[0]);
    if (path == nullptr) throw PyError();
    void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
    if (lib == nullptr) fail(PyExc_RuntimeError, dlerror());
#define DQ_LOOKUP(name)                                                             \
  abi.name = reinterpret_cast<decltype(abi.name)>(dlsym(lib, #name));               \
  if (abi.name == nullptr) fail(PyExc_RuntimeError, #name " is missing from the library");
    DQ_FUNCTIONS(DQ_LOOKUP)
#undef DQ_LOOKUP
    Py_INCREF(v[1]);
    Py_XSETREF(g_check, v[1]);
    Py_INCREF(v[2]);
    Py_XSETREF(g_ensure_init, v[2]);
    Py_RETURN_NONE;
  });
}

#define DQ_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {DQ_METHOD(setup),
                         DQ_METHOD(quant_act_int4),
                         DQ_METHOD(quant_act_int4_gated),
                         DQ_METHOD(quant_act_int4_rmsnorm),
                         DQ_METHOD(gemm_w4a4_int4),
                         DQ_METHOD(gemm_w4a4_int4_e4m3),
                         DQ_METHOD(linear_w4a4_int4),
                         DQ_METHOD(linear_a16w4),
                         DQ_METHOD(linear_w4a4_fp4),
                         DQ_METHOD(make_plan),
                         DQ_METHOD(perm_forward),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_host", "native half of ops.py", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__torch_host() {
#define DQ_INTERN(n)                               \
  names.n = PyUnicode_InternFromString(#n);        \
  if (names.n == nullptr) return nullptr;
  DQ_NAMES(DQ_INTERN)
#undef DQ_INTERN
  plan_type.tp_name = "dualquant_b200._torch_host.Plan";
  plan_type.tp_basicsize = sizeof(Plan);
  plan_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  plan_type.tp_traverse = plan_traverse;
  plan_type.tp_clear = plan_clear;
  plan_type.tp_dealloc = plan_dealloc;
  plan_type.tp_methods = plan_methods;
  if (PyType_Ready(&plan_type) < 0) return nullptr;
  return PyModule_Create(&module);
}
