// Host path of the torch-facing entry points as one CPython extension module (`sglang_b200._host`).
//
// A decode-sized layer takes the GPU about ten microseconds.  Through Python-level allocation, checks and ctypes
// marshalling its two or three launches cost the host fifty, which is what a caller waited for.  Each function here
// does the checks, takes one workspace and the outputs from torch's caching allocator and calls the C ABI
// (include/sglang_b200.h), so a layer costs the host about as much as its launches.
//
// A function returns None when its arguments are not the plain case it serves (CPU tensors, non-contiguous inputs,
// other types): the caller then takes the Python form, which names the rejected argument.  The C ABI is bound by
// path, so the module runs on the same build of the library as the ctypes binding.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/sglang_b200.h"

namespace {

// ---- the C ABI ------------------------------------------------------------------------------------------------
#define SGLB_HOST_FUNCTIONS(X)           \
  X(sglb200_last_error)                  \
  X(sglb200_per_token_group_quant_fp8)   \
  X(sglb200_silu_and_mul_quant_fp8)      \
  X(sglb200_gemm_workspace_bytes)        \
  X(sglb200_fp8_blockwise_scaled_mm)     \
  X(sglb200_block_fp8_linear_workspace_bytes) \
  X(sglb200_block_fp8_linear)            \
  X(sglb200_fused_experts_workspace_bytes) \
  X(sglb200_fused_experts)               \
  X(sglb200_topk_softmax)                \
  X(sglb200_moe_fused_gate)

struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  SGLB_HOST_FUNCTIONS(X)
#undef X
} abi;

PyObject* bind(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (path == nullptr) return nullptr;
  void* h = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (h == nullptr) {
    PyErr_SetString(PyExc_ImportError, dlerror());
    return nullptr;
  }
#define X(name)                                                                                        \
  abi.name = reinterpret_cast<decltype(&::name)>(dlsym(h, #name));                                     \
  if (abi.name == nullptr) {                                                                           \
    PyErr_SetString(PyExc_ImportError, "libsglang_b200 is older than its header: " #name " is missing"); \
    return nullptr;                                                                                    \
  }
  SGLB_HOST_FUNCTIONS(X)
#undef X
  Py_RETURN_NONE;
}

// A rejected call becomes the exception the reference op would raise.
PyObject* raise_last(int rc) {
  PyErr_SetString(rc == SGLB200_E_UNSUPPORTED ? PyExc_NotImplementedError : PyExc_RuntimeError, abi.sglb200_last_error());
  return nullptr;
}

// C++ exceptions of the allocator (out of memory) must not cross into the interpreter.
template <class F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
  }
  return nullptr;
}

// Truth as Python sees it (True, 1, numpy's bool); a failing __bool__ leaves its error for the caller's PyErr_Occurred.
bool flag(PyObject* o) { return PyObject_IsTrue(o) == 1; }

// ---- tensors --------------------------------------------------------------------------------------------------
using at::Tensor;

// The tensor behind a Python argument if it is a contiguous CUDA tensor, else nullptr.
const Tensor* cuda_contig(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.is_contiguous() ? &t : nullptr;
}

int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? 0 : t == at::kHalf ? 1 : t == at::kFloat ? 2 : -1;
}

Tensor make(at::IntArrayRef size, at::ScalarType dtype, c10::Device dev) {
  return at::detail::empty_cuda(size, dtype, dev, std::nullopt);
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

Tensor workspace(int64_t bytes, c10::Device dev) { return make({bytes > 0 ? bytes : 1}, at::kByte, dev); }

PyObject* pair(Tensor a, Tensor b) {
  PyObject* x = THPVariable_Wrap(std::move(a));
  PyObject* y = THPVariable_Wrap(std::move(b));
  PyObject* r = x && y ? PyTuple_Pack(2, x, y) : nullptr;
  Py_XDECREF(x);
  Py_XDECREF(y);
  return r;
}

constexpr float kFp8Max = 448.0f;

// ---- quantizer ------------------------------------------------------------------------------------------------
// quant(x, group_size, eps, column_major, tma_aligned) -> (codes, scales)
PyObject* quant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 5) Py_RETURN_NONE;
  const Tensor* xp = cuda_contig(args[0]);
  const int64_t group = PyLong_AsLongLong(args[1]);
  const double eps = PyFloat_AsDouble(args[2]);
  const bool colmajor = flag(args[3]), tma = flag(args[4]);
  if (PyErr_Occurred()) return nullptr;
  if (xp == nullptr || xp->dim() < 1 || (colmajor && xp->dim() != 2)) Py_RETURN_NONE;
  const Tensor& x = *xp;
  const int dt = dtype_code(x.scalar_type());
  const int64_t hidden = x.size(-1);
  if (dt < 0 || hidden <= 0 || group <= 0 || hidden % group != 0 || x.numel() == 0) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int64_t tokens = x.numel() / hidden, groups = hidden / group;
    Tensor q = make(x.sizes(), at::kFloat8_e4m3fn, x.device()), s;
    int64_t st = groups, sg = 1;
    if (colmajor) {
      const int64_t pad = tma ? (tokens + 3) / 4 * 4 : tokens;
      s = make({groups, pad}, at::kFloat, x.device()).as_strided({tokens, groups}, {1, pad});
      st = 1, sg = pad;
    } else {
      c10::DimVector shape(x.sizes().begin(), x.sizes().end());
      shape.back() = groups;
      s = make(shape, at::kFloat, x.device());
    }
    const int rc = abi.sglb200_per_token_group_quant_fp8(x.data_ptr(), dt, q.data_ptr(), static_cast<float*>(s.data_ptr()), tokens,
                                                         hidden, (int)group, (float)eps, -kFp8Max, kFp8Max, st, sg, stream_of(x));
    if (rc) return raise_last(rc);
    return pair(std::move(q), std::move(s));
  });
}

// silu_mul_quant(x [.., 2d], group_size, eps, num_rows | None) -> (codes [.., d], scales [.., d / group])
PyObject* silu_mul_quant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4) Py_RETURN_NONE;
  const Tensor* xp = cuda_contig(args[0]);
  const int64_t group = PyLong_AsLongLong(args[1]);
  const double eps = PyFloat_AsDouble(args[2]);
  if (PyErr_Occurred()) return nullptr;
  const Tensor* nr = nullptr;
  if (args[3] != Py_None && (nr = cuda_contig(args[3])) == nullptr) Py_RETURN_NONE;
  if (xp == nullptr || xp->dim() < 1) Py_RETURN_NONE;
  const Tensor& x = *xp;
  const int dt = dtype_code(x.scalar_type());
  const int64_t d = x.size(-1) / 2;
  if (dt < 0 || dt > 1 || d <= 0 || x.size(-1) % 2 || group <= 0 || d % group != 0 || x.numel() == 0) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    c10::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = d;
    Tensor q = make(shape, at::kFloat8_e4m3fn, x.device());
    shape.back() = d / group;
    Tensor s = make(shape, at::kFloat, x.device());
    const int rc = abi.sglb200_silu_and_mul_quant_fp8(x.data_ptr(), dt, q.data_ptr(), static_cast<float*>(s.data_ptr()),
                                                      x.numel() / (2 * d), d, (int)group, (float)eps,
                                                      nr ? static_cast<const int32_t*>(nr->data_ptr()) : nullptr, stream_of(x));
    if (rc) return raise_last(rc);
    return pair(std::move(q), std::move(s));
  });
}

// ---- dense layers ---------------------------------------------------------------------------------------------
// Weight [N, K] e4m3 with scales [ceil(N/128), ceil(K/128)] float32, or nullptr when it is anything else.
bool weight_ok(const Tensor* w, const Tensor* ws) {
  return w && ws && w->dim() == 2 && ws->dim() == 2 && w->scalar_type() == at::kFloat8_e4m3fn &&
         ws->scalar_type() == at::kFloat && ws->size(0) == (w->size(0) + 127) / 128 && ws->size(1) == (w->size(1) + 127) / 128;
}

// bias: absent, or one contiguous CUDA tensor of N values in the output type
bool bias_ok(PyObject* o, int64_t n, at::ScalarType out, const Tensor** bias) {
  *bias = nullptr;
  if (o == Py_None) return true;
  *bias = cuda_contig(o);
  return *bias != nullptr && (*bias)->numel() == n && (*bias)->scalar_type() == out;
}

// linear(x [.., K] 16-bit, weight, weight_scale, bias | None) -> [.., N] in x's type: quantise, multiply
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4) Py_RETURN_NONE;
  const Tensor *xp = cuda_contig(args[0]), *w = cuda_contig(args[1]), *ws = cuda_contig(args[2]), *bias;
  if (xp == nullptr || xp->dim() < 1 || !weight_ok(w, ws)) Py_RETURN_NONE;
  const Tensor& x = *xp;
  const int dt = dtype_code(x.scalar_type());
  const int64_t K = x.size(-1), N = w->size(0);
  if (dt < 0 || dt > 1 || K <= 0 || K % 128 != 0 || w->size(1) != K || x.numel() == 0 || x.device() != w->device() ||
      !bias_ok(args[3], N, x.scalar_type(), &bias))
    Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int64_t M = x.numel() / K;
    const int64_t bytes = abi.sglb200_block_fp8_linear_workspace_bytes(M, N, K);
    c10::DimVector shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    Tensor out = make(shape, x.scalar_type(), x.device()), mem;
    if (bytes) mem = workspace(bytes, x.device());
    const int rc = abi.sglb200_block_fp8_linear(x.data_ptr(), dt, w->data_ptr(), static_cast<const float*>(ws->data_ptr()), out.data_ptr(),
                                                bias ? bias->data_ptr() : nullptr, M, N, K, bytes ? mem.data_ptr() : nullptr, bytes, stream_of(x));
    if (rc) return raise_last(rc);
    return THPVariable_Wrap(std::move(out));
  });
}

// matmul(A [.., K] e4m3, weight, As [.., K/128] (contiguous, or 2-D with any strides), weight_scale, out_dtype, bias | None)
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 6) Py_RETURN_NONE;
  const Tensor *ap = cuda_contig(args[0]), *w = cuda_contig(args[1]), *ws = cuda_contig(args[3]), *bias;
  if (ap == nullptr || ap->dim() < 1 || !weight_ok(w, ws) || !THPVariable_Check(args[2]) || !THPDtype_Check(args[4]))
    Py_RETURN_NONE;
  const Tensor& a = *ap;
  const Tensor& as = THPVariable_Unpack(args[2]);
  const at::ScalarType out_t = reinterpret_cast<THPDtype*>(args[4])->scalar_type;
  const int dt = dtype_code(out_t);
  const int64_t K = a.size(-1), N = w->size(0);
  if (dt < 0 || dt > 1 || a.scalar_type() != at::kFloat8_e4m3fn || K <= 0 || w->size(1) != K || a.numel() == 0 ||
      a.device() != w->device() || !bias_ok(args[5], N, out_t, &bias) || !as.is_cuda() || as.scalar_type() != at::kFloat)
    Py_RETURN_NONE;
  const int64_t M = a.numel() / K, kb = (K + 127) / 128;
  int64_t sm = kb, sk = 1;
  if (as.is_contiguous()) {
    if (as.numel() != M * kb) Py_RETURN_NONE;
  } else {
    if (as.dim() != 2 || as.size(0) != M || as.size(1) != kb) Py_RETURN_NONE;
    sm = as.stride(0), sk = as.stride(1);
  }
  return guarded([&]() -> PyObject* {
    const int64_t scratch = abi.sglb200_gemm_workspace_bytes(M, N, K);
    c10::DimVector shape(a.sizes().begin(), a.sizes().end());
    shape.back() = N;
    Tensor out = make(shape, out_t, a.device()), mem;
    if (scratch) mem = workspace(scratch, a.device());
    const int rc = abi.sglb200_fp8_blockwise_scaled_mm(
        a.data_ptr(), w->data_ptr(), static_cast<const float*>(as.data_ptr()), static_cast<const float*>(ws->data_ptr()), out.data_ptr(),
        bias ? bias->data_ptr() : nullptr, M, N, K, sm, sk, dt, scratch ? mem.data_ptr() : nullptr, scratch, stream_of(a));
    if (rc) return raise_last(rc);
    return THPVariable_Wrap(std::move(out));
  });
}

// ---- routing --------------------------------------------------------------------------------------------------
// topk_softmax(logits [T, E], k, renormalize) -> (weights, ids)
PyObject* topk_softmax(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3) Py_RETURN_NONE;
  const Tensor* g = cuda_contig(args[0]);
  const int64_t k = PyLong_AsLongLong(args[1]);
  const bool renormalize = flag(args[2]);
  if (PyErr_Occurred()) return nullptr;
  if (g == nullptr || g->dim() != 2 || k < 1) Py_RETURN_NONE;
  const int dt = dtype_code(g->scalar_type());
  if (dt < 0) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    Tensor w = make({g->size(0), k}, at::kFloat, g->device()), ids = make({g->size(0), k}, at::kInt, g->device());
    const int rc = abi.sglb200_topk_softmax(g->data_ptr(), dt, g->size(0), (int)g->size(1), (int)k, renormalize, 0.f, nullptr,
                                            static_cast<float*>(w.data_ptr()), static_cast<int32_t*>(ids.data_ptr()), stream_of(*g));
    if (rc) return raise_last(rc);
    return pair(std::move(w), std::move(ids));
  });
}

// fused_gate(logits [T, E], bias [E], groups, topk_group, topk, shared, factor, scale_output) -> (weights, ids)
PyObject* fused_gate(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 8) Py_RETURN_NONE;
  const Tensor *g = cuda_contig(args[0]), *b = cuda_contig(args[1]);
  const int64_t groups = PyLong_AsLongLong(args[2]), kept = PyLong_AsLongLong(args[3]), k = PyLong_AsLongLong(args[4]),
                shared = PyLong_AsLongLong(args[5]);
  const double factor = PyFloat_AsDouble(args[6]);
  const bool scale_output = flag(args[7]);
  if (PyErr_Occurred()) return nullptr;
  if (g == nullptr || b == nullptr || g->dim() != 2 || b->numel() != g->size(1) || b->scalar_type() != g->scalar_type() || k < 1)
    Py_RETURN_NONE;
  const int dt = dtype_code(g->scalar_type());
  if (dt < 0) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    Tensor w = make({g->size(0), k}, at::kFloat, g->device()), ids = make({g->size(0), k}, at::kInt, g->device());
    const int rc = abi.sglb200_moe_fused_gate(g->data_ptr(), b->data_ptr(), dt, g->size(0), (int)g->size(1), (int)groups, (int)kept,
                                              (int)k, (int)shared, (float)factor, scale_output,
                                              static_cast<float*>(w.data_ptr()), static_cast<int32_t*>(ids.data_ptr()), stream_of(*g));
    if (rc) return raise_last(rc);
    return pair(std::move(w), std::move(ids));
  });
}

// ---- routed experts -------------------------------------------------------------------------------------------
bool experts_ok(const Tensor* w, const Tensor* s) {
  return w && s && w->dim() == 3 && s->dim() == 3 && w->scalar_type() == at::kFloat8_e4m3fn && s->scalar_type() == at::kFloat &&
         s->size(0) == w->size(0) && s->size(1) == (w->size(1) + 127) / 128 && s->size(2) == (w->size(2) + 127) / 128;
}

// fused_experts(x [T, H] 16-bit, w13, w13_scale, w2, w2_scale, weights [T, k] f32, ids [T, k] i32, factor, out [T, H])
//   -> True: x through the experts that `ids` names, weighted, summed over k, times factor, into out
PyObject* fused_experts(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 9) Py_RETURN_NONE;
  const Tensor *xp = cuda_contig(args[0]), *w1 = cuda_contig(args[1]), *s1 = cuda_contig(args[2]), *w2 = cuda_contig(args[3]),
               *s2 = cuda_contig(args[4]), *wt = cuda_contig(args[5]), *id = cuda_contig(args[6]), *out = cuda_contig(args[8]);
  const double factor = PyFloat_AsDouble(args[7]);
  if (PyErr_Occurred()) return nullptr;
  if (!xp || !wt || !id || !out || !experts_ok(w1, s1) || !experts_ok(w2, s2)) Py_RETURN_NONE;
  const Tensor& x = *xp;
  const int dt = dtype_code(x.scalar_type());
  if (dt < 0 || dt > 1 || x.dim() != 2 || id->dim() != 2 || id->scalar_type() != at::kInt || wt->scalar_type() != at::kFloat ||
      wt->sizes() != id->sizes() || id->size(0) != x.size(0) || out->scalar_type() != x.scalar_type() || x.device() != w1->device())
    Py_RETURN_NONE;
  const int64_t T = x.size(0), H = x.size(1), E = w1->size(0), N = w1->size(1), I = N / 2, Ho = w2->size(1), k = id->size(1);
  if (T == 0 || k == 0 || w1->size(2) != H || H % 128 != 0 || w2->size(0) != E || w2->size(2) != I || N % 2 || I % 128 != 0 ||
      out->numel() != T * Ho)
    Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    const int64_t bytes = abi.sglb200_fused_experts_workspace_bytes(T, k, (int)E, H, I, Ho, (float)factor);
    Tensor mem = workspace(bytes, x.device());
    const int rc = abi.sglb200_fused_experts(
        x.data_ptr(), dt, w1->data_ptr(), static_cast<const float*>(s1->data_ptr()), w2->data_ptr(), static_cast<const float*>(s2->data_ptr()),
        static_cast<const float*>(wt->data_ptr()), static_cast<const int32_t*>(id->data_ptr()), out->data_ptr(), T, k, (int)E, H, I, Ho,
        (float)factor, mem.data_ptr(), bytes, stream_of(x));
    if (rc) return raise_last(rc);
    Py_RETURN_TRUE;
  });
}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, "Bind the C ABI of the library at this path."},
#define M(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
    M(quant), M(silu_mul_quant), M(linear), M(matmul), M(topk_softmax), M(fused_gate), M(fused_experts),
#undef M
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
