// Native form of the calls in capi.py that a token loop makes.
//
// A decode-sized GEMM runs 5-12 us on the GPU; through ctypes a call cost the host 10-12 us, so every small call was
// bound by the host: about 1.5 us for the device context, 1 us for the stream, 0.4 us per tensor, and 2 us for the
// conversion of ten arguments, beside 3 us in the library.  The functions here take the same Python arguments and
// return True when they made the call.  They return False, having done nothing, for anything that is not the plain
// case (a tensor subclass, another dtype, a strided or host tensor, an argument that is no int, ...): capi.py then
// takes its general path, which raises the errors or converts the argument.
#include <torch/csrc/autograd/python_variable.h>

#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <climits>

#include "../../include/llmmm_c.h"

namespace {

// Thrown by the conversions below: not the plain case.
struct NotPlain {};

// Device pointer of a plain, contiguous CUDA tensor; DT = Undefined: any dtype.
template<c10::ScalarType DT>
void* pointer(PyObject* o)
{
  if (!THPVariable_CheckExact(o)) {
    throw NotPlain{};
  }
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || !t.is_contiguous() || (DT != c10::ScalarType::Undefined && t.scalar_type() != DT)) {
    throw NotPlain{};
  }
  return t.mutable_data_ptr();
}

void* bytes(PyObject* o) { return pointer<c10::ScalarType::Undefined>(o); }
float* f32(PyObject* o) { return static_cast<float*>(pointer<c10::ScalarType::Float>(o)); }
float* f32_or_null(PyObject* o) { return o == Py_None ? nullptr : f32(o); }
int* i32(PyObject* o) { return static_cast<int*>(pointer<c10::ScalarType::Int>(o)); }

int integer(PyObject* o)
{
  if (!PyLong_CheckExact(o)) {
    throw NotPlain{};
  }
  int        overflow = 0;
  const long v        = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow != 0 || v < INT_MIN || v > INT_MAX) {
    throw NotPlain{};
  }
  return (int)v;
}

float real(PyObject* o)
{
  if (!PyFloat_CheckExact(o)) {
    throw NotPlain{};
  }
  return (float)PyFloat_AS_DOUBLE(o);
}

// capi._stream: None (the current stream of the device), an object with a `cuda_stream`, or an integer handle.
llmmm_stream_t stream_handle(PyObject* o, c10::DeviceIndex device)
{
  if (o == Py_None) {
    return reinterpret_cast<llmmm_stream_t>(c10::cuda::getCurrentCUDAStream(device).stream());
  }
  PyObject* h = PyLong_CheckExact(o) ? Py_NewRef(o) : PyObject_GetAttrString(o, "cuda_stream");
  void*     p = h != nullptr && PyLong_CheckExact(h) ? PyLong_AsVoidPtr(h) : nullptr;
  const bool plain = h != nullptr && PyLong_CheckExact(h) && !PyErr_Occurred();
  Py_XDECREF(h);
  if (!plain) {
    PyErr_Clear();
    throw NotPlain{};
  }
  return static_cast<llmmm_stream_t>(p);
}

// Makes the call `fn(stream)` on the device of `first`, without the interpreter lock, and turns its status into True
// or RuntimeError as capi._check does.
template<class F>
PyObject* call_on(PyObject* first, PyObject* stream, F&& fn)
{
  const c10::Device          device = THPVariable_Unpack(first).device();
  const c10::cuda::CUDAGuard guard(device);
  const llmmm_stream_t       s = stream_handle(stream, device.index());
  int                        status;
  Py_BEGIN_ALLOW_THREADS;
  status = fn(s);
  Py_END_ALLOW_THREADS;
  if (status != 0) {
    PyErr_Format(PyExc_RuntimeError, "llmmm status %d: %s", status, llmmm_last_error());
    return nullptr;
  }
  Py_RETURN_TRUE;
}

// Runs `body`; whatever is not the plain case (or any C++ exception of a tensor without storage) is left to capi.py.
template<Py_ssize_t N, class F>
PyObject* plain_or_false(Py_ssize_t nargs, F&& body)
{
  if (nargs != N) {
    Py_RETURN_FALSE;
  }
  try {
    return body();
  }
  catch (...) {
    Py_RETURN_FALSE;
  }
}

PyObject* fp16_mm(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<7>(n, [&]() -> PyObject* {
    void* const A = bytes(a[0]);
    const auto  t = THPVariable_Unpack(a[0]).scalar_type();
    if (t == c10::ScalarType::Half) {
      void *B = pointer<c10::ScalarType::Half>(a[1]), *C = pointer<c10::ScalarType::Half>(a[2]);
      const int M = integer(a[3]), N = integer(a[4]), K = integer(a[5]);
      return call_on(a[0], a[6], [&](llmmm_stream_t s) { return llmmm_fp16_mm_f16(A, B, C, M, N, K, s); });
    }
    if (t == c10::ScalarType::BFloat16) {
      void *B = pointer<c10::ScalarType::BFloat16>(a[1]), *C = pointer<c10::ScalarType::BFloat16>(a[2]);
      const int M = integer(a[3]), N = integer(a[4]), K = integer(a[5]);
      return call_on(a[0], a[6], [&](llmmm_stream_t s) { return llmmm_fp16_mm_bf16(A, B, C, M, N, K, s); });
    }
    throw NotPlain{};
  });
}

PyObject* fp8_blockwise_mm(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<10>(n, [&]() -> PyObject* {
    void *A = bytes(a[0]), *B = bytes(a[2]), *C = bytes(a[4]);
    float *A_s = f32(a[1]), *B_s = f32(a[3]), *C_s = f32(a[5]);
    const int M = integer(a[6]), N = integer(a[7]), K = integer(a[8]);
    return call_on(a[0], a[9], [&](llmmm_stream_t s) { return llmmm_fp8_blockwise_mm_e4m3out(A, A_s, B, B_s, C, C_s, M, N, K, s); });
  });
}

PyObject* fp8_blockwise_mm_f32(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<9>(n, [&]() -> PyObject* {
    void *A = bytes(a[0]), *B = bytes(a[2]);
    float *A_s = f32(a[1]), *B_s = f32(a[3]), *C = f32(a[4]);
    const int M = integer(a[5]), N = integer(a[6]), K = integer(a[7]);
    return call_on(a[0], a[8], [&](llmmm_stream_t s) { return llmmm_fp8_blockwise_mm_f32out(A, A_s, B, B_s, C, M, N, K, s); });
  });
}

PyObject* fp8_blockwise_mm_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<10>(n, [&]() -> PyObject* {
    void *A = bytes(a[0]), *B = bytes(a[2]), *H = bytes(a[4]);
    float *A_s = f32(a[1]), *B_s = f32(a[3]), *H_s = f32(a[5]);
    const int M = integer(a[6]), I = integer(a[7]), K = integer(a[8]);
    return call_on(a[0], a[9], [&](llmmm_stream_t s) { return llmmm_fp8_blockwise_mm_swiglu_e4m3out(A, A_s, B, B_s, H, H_s, M, I, K, s); });
  });
}

// (cos and sin have been looked at by capi.py)
PyObject* fp8_blockwise_mm_qk_norm_rope(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<18>(n, [&]() -> PyObject* {
    void *A = bytes(a[0]), *B = bytes(a[2]), *C = bytes(a[4]);
    float *A_s = f32(a[1]), *B_s = f32(a[3]), *C_s = f32(a[5]);
    int*  pos = i32(a[6]);
    float *cos = f32(a[7]), *sin = f32(a[8]), *q_w = f32_or_null(a[9]), *k_w = f32_or_null(a[10]);
    const float eps = real(a[11]);
    const int   n_q = integer(a[12]), n_kv = integer(a[13]), M = integer(a[14]), N = integer(a[15]), K = integer(a[16]);
    const int   rows = (int)THPVariable_Unpack(a[7]).size(0);
    return call_on(a[0], a[17], [&](llmmm_stream_t s) {
      return llmmm_fp8_blockwise_mm_qk_norm_rope_e4m3out(A, A_s, B, B_s, C, C_s, pos, cos, sin, rows, q_w, k_w, eps, n_q, n_kv, M, N, K, s);
    });
  });
}

template<int (*FN)(const float*, void*, float*, int, int, llmmm_stream_t)>
PyObject* quantise(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<6>(n, [&]() -> PyObject* {
    float*    x = f32(a[0]);
    void*     q = bytes(a[1]);
    float*    scale = f32(a[2]);
    const int M = integer(a[3]), K = integer(a[4]);
    return call_on(a[0], a[5], [&](llmmm_stream_t s) { return FN(x, q, scale, M, K, s); });
  });
}

PyObject* fp8_rmsnorm_quant_1x128(PyObject*, PyObject* const* a, Py_ssize_t n)
{
  return plain_or_false<8>(n, [&]() -> PyObject* {
    float *     x = f32(a[0]), *w = f32(a[1]);
    const float eps = real(a[2]);
    void*       q = bytes(a[3]);
    float*      scale = f32(a[4]);
    const int   M = integer(a[5]), K = integer(a[6]);
    return call_on(a[0], a[7], [&](llmmm_stream_t s) { return llmmm_fp8_rmsnorm_quant_1x128(x, w, eps, q, scale, M, K, s); });
  });
}

#define LLMMM_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef METHODS[] = {
  LLMMM_METHOD("fp16_mm", fp16_mm),
  LLMMM_METHOD("fp8_blockwise_mm", fp8_blockwise_mm),
  LLMMM_METHOD("fp8_blockwise_mm_f32", fp8_blockwise_mm_f32),
  LLMMM_METHOD("fp8_blockwise_mm_swiglu", fp8_blockwise_mm_swiglu),
  LLMMM_METHOD("fp8_blockwise_mm_qk_norm_rope", fp8_blockwise_mm_qk_norm_rope),
  LLMMM_METHOD("fp8_quant_1x128", quantise<llmmm_fp8_quant_1x128>),
  LLMMM_METHOD("fp8_quant_128x128", quantise<llmmm_fp8_quant_128x128>),
  LLMMM_METHOD("fp8_rmsnorm_quant_1x128", fp8_rmsnorm_quant_1x128),
  {nullptr, nullptr, 0, nullptr},
};

PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, METHODS};

}  // namespace

PyMODINIT_FUNC PyInit__binding()
{
  PyObject* m = PyModule_Create(&MODULE);
  if (m != nullptr && PyModule_AddStringConstant(m, "BUILT_FOR", LLMMM_BUILT_FOR) != 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
