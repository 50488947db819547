// The operator calls of sofie_b200/ops.py on torch tensors, natively: argument unpacking, the output tensor from torch's caching
// allocator, the descriptor and the call through the C ABI of libSOFIE_cuda. A call costs the host about as much as the kernel
// launch itself; the same steps in Python with ctypes were 10 us, which is what bounded every call below a few hundred kilobytes.
// Nothing here computes, and nothing falls back: a status other than 0 raises what sofie_b200.capi.check raises for it.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <string>
#include <vector>

#include "sofie_cuda.h"

namespace {

struct Raised {}; // a Python exception is set

[[noreturn]] void raise(PyObject *type, const char *text)
{
   PyErr_SetString(type, text);
   throw Raised();
}

const at::Tensor &tensor(PyObject *o)
{
   if (!THPVariable_Check(o)) raise(PyExc_TypeError, "a torch tensor is expected");
   return THPVariable_Unpack(o);
}
void *data(const at::Tensor &t)
{
   if (!(t.is_cuda() && t.is_contiguous())) raise(PyExc_AssertionError, "tensors passed to libSOFIE_cuda must be contiguous CUDA tensors");
   return t.data_ptr();
}
void *data(PyObject *o) { return o == Py_None ? nullptr : data(tensor(o)); }
template <typename T>
T *as(PyObject *o) { return static_cast<T *>(data(o)); }
template <typename T>
T *as(const at::Tensor &t) { return static_cast<T *>(data(t)); }

int64_t integer(PyObject *o)
{
   const long long v = PyLong_AsLongLong(o);
   if (v == -1 && PyErr_Occurred()) throw Raised();
   return v;
}
int32_t i32(PyObject *o) { return static_cast<int32_t>(integer(o)); }
// what int(o) gives: a zero point may come as a float or as a NumPy or torch scalar
int32_t as_int32(PyObject *o)
{
   PyObject *v = PyNumber_Long(o);
   if (!v) throw Raised();
   const long long n = PyLong_AsLongLong(v);
   Py_DECREF(v);
   if (n == -1 && PyErr_Occurred()) throw Raised();
   return static_cast<int32_t>(n);
}
float f32(PyObject *o)
{
   const double v = PyFloat_AsDouble(o);
   if (v == -1.0 && PyErr_Occurred()) throw Raised();
   return static_cast<float>(v);
}
bool truth(PyObject *o)
{
   const int v = PyObject_IsTrue(o);
   if (v < 0) throw Raised();
   return v != 0;
}
// The first N of a sequence of integers: of exactly N, or of N or more.
template <size_t N>
std::array<int32_t, N> ints(PyObject *o, bool exactly)
{
   PyObject *s = PySequence_Fast(o, "a sequence of integers is expected");
   if (!s) throw Raised();
   std::array<int32_t, N> v{};
   const Py_ssize_t size = PySequence_Fast_GET_SIZE(s);
   const bool fits = exactly ? size == (Py_ssize_t)N : size >= (Py_ssize_t)N;
   try {
      for (size_t i = 0; fits && i < N; i++) v[i] = i32(PySequence_Fast_GET_ITEM(s, i));
   } catch (...) {
      Py_DECREF(s);
      throw;
   }
   Py_DECREF(s);
   if (!fits) raise(exactly ? PyExc_ValueError : PyExc_IndexError, "a sequence of another length is expected");
   return v;
}
std::array<int32_t, 2> pair(PyObject *o) { return ints<2>(o, false); } // of a longer padding or kernel, the first two
// the extents of a tensor of rank N
template <size_t N>
std::array<int32_t, N> extents(const at::Tensor &t)
{
   if (t.dim() != (int64_t)N) raise(PyExc_ValueError, "a tensor of another rank is expected");
   std::array<int32_t, N> v;
   for (size_t i = 0; i < N; i++) v[i] = (int32_t)t.size((int64_t)i);
   return v;
}
std::array<int32_t, 4> image_shape(PyObject *shape, const at::Tensor &X) { return shape != Py_None ? ints<4>(shape, true) : extents<4>(X); }

void *stream() { return at::cuda::getCurrentCUDAStream().stream(); }

at::Tensor make(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like)
{
   return at::Tensor(at::detail::empty_cuda(shape, type, like.device(), std::nullopt));
}
// the result of an operator on 32-bit values: of X's type; a type of fewer bytes holds less than the kernel would read and write
at::Tensor make_like(const at::Tensor &X)
{
   if (X.element_size() < 4) raise(PyExc_AssertionError, "a tensor of float32 values is expected");
   return make(X.sizes(), X.scalar_type(), X);
}
at::Tensor make_or(PyObject *out, at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like)
{
   return out == Py_None ? make(shape, type, like) : tensor(out);
}

void check(int rc, const char *name)
{
   if (rc == 0) return;
   PyObject *capi = PyImport_ImportModule("sofie_b200.capi");
   PyObject *r = capi ? PyObject_CallMethod(capi, "check", "is", rc, name) : nullptr;
   Py_XDECREF(r);
   Py_XDECREF(capi);
   if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, name);
   throw Raised();
}
// The call itself runs without the interpreter lock (several threads may launch at the same time), as a ctypes call does.
#define SOFIE_CALL(fn, ...)              \
   do {                                  \
      int rc__;                          \
      Py_BEGIN_ALLOW_THREADS;            \
      rc__ = fn(__VA_ARGS__);            \
      Py_END_ALLOW_THREADS;              \
      check(rc__, #fn);                  \
   } while (0)

using Args = PyObject *const *;

void require(bool ok, const char *what)
{
   if (!ok) raise(PyExc_AssertionError, what);
}

// A, B, C, transA, transB, alpha, beta, relu, out, workspace
PyObject *gemm_f32(Args a)
{
   const at::Tensor &A = tensor(a[0]), &B = tensor(a[1]);
   const bool tA = truth(a[3]), tB = truth(a[4]);
   const int64_t M = A.size(tA ? 1 : 0), K = A.size(tA ? 0 : 1), N = B.size(tB ? 0 : 1);
   require(B.size(tB ? 1 : 0) == K, "the operands' inner dimensions differ");
   int32_t bias = 0;
   if (a[2] != Py_None) {
      const int64_t n = tensor(a[2]).numel();
      require(n == N || n == M * N, "C is neither a row nor of the output's shape");
      bias = n == N ? 1 : 2;
   }
   at::Tensor Y = make_or(a[8], {M, N}, at::kFloat, A);
   const sofie_gemm_f32_desc d = {(int32_t)M, (int32_t)N, (int32_t)K, tA, tB, f32(a[5]), f32(a[6]), bias, truth(a[7])};
   void *const s = stream();
   const float *pA = as<float>(A), *pB = as<float>(B), *pC = as<float>(a[2]);
   float *pY = as<float>(Y);
   // a workspace where one makes the product faster, from torch's pool of this stream; without memory for it the product does without
   const size_t bytes = truth(a[9]) ? sofie_cuda_gemm_f32_workspace(&d) : 0;
   at::Tensor workspace;
   if (bytes) {
      try {
         workspace = make({(int64_t)bytes}, at::kByte, A);
      } catch (const c10::OutOfMemoryError &) {
      }
   }
   void *const w = workspace.defined() ? workspace.data_ptr() : nullptr;
   SOFIE_CALL(sofie_cuda_gemm_f32_ws, s, &d, pA, pB, pC, pY, w, w ? bytes : 0);
   return THPVariable_Wrap(Y);
}

struct ConvShape {
   int32_t N, C, H, W, Cout, kH, kW, oH, oW;
   std::array<int64_t, 4> y;
};
ConvShape conv_shape(const at::Tensor &X, const at::Tensor &W, PyObject *shape, PyObject *kernel, bool packed, const std::array<int32_t, 2> &pad,
                     const std::array<int32_t, 2> &stride, const std::array<int32_t, 2> &dil, int32_t pool, int32_t y_layout)
{
   ConvShape c;
   const auto s = image_shape(shape, X);
   c.N = s[0], c.C = s[1], c.H = s[2], c.W = s[3];
   c.Cout = (int32_t)W.size(0);
   if (packed) {
      const auto k = pair(kernel);
      c.kH = k[0], c.kW = k[1];
   } else {
      c.kH = (int32_t)W.size(2), c.kW = (int32_t)W.size(3);
   }
   c.oH = (c.H + 2 * pad[0] - (dil[0] * (c.kH - 1) + 1)) / stride[0] + 1;
   c.oW = (c.W + 2 * pad[1] - (dil[1] * (c.kW - 1) + 1)) / stride[1] + 1;
   if (pool == 2) c.oH /= 2, c.oW /= 2;
   // a kernel larger than the padded image: the call reports it, the output only has to exist
   const int64_t oh = c.oH < 0 ? 0 : c.oH, ow = c.oW < 0 ? 0 : c.oW;
   c.y = y_layout == SOFIE_LAYOUT_NHWC ? std::array<int64_t, 4>{c.N, oh, ow, c.Cout} : std::array<int64_t, 4>{c.N, c.Cout, oh, ow};
   return c;
}

// X, W, bias, shape, pad, stride, dil, group, relu, pool, x_layout, y_layout, w_packed, kernel, out
PyObject *conv2d_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]), &W = tensor(a[1]);
   const auto pad = pair(a[4]), stride = pair(a[5]), dil = pair(a[6]);
   require(stride[0] > 0 && stride[1] > 0, "strides must be positive");
   const int32_t pool = i32(a[9]), yl = i32(a[11]);
   const bool packed = truth(a[12]);
   const ConvShape c = conv_shape(X, W, a[3], a[13], packed, pad, stride, dil, pool, yl);
   at::Tensor Y = make_or(a[14], c.y, at::kFloat, X);
   const sofie_conv2d_desc d = {c.N, c.C, c.H, c.W, c.Cout, c.kH, c.kW, pad[0], pad[1], stride[0], stride[1], dil[0], dil[1], i32(a[7]),
                                i32(a[10]), yl, packed, truth(a[8]), pool};
   void *const s = ::stream();
   const float *pX = as<float>(X), *pW = as<float>(W), *pB = as<float>(a[2]);
   float *pY = as<float>(Y);
   SOFIE_CALL(sofie_cuda_conv2d_f32, s, &d, pX, pW, pB, pY);
   return THPVariable_Wrap(Y);
}

// X, W, mult, bias, shape, pad, stride, x_zp, y_zp, relu, pool, x_layout, y_layout, w_packed, kernel
PyObject *qlinear_conv2d(Args a)
{
   const at::Tensor &X = tensor(a[0]), &W = tensor(a[1]);
   const auto pad = pair(a[5]), stride = pair(a[6]);
   require(stride[0] > 0 && stride[1] > 0, "strides must be positive");
   const int32_t pool = i32(a[10]), yl = i32(a[12]);
   const bool packed = truth(a[13]);
   const ConvShape c = conv_shape(X, W, a[4], a[14], packed, pad, stride, {1, 1}, pool, yl);
   at::Tensor Y = make(c.y, at::kByte, X);
   const sofie_qconv2d_desc d = {c.N, c.C, c.H, c.W, c.Cout, c.kH, c.kW, pad[0], pad[1], stride[0], stride[1], i32(a[11]), yl, packed,
                                 as_int32(a[7]), as_int32(a[8]), truth(a[9]), pool};
   void *const s = ::stream();
   const uint8_t *pX = as<uint8_t>(X);
   const int8_t *pW = as<int8_t>(W);
   const float *pm = as<float>(a[2]);
   const int32_t *pb = as<int32_t>(a[3]);
   uint8_t *pY = as<uint8_t>(Y);
   SOFIE_CALL(sofie_cuda_qlinear_conv2d, s, &d, pX, pW, pm, pb, pY);
   return THPVariable_Wrap(Y);
}

// X, out
PyObject *relu_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = a[1] == Py_None ? make_like(X) : tensor(a[1]);
   void *const s = stream();
   const float *pX = as<float>(X);
   float *pY = as<float>(Y);
   const size_t n = (size_t)X.numel();
   SOFIE_CALL(sofie_cuda_relu_f32, s, pX, pY, n);
   return THPVariable_Wrap(Y);
}

// X, op, alpha
PyObject *unary_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = make_like(X);
   void *const s = stream();
   const int32_t op = i32(a[1]);
   const float alpha = f32(a[2]);
   const float *pX = as<float>(X);
   float *pY = as<float>(Y);
   const size_t n = (size_t)X.numel();
   SOFIE_CALL(sofie_cuda_unary_f32, s, op, alpha, pX, pY, n);
   return THPVariable_Wrap(Y);
}

// A, B, op
PyObject *binary_f32(Args a)
{
   const at::Tensor &A = tensor(a[0]), &B = tensor(a[1]);
   const int64_t ra = A.dim(), rb = B.dim(), rank = ra > rb ? ra : rb;
   if (rank > 4) raise(PyExc_ValueError, "binary operators are built for rank <= 4");
   sofie_binary_desc d = {};
   d.op = i32(a[2]);
   int64_t da = 1, db = 1;
   for (int i = 3; i >= 0; i--) {
      const int64_t at_a = ra - 4 + i, at_b = rb - 4 + i, na = at_a >= 0 ? A.size(at_a) : 1, nb = at_b >= 0 ? B.size(at_b) : 1;
      if (na != nb && na != 1 && nb != 1) raise(PyExc_RuntimeError, "the operands' shapes cannot be broadcast together");
      d.shape[i] = na == 1 ? nb : na;
      d.a_stride[i] = na == 1 ? 0 : da;
      d.b_stride[i] = nb == 1 ? 0 : db;
      da *= na, db *= nb;
   }
   at::Tensor Y = make(at::IntArrayRef(d.shape + (4 - rank), (size_t)rank), at::kFloat, A);
   void *const s = stream();
   const float *pA = as<float>(A), *pB = as<float>(B);
   float *pY = as<float>(Y);
   SOFIE_CALL(sofie_cuda_binary_f32, s, &d, pA, pB, pY);
   return THPVariable_Wrap(Y);
}

// X, scale, bias, mean, N, C, HW, layout, relu
PyObject *batchnorm_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = make_like(X);
   const sofie_batchnorm_desc d = {i32(a[4]), i32(a[5]), i32(a[6]), i32(a[7]), truth(a[8])};
   void *const s = stream();
   const float *pX = as<float>(X), *ps = as<float>(a[1]), *pb = as<float>(a[2]), *pm = as<float>(a[3]);
   float *pY = as<float>(Y);
   SOFIE_CALL(sofie_cuda_batchnorm_f32, s, &d, pX, ps, pb, pm, pY);
   return THPVariable_Wrap(Y);
}

// X, mode, kernel, stride, pads, count_include_pad, layout, shape
PyObject *pool2d_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   const auto k = pair(a[2]), st = pair(a[3]);
   const auto p = ints<4>(a[4], true);
   require(st[0] > 0 && st[1] > 0, "strides must be positive");
   const auto n = image_shape(a[7], X);
   auto out = [&](int i) {
      const int64_t v = n[2 + i] + p[i] + p[2 + i] - k[i] + 1;
      return v <= 0 ? int64_t(0) : (v + st[i] - 1) / st[i];
   };
   const int64_t oH = out(0), oW = out(1);
   const int32_t layout = i32(a[6]);
   at::Tensor Y = layout == SOFIE_LAYOUT_NHWC ? make({n[0], oH, oW, n[1]}, at::kFloat, X) : make({n[0], n[1], oH, oW}, at::kFloat, X);
   const sofie_pool2d_desc d = {i32(a[1]), n[0], n[1], n[2], n[3], k[0], k[1], st[0], st[1], {p[0], p[1], p[2], p[3]}, i32(a[5]), layout};
   void *const s = stream();
   const float *pX = as<float>(X);
   float *pY = as<float>(Y);
   SOFIE_CALL(sofie_cuda_pool2d_f32, s, &d, pX, pY);
   return THPVariable_Wrap(Y);
}

// X, kernel, stride, layout, shape
PyObject *maxpool2d_u8(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   const auto k = pair(a[1]), st = pair(a[2]);
   require(st[0] > 0 && st[1] > 0, "strides must be positive");
   const auto n = image_shape(a[4], X);
   const int64_t oH = n[2] < k[0] ? 0 : (n[2] - k[0]) / st[0] + 1, oW = n[3] < k[1] ? 0 : (n[3] - k[1]) / st[1] + 1;
   const int32_t layout = i32(a[3]);
   at::Tensor Y = layout == SOFIE_LAYOUT_NHWC ? make({n[0], oH, oW, n[1]}, at::kByte, X) : make({n[0], n[1], oH, oW}, at::kByte, X);
   void *const s = stream();
   const uint8_t *pX = as<uint8_t>(X);
   uint8_t *pY = as<uint8_t>(Y);
   SOFIE_CALL(sofie_cuda_maxpool2d_u8, s, pX, pY, n[0], n[1], n[2], n[3], k[0], k[1], st[0], st[1], layout);
   return THPVariable_Wrap(Y);
}

// X, axis
PyObject *softmax_f32(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   const int64_t rank = X.dim();
   if (rank == 0) raise(PyExc_ZeroDivisionError, "Softmax of a scalar");
   const int64_t axis = ((integer(a[1]) % rank) + rank) % rank;
   size_t outer = 1, inner = 1;
   for (int64_t i = 0; i < axis; i++) outer *= (size_t)X.size(i);
   for (int64_t i = axis + 1; i < rank; i++) inner *= (size_t)X.size(i);
   const size_t len = (size_t)X.size(axis);
   at::Tensor Y = make_like(X);
   void *const s = stream();
   const float *pX = as<float>(X);
   float *pY = as<float>(Y);
   SOFIE_CALL(sofie_cuda_softmax_f32, s, pX, pY, outer, len, inner);
   return THPVariable_Wrap(Y);
}

// X, to_nhwc
PyObject *change_layout(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   require(X.dim() == 4, "a tensor of rank 4 is expected");
   const bool to_nhwc = truth(a[1]), f = X.scalar_type() == at::kFloat;
   const int64_t N = X.size(0), C = X.size(to_nhwc ? 1 : 3), H = X.size(to_nhwc ? 2 : 1), W = X.size(to_nhwc ? 3 : 2);
   at::Tensor Y = to_nhwc ? make({N, H, W, C}, X.scalar_type(), X) : make({N, C, H, W}, X.scalar_type(), X);
   void *const s = stream();
   void *const pX = data(X), *const pY = data(Y);
   const int32_t n = (int32_t)N, c = (int32_t)C, h = (int32_t)H, w = (int32_t)W;
   if (f && to_nhwc) SOFIE_CALL(sofie_cuda_nchw_to_nhwc_f32, s, (const float *)pX, (float *)pY, n, c, h, w);
   else if (f) SOFIE_CALL(sofie_cuda_nhwc_to_nchw_f32, s, (const float *)pX, (float *)pY, n, c, h, w);
   else if (to_nhwc) SOFIE_CALL(sofie_cuda_nchw_to_nhwc_u8, s, (const uint8_t *)pX, (uint8_t *)pY, n, c, h, w);
   else SOFIE_CALL(sofie_cuda_nhwc_to_nchw_u8, s, (const uint8_t *)pX, (uint8_t *)pY, n, c, h, w);
   return THPVariable_Wrap(Y);
}

// X, scale, zp
PyObject *quantize_u8(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = make(X.sizes(), at::kByte, X);
   void *const s = stream();
   const float scale = f32(a[1]);
   const int32_t zp = as_int32(a[2]);
   const float *pX = as<float>(X);
   uint8_t *pY = as<uint8_t>(Y);
   const size_t n = (size_t)X.numel();
   SOFIE_CALL(sofie_cuda_quantize_u8, s, pX, pY, n, scale, zp);
   return THPVariable_Wrap(Y);
}
// X, scale, zp
PyObject *dequantize_u8(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = make(X.sizes(), at::kFloat, X);
   void *const s = stream();
   const float scale = f32(a[1]);
   const int32_t zp = as_int32(a[2]);
   const uint8_t *pX = as<uint8_t>(X);
   float *pY = as<float>(Y);
   const size_t n = (size_t)X.numel();
   SOFIE_CALL(sofie_cuda_dequantize_u8, s, pX, pY, n, scale, zp);
   return THPVariable_Wrap(Y);
}
// X, scale
PyObject *quantize_e4m3(Args a)
{
   const at::Tensor &X = tensor(a[0]);
   at::Tensor Y = make(X.sizes(), at::kByte, X);
   void *const s = stream();
   const float scale = f32(a[1]);
   void *const pX = data(X);
   uint8_t *pY = as<uint8_t>(Y);
   const size_t n = (size_t)X.numel();
   if (X.scalar_type() == at::kFloat) {
      SOFIE_CALL(sofie_cuda_quantize_e4m3_f32, s, (const float *)pX, pY, n, scale);
   } else {
      require(X.element_size() == 2 && X.scalar_type() != at::kHalf, "quantize_e4m3 takes float32 or bfloat16 (or its bits)");
      SOFIE_CALL(sofie_cuda_quantize_e4m3_bf16, s, (const uint16_t *)pX, pY, n, scale);
   }
   return THPVariable_Wrap(Y);
}

// A, W, mult, corr, w_is_nk, y_zp, relu, y_scale (None: uint8 result)
PyObject *qlinear_matmul(Args a)
{
   const at::Tensor &A = tensor(a[0]), &W = tensor(a[1]);
   const bool nk = truth(a[4]), to_f32 = a[7] != Py_None;
   const auto mk = extents<2>(A);
   const int64_t M = mk[0], K = mk[1], N = W.size(nk ? 0 : 1);
   at::Tensor Y = make({M, N}, to_f32 ? at::kFloat : at::kByte, A);
   const sofie_qgemm_desc d = {(int32_t)M, (int32_t)N, (int32_t)K, nk, as_int32(a[5]), truth(a[6])};
   void *const s = stream();
   const uint8_t *pA = as<uint8_t>(A);
   const int8_t *pW = as<int8_t>(W);
   const float *pm = as<float>(a[2]);
   const int32_t *pc = as<int32_t>(a[3]);
   void *const pY = data(Y);
   if (to_f32) {
      const float scale = f32(a[7]);
      SOFIE_CALL(sofie_cuda_qlinear_matmul_f32, s, &d, pA, pW, pm, pc, scale, (float *)pY);
   } else {
      SOFIE_CALL(sofie_cuda_qlinear_matmul, s, &d, pA, pW, pm, pc, (uint8_t *)pY);
   }
   return THPVariable_Wrap(Y);
}

// A, W, bias, a_scale, w_scale, relu, q_scale, want_bf16, to_f32
PyObject *gemm_e4m3(Args a)
{
   const at::Tensor &A = tensor(a[0]), &W = tensor(a[1]);
   const auto mk = extents<2>(A);
   const int64_t M = mk[0], K = mk[1], N = W.size(0);
   const sofie_fp8_gemm_desc d = {(int32_t)M, (int32_t)N, (int32_t)K, f32(a[3]), f32(a[4]), truth(a[5]), f32(a[6])};
   void *const s = stream();
   const uint8_t *pA = as<uint8_t>(A), *pW = as<uint8_t>(W);
   const float *pb = as<float>(a[2]);
   if (truth(a[8])) {
      at::Tensor Y = make({M, N}, at::kFloat, A);
      float *pY = as<float>(Y);
      SOFIE_CALL(sofie_cuda_gemm_e4m3_f32, s, &d, pA, pW, pb, pY);
      return THPVariable_Wrap(Y);
   }
   at::Tensor Y, Yq;
   if (truth(a[7])) Y = make({M, N}, at::kBFloat16, A);
   if (d.q_scale > 0.f) Yq = make({M, N}, at::kByte, A);
   uint16_t *pY = Y.defined() ? as<uint16_t>(Y) : nullptr;
   uint8_t *pq = Yq.defined() ? as<uint8_t>(Yq) : nullptr;
   SOFIE_CALL(sofie_cuda_gemm_e4m3, s, &d, pA, pW, pb, pY, pq);
   PyObject *y = Y.defined() ? THPVariable_Wrap(Y) : Py_NewRef(Py_None), *q = Yq.defined() ? THPVariable_Wrap(Yq) : Py_NewRef(Py_None);
   PyObject *both = PyTuple_New(2);
   PyTuple_SET_ITEM(both, 0, y);
   PyTuple_SET_ITEM(both, 1, q);
   return both;
}

template <PyObject *(*F)(Args), int N>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n)
{
   HANDLE_TH_ERRORS
   if (n != N) {
      PyErr_Format(PyExc_TypeError, "%d arguments are expected, got %zd", N, n);
      return nullptr;
   }
   try {
      return F(args);
   } catch (const Raised &) {
      return nullptr;
   }
   END_HANDLE_TH_ERRORS
}

#define SOFIE_ENTRY(name, n) {#name, (PyCFunction)(void (*)(void))entry<name, n>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {SOFIE_ENTRY(gemm_f32, 10),       SOFIE_ENTRY(conv2d_f32, 15),     SOFIE_ENTRY(qlinear_conv2d, 15), SOFIE_ENTRY(relu_f32, 2),
                         SOFIE_ENTRY(unary_f32, 3),      SOFIE_ENTRY(binary_f32, 3),      SOFIE_ENTRY(batchnorm_f32, 9),   SOFIE_ENTRY(pool2d_f32, 8),
                         SOFIE_ENTRY(maxpool2d_u8, 5),   SOFIE_ENTRY(softmax_f32, 2),     SOFIE_ENTRY(change_layout, 2),   SOFIE_ENTRY(quantize_u8, 3),
                         SOFIE_ENTRY(dequantize_u8, 3),  SOFIE_ENTRY(quantize_e4m3, 2),   SOFIE_ENTRY(qlinear_matmul, 8),  SOFIE_ENTRY(gemm_e4m3, 9),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ops", "Operator calls of libSOFIE_cuda on torch tensors", -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__ops() { return PyModule_Create(&module); }
