// Elementwise family next to the contractions: unary activations and maths, binary operators with
// broadcasting, inference-mode BatchNormalization. All are HBM-bound: 16-byte accesses where the
// tensors allow, a grid of a few waves of 148 SMs. The arithmetic follows the text the reference
// emits for each operator (cited per case), evaluated in the same precision.
#include "common.cuh"

#include <initializer_list>
#include <utility>

namespace sofie {
namespace {

constexpr int kActThreads = 256;

inline int act_grid(size_t items)
{
   size_t blocks = (items + kActThreads - 1) / kActThreads;
   const size_t cap = size_t(kNumSMs) * 8;
   if (blocks > cap) blocks = cap;
   return blocks ? (int)blocks : 1;
}

template <int OP>
__device__ __forceinline__ float unary_apply(float x, float alpha)
{
   switch (OP) {
   case SOFIE_UNARY_SIGMOID: return __frcp_rn(__fadd_rn(1.f, expf(-x)));               // ROperator_Sigmoid.hxx:59 (1 / y, rounded as a division)
   case SOFIE_UNARY_TANH: return tanhf(x);                                             // ROperator_Tanh.hxx:60
   case SOFIE_UNARY_LEAKY_RELU: return x >= 0.f ? x : __fmul_rn(alpha, x);             // ROperator_LeakyRelu.hxx:73
   case SOFIE_UNARY_SELU: {                                                            // ROperator_Selu.hxx:59 (double constants)
      const double neg = 1.6732632423543772848170429916717 * (double)(expf(x) - 1.f);
      return (float)(1.0507009873554804934193349852946 * ((double)fmaxf(0.f, x) + fmin(0.0, neg)));
   }
   case SOFIE_UNARY_ELU: return x >= 0.f ? x : __fsub_rn(__fmul_rn(alpha, expf(x)), 1.f); // ROperator_Elu.hxx:71 (as written there)
   case SOFIE_UNARY_NEG: return -x;
   case SOFIE_UNARY_EXP: return expf(x);
   case SOFIE_UNARY_LOG: return logf(x);
   case SOFIE_UNARY_SQRT: return sqrtf(x);
   case SOFIE_UNARY_RECIPROCAL: return __frcp_rn(x); // as a division rounds
   case SOFIE_UNARY_ERF: return erff(x);                                               // ROperator_Erf.hxx:58
   case SOFIE_UNARY_SWISH: return __fdiv_rn(x, __fadd_rn(1.f, expf(-x)));              // ROperator_Swish.hxx:59
   case SOFIE_UNARY_COS: return cosf(x);
   case SOFIE_UNARY_SIN: return sinf(x);
   default: return fabsf(x); // SOFIE_UNARY_ABS
   }
}

template <int OP>
__global__ void __launch_bounds__(kActThreads) unary_f32_kernel(float alpha, const float *__restrict__ X, float *__restrict__ Y, size_t n, bool vec)
{
   griddep_launch_dependents();
   griddep_wait(X); // X is the previous kernel's output
   const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nthreads = (size_t)gridDim.x * blockDim.x;
   const size_t n4 = vec ? n / 4 : 0;
   // four loads under way before the first value is worked on: with two, functions of twenty instructions a value kept too few (sigmoid of 134 MB 59.4 -> 47.0 us, part
   // of it the reciprocal in place of the division)
   size_t i = tid;
   for (; i + 3 * nthreads < n4; i += 4 * nthreads) {
      float4 v[4];
#pragma unroll
      for (int k = 0; k < 4; k++) v[k] = reinterpret_cast<const float4 *>(X)[i + k * nthreads];
#pragma unroll
      for (int k = 0; k < 4; k++)
         reinterpret_cast<float4 *>(Y)[i + k * nthreads] =
            make_float4(unary_apply<OP>(v[k].x, alpha), unary_apply<OP>(v[k].y, alpha), unary_apply<OP>(v[k].z, alpha), unary_apply<OP>(v[k].w, alpha));
   }
   for (; i < n4; i += nthreads) {
      const float4 v = reinterpret_cast<const float4 *>(X)[i];
      reinterpret_cast<float4 *>(Y)[i] =
         make_float4(unary_apply<OP>(v.x, alpha), unary_apply<OP>(v.y, alpha), unary_apply<OP>(v.z, alpha), unary_apply<OP>(v.w, alpha));
   }
   for (size_t j = n4 * 4 + tid; j < n; j += nthreads) Y[j] = unary_apply<OP>(X[j], alpha);
}

using UnaryKernel = void (*)(float, const float *, float *, size_t, bool);
template <int... OP>
UnaryKernel unary_kernel(int op, std::integer_sequence<int, OP...>)
{
   static constexpr UnaryKernel table[] = {unary_f32_kernel<OP>...};
   return table[op];
}

__device__ __forceinline__ float binary_apply(int op, float a, float b)
{
   switch (op) { // ROperator_BasicBinary.hxx:18-43
   case SOFIE_BINARY_ADD: return __fadd_rn(a, b);
   case SOFIE_BINARY_SUB: return __fsub_rn(a, b);
   case SOFIE_BINARY_MUL: return __fmul_rn(a, b);
   default: return __fdiv_rn(a, b);
   }
}

// Two tensors in, one out: 32-byte accesses keep more in flight. 134 MB tensors 71.7 -> 67.6 us (6.0 TB/s), 1 GB tensors 513 -> 487 us;
// for one tensor in they gain nothing (Relu 49.2 us both ways) or lose (Sigmoid 51.1 -> 55.3 us), so those stay with 16 bytes.
__global__ void binary_same_f32_kernel(int op, const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ Y, size_t n,
                                       int vec)
{
   griddep_launch_dependents();
   griddep_wait(A, B);
   const size_t tid = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nthreads = (size_t)gridDim.x * blockDim.x;
   const size_t n4 = vec == 4 ? n / 4 : 0, n8 = vec == 8 ? n / 8 : 0;
#pragma unroll 2
   for (size_t i = tid; i < n8; i += nthreads) {
      float a[8], b[8];
      load_f32x8(A + 8 * i, a);
      load_f32x8(B + 8 * i, b);
#pragma unroll
      for (int j = 0; j < 8; j++) a[j] = binary_apply(op, a[j], b[j]);
      store_f32x8(Y + 8 * i, a);
   }
#pragma unroll 2
   for (size_t i = tid; i < n4; i += nthreads) {
      const float4 a = reinterpret_cast<const float4 *>(A)[i], b = reinterpret_cast<const float4 *>(B)[i];
      reinterpret_cast<float4 *>(Y)[i] =
         make_float4(binary_apply(op, a.x, b.x), binary_apply(op, a.y, b.y), binary_apply(op, a.z, b.z), binary_apply(op, a.w, b.w));
   }
   for (size_t i = n8 * 8 + n4 * 4 + tid; i < n; i += nthreads) Y[i] = binary_apply(op, A[i], B[i]);
}

// Broadcasting. The dimensions are merged as far as both operands allow (an [N,C,H,W] tensor and a [C,1,1] one become [N,C,HW]); a
// thread writes four consecutive outputs. An operand that lies like the output is read as one 16-byte word, the other by
// coordinates: those of the first output by multiplications (FastDiv), the next ones by counting on. Measured on [512,16,64,64]
// times [16,1,1]: 250 us with four 64-bit divisions per element, 43 us here (a copy of the bytes takes 41).
struct BcastDims {
   FastDiv shape[4]; // innermost first
   uint32_t a[4], b[4];
};
template <bool A_DENSE, bool B_DENSE>
__global__ void __launch_bounds__(kActThreads) binary_bcast_f32_kernel(BcastDims d, int op, const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ Y,
                                                                      uint32_t n, bool vec)
{
   griddep_launch_dependents();
   griddep_wait(A, B);
   const uint32_t nthreads = gridDim.x * blockDim.x;
   for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += nthreads * 4) {
      uint32_t c[4], rem = i, ao = 0, bo = 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
         if (k < 3) rem = d.shape[k].divmod(rem, c[k]);
         else c[k] = rem;
         if (!A_DENSE) ao += c[k] * d.a[k];
         if (!B_DENSE) bo += c[k] * d.b[k];
      }
      const bool full = vec && i + 4 <= n;
      float a[4], b[4], y[4];
      if (A_DENSE && full) {
         const float4 v = *reinterpret_cast<const float4 *>(A + i);
         a[0] = v.x, a[1] = v.y, a[2] = v.z, a[3] = v.w;
      }
      if (B_DENSE && full) {
         const float4 v = *reinterpret_cast<const float4 *>(B + i);
         b[0] = v.x, b[1] = v.y, b[2] = v.z, b[3] = v.w;
      }
      if (full && c[0] + 4 <= d.shape[0].d && (A_DENSE || d.a[0] == 0) && (B_DENSE || d.b[0] == 0)) {
         // one run of the innermost dimension, along which the broadcast operand stands still
         if (!A_DENSE) a[0] = a[1] = a[2] = a[3] = A[ao];
         if (!B_DENSE) b[0] = b[1] = b[2] = b[3] = B[bo];
      } else {
#pragma unroll
         for (int j = 0; j < 4; j++) {
            if (i + j >= n) break;
            if (A_DENSE ? !full : true) a[j] = A[A_DENSE ? i + j : ao];
            if (B_DENSE ? !full : true) b[j] = B[B_DENSE ? i + j : bo];
            // the next coordinate: one step along the innermost dimension, carried outwards
            ao += d.a[0], bo += d.b[0];
            c[0]++;
#pragma unroll
            for (int k = 0; k < 3; k++) {
               if (c[k] != d.shape[k].d) break;
               ao += d.a[k + 1] - c[k] * d.a[k];
               bo += d.b[k + 1] - c[k] * d.b[k];
               c[k] = 0;
               c[k + 1]++;
            }
         }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) y[j] = binary_apply(op, a[j], b[j]);
      if (full) {
         *reinterpret_cast<float4 *>(Y + i) = make_float4(y[0], y[1], y[2], y[3]);
      } else {
#pragma unroll
         for (int j = 0; j < 4; j++)
            if (i + j < n) Y[i + j] = y[j];
      }
   }
}

// The same without the limits of 2^31 outputs and 32-bit offsets: the output index is split into up to four coordinates; a broadcast dimension of an
// operand has stride 0.
__global__ void binary_bcast_large_f32_kernel(sofie_binary_desc d, const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ Y, size_t n)
{
   griddep_launch_dependents();
   griddep_wait(A, B);
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
      size_t rem = i, ao = 0, bo = 0;
#pragma unroll
      for (int k = 3; k >= 0; k--) {
         const size_t c = rem % (size_t)d.shape[k];
         rem /= (size_t)d.shape[k];
         ao += c * (size_t)d.a_stride[k];
         bo += c * (size_t)d.b_stride[k];
      }
      Y[i] = binary_apply(d.op, A[ao], B[bo]);
   }
}

// y = ((x - mean[c]) * scale[c]) + bias[c], optional Relu; the three steps are separate roundings as
// in the emitted scopy / saxpy / multiply / saxpy sequence (ROperator_BatchNormalization.hxx:200-226).
__device__ __forceinline__ float batchnorm_apply(float x, float mean, float scale, float bias, int relu)
{
   const float y = __fadd_rn(__fmul_rn(__fsub_rn(x, mean), scale), bias);
   return relu ? relu_ref(y) : y;
}

// Four consecutive elements per thread. `inner` elements in a row share a channel (HW, or 1 with the channels innermost). Measured
// on [512,16,64,64]: 116 us with 64-bit divisions per element, 42 us here.
__global__ void __launch_bounds__(kActThreads) batchnorm_f32_kernel(FastDiv inner, FastDiv channels, const float *__restrict__ X, const float *__restrict__ scale,
                                                                   const float *__restrict__ bias, const float *__restrict__ mean, float *__restrict__ Y, uint32_t n, int relu, bool vec)
{
   griddep_launch_dependents();
   griddep_wait(X, scale, bias, mean);
   const uint32_t nthreads = gridDim.x * blockDim.x;
   for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += nthreads * 4) {
      uint32_t in, c;
      channels.divmod(inner.divmod(i, in), c);
      const bool full = vec && i + 4 <= n;
      float x[4] = {};
      if (full) {
         const float4 v = *reinterpret_cast<const float4 *>(X + i);
         x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
      }
      if (full && in + 4 <= inner.d) {
         const float m = mean[c], s = scale[c], b = bias[c];
#pragma unroll
         for (int j = 0; j < 4; j++) x[j] = batchnorm_apply(x[j], m, s, b, relu);
      } else {
#pragma unroll
         for (int j = 0; j < 4; j++) {
            if (i + j >= n) break;
            if (!full) x[j] = X[i + j];
            x[j] = batchnorm_apply(x[j], mean[c], scale[c], bias[c], relu);
            if (++in == inner.d) {
               in = 0;
               if (++c == channels.d) c = 0;
            }
         }
      }
      if (full) {
         *reinterpret_cast<float4 *>(Y + i) = make_float4(x[0], x[1], x[2], x[3]);
      } else {
#pragma unroll
         for (int j = 0; j < 4; j++)
            if (i + j < n) Y[i + j] = x[j];
      }
   }
}
__global__ void batchnorm_large_f32_kernel(sofie_batchnorm_desc d, const float *__restrict__ X, const float *__restrict__ scale,
                                           const float *__restrict__ bias, const float *__restrict__ mean, float *__restrict__ Y, size_t n)
{
   griddep_launch_dependents();
   griddep_wait(X, scale, bias, mean);
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
      const int c = d.layout == SOFIE_LAYOUT_NHWC ? (int)(i % (size_t)d.C) : (int)((i / (size_t)d.HW) % (size_t)d.C);
      Y[i] = batchnorm_apply(X[i], mean[c], scale[c], bias[c], d.relu);
   }
}

// floats per access: as wide as all of the pointers allow
inline int access_width(std::initializer_list<const void *> pointers)
{
   uintptr_t bits = 0;
   for (const void *p : pointers) bits |= reinterpret_cast<uintptr_t>(p);
   return (bits & 31) == 0 ? 8 : ((bits & 15) == 0 ? 4 : 1);
}
inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

} // namespace
} // namespace sofie

using namespace sofie;

extern "C" int sofie_cuda_unary_f32(void *stream, int32_t op, float alpha, const float *X, float *Y, size_t n)
{
   SOFIE_REQUIRE(op >= SOFIE_UNARY_SIGMOID && op <= SOFIE_UNARY_SIN, "unknown unary operator %d", op);
   if (n == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(X && Y, "NULL tensor");
   const bool vec = aligned16(X) && aligned16(Y);
   const UnaryKernel kernel = unary_kernel(op, std::make_integer_sequence<int, SOFIE_UNARY_SIN + 1>());
   SOFIE_CUDA_TRY(launch_dependent(kernel, dim3(act_grid(vec ? n / 4 + 1 : n)), dim3(kActThreads), 0, as_stream(stream), alpha, X, Y, n, vec));
   return SOFIE_CUDA_OK;
}

extern "C" int sofie_cuda_binary_f32(void *stream, const sofie_binary_desc *d, const float *A, const float *B, float *Y)
{
   SOFIE_REQUIRE(d != nullptr, "NULL descriptor");
   SOFIE_REQUIRE(d->op >= SOFIE_BINARY_ADD && d->op <= SOFIE_BINARY_DIV, "unknown binary operator %d", d->op);
   size_t n = 1;
   bool same = true;
   size_t dense = 1;
   for (int k = 3; k >= 0; k--) {
      SOFIE_REQUIRE(d->shape[k] >= 0 && d->a_stride[k] >= 0 && d->b_stride[k] >= 0, "negative extent or stride");
      if (d->shape[k] > 1) same = same && (size_t)d->a_stride[k] == dense && (size_t)d->b_stride[k] == dense;
      dense *= (size_t)d->shape[k];
      n *= (size_t)d->shape[k];
   }
   if (n == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(A && B && Y, "NULL tensor");
   cudaStream_t s = as_stream(stream);
   if (same) {
      const int vec = access_width({A, B, Y});
      SOFIE_CUDA_TRY(launch_dependent(binary_same_f32_kernel, dim3(act_grid(n / vec + 1)), dim3(kActThreads), 0, s, d->op, A, B, Y, n, vec));
      return SOFIE_CUDA_OK;
   }
   // coordinates of the outputs and offsets of the operands in 32 bits, where they fit: an operand may be a view of something larger
   uint64_t last_a = 0, last_b = 0;
   bool narrow = n < (size_t(1) << 31) - 4096 * 1024;
   for (int k = 0; k < 4; k++) {
      if (d->shape[k] == 1) continue;
      narrow = narrow && d->a_stride[k] <= UINT32_MAX && d->b_stride[k] <= UINT32_MAX;
      last_a += (uint64_t)(d->shape[k] - 1) * (uint64_t)d->a_stride[k];
      last_b += (uint64_t)(d->shape[k] - 1) * (uint64_t)d->b_stride[k];
   }
   if (!narrow || last_a > UINT32_MAX || last_b > UINT32_MAX) {
      SOFIE_CUDA_TRY(launch_dependent(binary_bcast_large_f32_kernel, dim3(act_grid(n)), dim3(kActThreads), 0, s, *d, A, B, Y, n));
      return SOFIE_CUDA_OK;
   }
   // merge dimensions, innermost first: the next one continues the current one where both operands' strides do
   BcastDims b;
   int64_t shape[4] = {1, 1, 1, 1}, as[4] = {}, bs[4] = {};
   int dims = 0;
   for (int k = 3; k >= 0; k--) {
      if (d->shape[k] == 1) continue;
      if (dims && d->a_stride[k] == as[dims - 1] * shape[dims - 1] && d->b_stride[k] == bs[dims - 1] * shape[dims - 1]) {
         shape[dims - 1] *= d->shape[k];
         continue;
      }
      shape[dims] = d->shape[k], as[dims] = d->a_stride[k], bs[dims] = d->b_stride[k];
      dims++;
   }
   bool a_dense = true, b_dense = true;
   int64_t run = 1;
   for (int k = 0; k < 4; k++) {
      b.shape[k] = FastDiv((uint32_t)shape[k]);
      b.a[k] = (uint32_t)as[k], b.b[k] = (uint32_t)bs[k];
      if (k < dims) a_dense = a_dense && as[k] == run, b_dense = b_dense && bs[k] == run;
      run *= shape[k];
   }
   const bool vec = aligned16(Y) && (!a_dense || aligned16(A)) && (!b_dense || aligned16(B));
   auto kernel = a_dense ? binary_bcast_f32_kernel<true, false> : (b_dense ? binary_bcast_f32_kernel<false, true> : binary_bcast_f32_kernel<false, false>);
   SOFIE_CUDA_TRY(launch_dependent(kernel, dim3(act_grid(n / 4 + 1)), dim3(kActThreads), 0, s, b, d->op, A, B, Y, (uint32_t)n, vec));
   return SOFIE_CUDA_OK;
}

extern "C" int sofie_cuda_batchnorm_f32(void *stream, const sofie_batchnorm_desc *d, const float *X, const float *scale, const float *bias,
                                        const float *mean, float *Y)
{
   SOFIE_REQUIRE(d != nullptr, "NULL descriptor");
   SOFIE_REQUIRE(d->N >= 0 && d->C > 0 && d->HW > 0, "bad BatchNormalization shape %d x %d x %d", d->N, d->C, d->HW);
   SOFIE_REQUIRE(d->layout == SOFIE_LAYOUT_NCHW || d->layout == SOFIE_LAYOUT_NHWC, "unknown layout");
   const size_t n = (size_t)d->N * d->C * d->HW;
   if (n == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(X && Y && scale && bias && mean, "NULL tensor");
   if (n >= (size_t(1) << 31) - 4096 * 1024) {
      SOFIE_CUDA_TRY(launch_dependent(batchnorm_large_f32_kernel, dim3(act_grid(n)), dim3(kActThreads), 0, as_stream(stream), *d, X, scale, bias, mean, Y, n));
      return SOFIE_CUDA_OK;
   }
   const FastDiv inner(d->layout == SOFIE_LAYOUT_NHWC ? 1 : (uint32_t)d->HW), channels((uint32_t)d->C);
   SOFIE_CUDA_TRY(launch_dependent(batchnorm_f32_kernel, dim3(act_grid(n / 4 + 1)), dim3(kActThreads), 0, as_stream(stream), inner, channels, X, scale, bias, mean, Y,
                                   (uint32_t)n, d->relu, aligned16(X) && aligned16(Y)));
   return SOFIE_CUDA_OK;
}
