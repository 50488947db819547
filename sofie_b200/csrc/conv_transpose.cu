// ConvTranspose 2-D (group 1), the gather form: an output pixel (oh, ow) collects, for every filter tap
// (r, s), the input pixel ih = (oh + pad - r * dil) / stride when that division is exact and in range.
// Nothing like the reference's per-image filter GEMM + col2im scatter (ROperator_ConvTranspose.icc:364-474,
// SOFIE_common.hxx:576-620) is materialised: no xcol buffer, no zero fill, no second pass for the bias.
// A thread owns one output pixel of four consecutive output channels, so that an input value is read
// once for four filters; threads of a warp walk ow, which makes the input reads contiguous at stride 1.
// X [N,C,H,W], W [C,Cout,kH,kW] (the ONNX layout), Y [N,Cout,oH,oW], fp32 FMA, taps in (r, s, ic) order.
#include "common.cuh"

#include <algorithm>
#include <type_traits>

namespace sofie {
namespace {

constexpr int kOcPerThread = 4;
constexpr int kThreads = 256;

// grid-stride launch: at most eight waves of blocks
inline int grid_for(size_t work_items)
{
   size_t blocks = ceil_div<size_t>(work_items, kThreads);
   const size_t cap = size_t(kNumSMs) * 8;
   return (int)(blocks > cap ? cap : (blocks == 0 ? 1 : blocks));
}

__global__ void __launch_bounds__(kThreads)
conv_transpose2d_f32_kernel(sofie_conv_transpose2d_desc d, int oH, int oW, size_t total, const float *__restrict__ X,
                            const float *__restrict__ Wt, const float *__restrict__ bias, float *__restrict__ Y)
{
   const int ocg = (d.Cout + kOcPerThread - 1) / kOcPerThread;
   const size_t in_hw = (size_t)d.H * d.W, out_hw = (size_t)oH * oW, taps = (size_t)d.kH * d.kW;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
      const int ow = (int)(i % oW);
      size_t t = i / oW;
      const int oh = (int)(t % oH);
      t /= oH;
      const int oc0 = (int)(t % ocg) * kOcPerThread;
      const int n = (int)(t / ocg);
      float acc[kOcPerThread] = {0.f, 0.f, 0.f, 0.f};
      const float *x = X + (size_t)n * d.C * in_hw;
      for (int r = 0; r < d.kH; r++) {
         const int th = oh + d.pad_h - r * d.dil_h;
         if (th < 0 || th % d.stride_h) continue;
         const int ih = th / d.stride_h;
         if (ih >= d.H) continue;
         for (int s = 0; s < d.kW; s++) {
            const int tw = ow + d.pad_w - s * d.dil_w;
            if (tw < 0 || tw % d.stride_w) continue;
            const int iw = tw / d.stride_w;
            if (iw >= d.W) continue;
            const float *xp = x + (size_t)ih * d.W + iw;
            const float *wp = Wt + (size_t)oc0 * taps + (size_t)r * d.kW + s;
            for (int ic = 0; ic < d.C; ic++) {
               const float v = __ldg(xp + (size_t)ic * in_hw);
               const float *w = wp + (size_t)ic * d.Cout * taps;
#pragma unroll
               for (int j = 0; j < kOcPerThread; j++)
                  if (oc0 + j < d.Cout) acc[j] = fmaf(v, __ldg(w + (size_t)j * taps), acc[j]);
            }
         }
      }
#pragma unroll
      for (int j = 0; j < kOcPerThread; j++) {
         if (oc0 + j < d.Cout) {
            float v = acc[j] + (bias ? __ldg(bias + oc0 + j) : 0.f);
            if (d.relu) v = relu_ref(v);
            Y[((size_t)n * d.Cout + oc0 + j) * out_hw + (size_t)oh * oW + ow] = v;
         }
      }
   }
}

// ---- the direct form with the filters in shared memory ------------------------------------------------------------
// A thread owns one output pixel and OC output channels. Threads are numbered by the column's residue modulo the stride before the column,
// so that a warp's pixels share their taps (no divergence) and read neighbouring input pixels; the filters of the block's channels are
// staged [channel][tap][OC], CK input channels at a time, and read as 16-byte broadcasts. A channel's product goes to one of four sums by the
// channel's number modulo four (those past the last multiple of four to the first): chains a quarter as long, whose error against float64 is about half of one chain's.
// Against one thread per pixel and four channels with the filters from global memory: 32 -> 16 channels, 2 x 2 / 2 on 12 x 12, 1 / 64 / 1024 images 25 -> 9,
// 55 -> 14, 785 -> 138 us; 16 -> 16, 3 x 3 / 1 on 64 x 64, 16 images 104 -> 27; error against float64 1.04e-7 -> 7.0e-8 and 2.1e-7 -> 1.2e-7. The product form
// below is nearer to float64 still where it takes the tensor cores' three-part kernel, and stays where the caller asks for it.
// At stride one with one input channel (or two and one tap) there is nothing to share, and as long as one wave of threads does, the pixel's thread with
// the filters from global memory is there first: 8 x 8, one channel, 7 x 7 taps 18.4 us against 21.8, 3 x 3 5.4 against 6.1. Two channels and 3 x 3: 6.8
// against 6.1; 64 images of 28 x 28, 1 -> 16 channels, 3 x 3: 17.4 against 13.0.
// EXACT: sums in 64 bits, in one chain, for layers of few products an output (launch_few_products); fewer channels a thread where threads are few. With the divisions by the strides as multiplications it takes 0.81 to 0.98
// of the time that sums in 32 bits took with divisions, by the number of blocks; those take 0.93 of it on 900 layers of more products. Four chains in 64 bits: 1.15 of one's time.
constexpr int kPhaseThreads = 128;
constexpr int kPhaseFilterBytes = 32 * 1024;
template <int OC, bool EXACT>
__global__ void __launch_bounds__(kPhaseThreads)
conv_transpose_phase_kernel(sofie_conv_transpose2d_desc d, int oW, FastDiv columns, FastDiv strides_h, FastDiv strides_w, FastDiv rows, uint32_t positions, int CK, const float *__restrict__ X,
                            const float *__restrict__ Wt, const float *__restrict__ bias, float *__restrict__ Y)
{
   using T = std::conditional_t<EXACT, double, float>;
   constexpr int CHAINS = EXACT ? 1 : 4;
   extern __shared__ __align__(16) unsigned char phase_smem[];
   T *filters = reinterpret_cast<T *>(phase_smem);
   const size_t in_hw = (size_t)d.H * d.W, out_hw = (size_t)rows.d * oW;
   const int taps = d.kH * d.kW, oc0 = blockIdx.y * OC;
   // (n, oh, residue, column) of the thread, in 32 bits (more positions than that are the other kernel's)
   uint32_t t = blockIdx.x * (uint32_t)kPhaseThreads + threadIdx.x, column, phase, row;
   bool active = t < positions;
   const size_t n = rows.divmod(strides_w.divmod(columns.divmod(t, column), phase), row);
   const int ow = (int)column * d.stride_w + (int)phase, oh = (int)row;
   active = active && ow < oW;
   T acc[CHAINS][OC];
#pragma unroll
   for (int k = 0; k < CHAINS; k++)
#pragma unroll
      for (int j = 0; j < OC; j++) acc[k][j] = 0;
   const float *x = X + (active ? n : 0) * d.C * in_hw;
   for (int c0 = 0; c0 < d.C; c0 += CK) {
      const int ck = min(CK, d.C - c0);
      __syncthreads(); // the filters before these are no longer read
      for (int i = threadIdx.x; i < ck * taps * OC; i += kPhaseThreads) {
         const unsigned j = i % OC, tap = (unsigned)i / OC % taps, c = (unsigned)i / OC / taps;
         filters[i] = oc0 + (int)j < d.Cout ? __ldg(Wt + ((size_t)(c0 + c) * d.Cout + oc0 + j) * taps + tap) : 0.f;
      }
      __syncthreads();
      if (!active) continue;
      for (int r = 0; r < d.kH; r++) {
         const int th = oh + d.pad_h - r * d.dil_h;
         if (th < 0) continue;
         uint32_t rest;
         const int ih = (int)strides_h.divmod((uint32_t)th, rest);
         if (rest || ih >= d.H) continue;
         for (int s = 0; s < d.kW; s++) {
            const int tw = ow + d.pad_w - s * d.dil_w;
            if (tw < 0) continue;
            const int iw = (int)strides_w.divmod((uint32_t)tw, rest);
            if (rest || iw >= d.W) continue;
            const float *xp = x + (size_t)c0 * in_hw + (size_t)ih * d.W + iw;
            const T *wp = filters + (r * d.kW + s) * OC;
            auto add = [&](float v, const T *w, T(&a)[OC]) {
               if constexpr (EXACT) {
#pragma unroll
                  for (int j = 0; j < OC; j += 2) {
                     const double2 f = *reinterpret_cast<const double2 *>(w + j);
                     a[j] = fma((double)v, f.x, a[j]);
                     a[j + 1] = fma((double)v, f.y, a[j + 1]);
                  }
               } else {
#pragma unroll
                  for (int j = 0; j < OC; j += 4) {
                     const float4 f = *reinterpret_cast<const float4 *>(w + j);
                     a[j] = fmaf(v, f.x, a[j]);
                     a[j + 1] = fmaf(v, f.y, a[j + 1]);
                     a[j + 2] = fmaf(v, f.z, a[j + 2]);
                     a[j + 3] = fmaf(v, f.w, a[j + 3]);
                  }
               }
            };
            int c = 0;
            for (; c + 16 <= ck; c += 16) { // sixteen loads under way
               float v[16];
#pragma unroll
               for (int k = 0; k < 16; k++) v[k] = __ldg(xp + (size_t)(c + k) * in_hw);
#pragma unroll
               for (int k = 0; k < 16; k++) add(v[k], wp + (c + k) * taps * OC, acc[k % CHAINS]);
            }
            for (; c + 4 <= ck; c += 4) {
               float v[4];
#pragma unroll
               for (int k = 0; k < 4; k++) v[k] = __ldg(xp + (size_t)(c + k) * in_hw);
#pragma unroll
               for (int k = 0; k < 4; k++) add(v[k], wp + (c + k) * taps * OC, acc[k % CHAINS]);
            }
            for (; c < ck; c++) add(__ldg(xp + (size_t)c * in_hw), wp + c * taps * OC, acc[0]);
         }
      }
   }
   if (!active) return;
#pragma unroll
   for (int j = 0; j < OC; j++) {
      if (oc0 + j < d.Cout) {
         float v;
         if constexpr (EXACT) v = (float)(acc[0][j] + (bias ? (double)__ldg(bias + oc0 + j) : 0.0));
         else v = ((acc[0][j] + acc[1][j]) + (acc[2][j] + acc[3][j])) + (bias ? __ldg(bias + oc0 + j) : 0.f);
         if (d.relu) v = relu_ref(v);
         Y[(n * d.Cout + oc0 + j) * out_hw + (size_t)oh * oW + ow] = v;
      }
   }
}

template <int OC, bool EXACT>
int launch_phase(cudaStream_t s, const sofie_conv_transpose2d_desc &d, int oH, int oW, const float *X, const float *W, const float *bias, float *Y)
{
   const int columns = ceil_div(oW, d.stride_w);
   const size_t positions = (size_t)d.N * oH * d.stride_w * columns, channel = (size_t)d.kH * d.kW * OC * (EXACT ? sizeof(double) : sizeof(float));
   const int fit = (int)(kPhaseFilterBytes / channel), CK = fit >= d.C ? d.C : fit / 4 * 4;
   const size_t blocks = ceil_div<size_t>(positions, kPhaseThreads);
   if (CK < 1 || positions > 0x7FFFFFFFu || ceil_div(d.Cout, OC) > 65535) return -1;
   conv_transpose_phase_kernel<OC, EXACT><<<dim3((unsigned)blocks, ceil_div(d.Cout, OC)), kPhaseThreads, CK * channel, s>>>(d, oW, FastDiv(columns), FastDiv(d.stride_h), FastDiv(d.stride_w), FastDiv(oH), (uint32_t)positions, CK, X,
                                                                                                                                           W, bias, Y);
   SOFIE_LAUNCH_CHECK("conv_transpose_phase_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}
// Channels of a thread where sums are in 64 bits: as many as leave two blocks an SM, down to two
int phase_channels(const sofie_conv_transpose2d_desc &d, int oH, int oW)
{
   const size_t blocks = ceil_div<size_t>((size_t)d.N * oH * d.stride_w * ceil_div(oW, d.stride_w), kPhaseThreads);
   for (int OC = d.Cout <= 4 ? 4 : 8; OC > 2; OC /= 2)
      if (blocks * ceil_div(d.Cout, OC) >= 2 * kNumSMs) return OC;
   return d.Cout <= 4 ? 2 : 4;
}
int launch_phase_exact(cudaStream_t s, const sofie_conv_transpose2d_desc &d, int oH, int oW, const float *X, const float *W, const float *bias, float *Y)
{
   const int OC = phase_channels(d, oH, oW);
   if (OC == 2) return launch_phase<2, true>(s, d, oH, oW, X, W, bias, Y);
   if (OC == 4) return launch_phase<4, true>(s, d, oH, oW, X, W, bias, Y);
   return launch_phase<8, true>(s, d, oH, oW, X, W, bias, Y);
}

int launch_direct(cudaStream_t s, const sofie_conv_transpose2d_desc &d, int oH, int oW, const float *X, const float *W, const float *bias, float *Y)
{
   const size_t total = (size_t)d.N * ((d.Cout + kOcPerThread - 1) / kOcPerThread) * oH * oW;
   const bool alone = d.stride_h == 1 && d.stride_w == 1 && d.C * min(d.kH * d.kW, 2) <= 2 && total <= 1u << 17;
   const int rc = alone ? -1 : d.Cout <= 4 ? launch_phase<4, false>(s, d, oH, oW, X, W, bias, Y) : launch_phase<8, false>(s, d, oH, oW, X, W, bias, Y);
   if (rc >= 0) return rc;
   // also: filters of which not four channels fit beside one another, 2^31 outputs or more
   conv_transpose2d_f32_kernel<<<grid_for(total), kThreads, 0, s>>>(d, oH, oW, total, X, W, bias, Y);
   SOFIE_LAUNCH_CHECK("conv_transpose2d_f32_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// ---- few products an output: one launch, sums in 64 bits ----------------------------------------------------------
// The product form below is four launches and writes every tap's product to memory and reads it back; where an output has few products those are its time, and the
// direct form above waits for one channel's filters and inputs after the other's. Here a block owns a band of output rows of one image and OC output channels: the band's
// inputs and the filters are converted to double once, on their way into shared memory, and a thread sums four channels of PX outputs in double, so that the result is the exact
// sum rounded once (error against float64 2.5e-8; 3.5e-8 to 1.3e-7 the product form, 4.3e-8 to 5.5e-8 the direct one). A warp's outputs share their phase (row and column
// modulo the strides) and so their taps; OC / 4 neighbouring lanes share an output's inputs. Or the direct form runs, its sums in 64 bits too (launch_few_products).
// What bounds it: round trips at sixteen warps an SM, to L2 while a block stages and to shared memory while it sums; no pipe is busy, at 64 images or at 1024 (issue slots 31 and 29 %, fp64
// 15 and 16 %, shared memory 17 and 23 %). 32 -> 16 channels, 2 x 2 / 2 on 12 x 12, 1 / 64 / 1024 images: 13.6 -> 5.3, 16.3 -> 10.6, 103 -> 85 us against
// the product form; 16 -> 3, 3 x 3 / 2 on 24 x 24: 12.9 -> 6.4, 21.5 -> 13.9, 184 -> 117. Its channels in registers two or four at a time: the same or slower (96, 127 at 1024).
constexpr int kSumThreads = 256;
constexpr int kSumBytes = 96 * 1024; // of shared memory: two blocks an SM
struct SumGeom {
   sofie_conv_transpose2d_desc d;
   int oH, oW, bands, steps, lines; // bands of an image, steps (times the stride: output rows) of a band, input rows it may read
};

__host__ __device__ inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((b - 1 - a) / b); }

template <int OC, int PX>
__global__ void __launch_bounds__(kSumThreads, 2)
conv_transpose_sum_kernel(SumGeom g, FastDiv bands, FastDiv columns, FastDiv taps, FastDiv phase_units, FastDiv phase_columns, int line, const float *__restrict__ X, const float *__restrict__ Wt,
                          const float *__restrict__ bias, float *__restrict__ Y)
{
   extern __shared__ __align__(16) double staged[];
   const sofie_conv_transpose2d_desc &d = g.d;
   griddep_launch_dependents();
   griddep_wait(X, Wt, bias);
   const int oc0 = blockIdx.y * OC, outs = min(OC, d.Cout - oc0);
   // [channel][tap][OC], [channel][row][column]; of every filter row (column) the phase that it is a tap of and how far below the output's step its input lies
   double *filters = staged, *inputs = staged + d.C * (int)taps.d * OC;
   int2 *tap_rows = reinterpret_cast<int2 *>(inputs + d.C * line), *tap_columns = tap_rows + d.kH;
   for (int i = threadIdx.x; i < d.kH + d.kW; i += kSumThreads) {
      const bool column = i >= d.kH;
      const int stride = column ? d.stride_w : d.stride_h, at = column ? (i - d.kH) * d.dil_w - d.pad_w : i * d.dil_h - d.pad_h, step = floor_div(at, stride);
      tap_rows[i] = make_int2(at - step * stride, -step);
   }
   uint32_t band;
   const uint32_t n = bands.divmod(blockIdx.x, band);
   const int oh0 = (int)band * g.steps * d.stride_h, rows = min(g.steps * d.stride_h, g.oH - oh0);
   // input rows that an output row of the band has a tap on
   const int first = max(0, floor_div(oh0 + d.pad_h - (d.kH - 1) * d.dil_h, d.stride_h)), last = min(d.H - 1, (oh0 + rows - 1 + d.pad_h) / d.stride_h);
   const int lines = max(0, last - first + 1);
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   // half of the warps fetch the filters, half the inputs: a warp walks the consecutive values of every fourth input channel, eight loads under way
   auto stage = [&](int span, auto source, auto store) {
      int c = warp & 3, base = 0;
      auto next = [&] {
         base += 32;
         if (base >= span) base = 0, c += 4;
      };
      while (c < d.C) {
         const int c0 = c, base0 = base;
         float v[8];
#pragma unroll
         for (int k = 0; k < 8; k++, next()) v[k] = c < d.C && base + lane < span ? load_dependent(source(c) + base + lane) : 0.f;
         c = c0, base = base0;
#pragma unroll
         for (int k = 0; k < 8; k++, next())
            if (c < d.C && base + lane < span) store(c, base + lane, (double)v[k]);
      }
   };
   if (warp < 4) {
      stage(outs * (int)taps.d, [&](int c) { return Wt + ((size_t)c * d.Cout + oc0) * taps.d; }, // the block's filters of an input channel are consecutive
            [&](int c, int e, double v) {
               uint32_t tap;
               const uint32_t j = taps.divmod((uint32_t)e, tap);
               filters[(c * taps.d + tap) * OC + j] = v;
            });
      if (outs < OC)
         for (int i = threadIdx.x; i < d.C * (int)taps.d; i += kSumThreads / 2)
            for (int j = outs; j < OC; j++) filters[i * OC + j] = 0.0;
   } else if (lines > 0) {
      // a channel's rows are consecutive in X and here
      const float *x = X + ((size_t)n * d.C * d.H + first) * d.W;
      stage(lines * d.W, [&](int c) { return x + (size_t)c * d.H * d.W; }, [&](int c, int e, double v) { inputs[c * line + e] = v; });
   }
   __syncthreads();
   constexpr int LG = OC / 4, PXW = 32 / LG * PX; // lanes that share an output's channels, positions of a warp
   const int oc = lane % LG * 4, units = (int)phase_units.d;
   for (int u = warp; u < units * d.stride_h * d.stride_w; u += kSumThreads / 32) {
      uint32_t rw, in_phase;
      const int rh = (int)phase_columns.divmod(phase_units.divmod((uint32_t)u, in_phase), rw), i0 = (int)in_phase * PXW + lane / LG;
      int step_h[PX], step_w[PX]; // the output is in row stride * step + phase
      double acc[PX][4];
#pragma unroll
      for (int q = 0; q < PX; q++) {
         uint32_t column;
         step_h[q] = (int)band * g.steps + (int)columns.divmod((uint32_t)(i0 + q * (32 / LG)), column);
         step_w[q] = (int)column;
#pragma unroll
         for (int j = 0; j < 4; j++) acc[q][j] = 0.0;
      }
      for (int r = 0; r < d.kH; r++) {
         const int2 row = tap_rows[r];
         if (row.x != rh) continue;
         for (int s = 0; s < d.kW; s++) {
            const int2 across = tap_columns[s];
            if (across.x != (int)rw) continue;
            const double *w = filters + (r * d.kW + s) * OC + oc;
            const double *x[PX];
            bool in[PX];
            bool any = false;
#pragma unroll
            for (int q = 0; q < PX; q++) {
               const int ih = step_h[q] + row.y, iw = step_w[q] + across.y;
               in[q] = ih >= first && ih <= last && iw >= 0 && iw < d.W;
               x[q] = inputs + (in[q] ? (ih - first) * d.W + iw : 0);
               any = any || in[q];
            }
            if (!any) continue;
#pragma unroll 4
            for (int c = 0; c < d.C; c++) {
               const double2 f0 = *reinterpret_cast<const double2 *>(w), f1 = *reinterpret_cast<const double2 *>(w + 2);
               w += taps.d * OC;
#pragma unroll
               for (int q = 0; q < PX; q++) {
                  const double v = *x[q];
                  x[q] += line;
                  if (in[q]) { // a tap outside is no product: an infinite weight does not count there
                     acc[q][0] = fma(v, f0.x, acc[q][0]);
                     acc[q][1] = fma(v, f0.y, acc[q][1]);
                     acc[q][2] = fma(v, f1.x, acc[q][2]);
                     acc[q][3] = fma(v, f1.y, acc[q][3]);
                  }
               }
            }
         }
      }
#pragma unroll
      for (int q = 0; q < PX; q++) {
         const int oh = d.stride_h * step_h[q] + rh, ow = d.stride_w * step_w[q] + (int)rw;
         if (oh >= oh0 + rows || ow >= g.oW) continue;
#pragma unroll
         for (int j = 0; j < 4; j++) {
            if (oc + j < outs) {
               float v = (float)(acc[q][j] + (bias ? (double)__ldg(bias + oc0 + oc + j) : 0.0));
               if (d.relu) v = relu_ref(v);
               Y[(((size_t)n * d.Cout + oc0 + oc + j) * g.oH + oh) * g.oW + ow] = v;
            }
         }
      }
   }
}

// How the kernel would cut a layer up; fits: the filters and one row of outputs' inputs do in shared memory
struct SumPlan {
   bool fits = false;
   int OC, PX, per, columns, halo, bands, groups;
   size_t filters, row; // bytes: the filters, an input row of all channels
};

SumPlan plan_sum(const sofie_conv_transpose2d_desc &d, int oH, int oW)
{
   SumPlan p;
   p.OC = d.Cout <= 4 ? 4 : d.Cout <= 8 ? 8 : 16;
   p.groups = ceil_div(d.Cout, p.OC), p.columns = ceil_div(oW, d.stride_w), p.halo = ceil_div((d.kH - 1) * d.dil_h, d.stride_h) + 1;
   p.filters = (size_t)d.C * d.kH * d.kW * p.OC * sizeof(double), p.row = (size_t)d.C * d.W * sizeof(double);
   if (p.groups > 65535 || p.filters + p.row * (1 + p.halo) > kSumBytes || d.kH + d.kW > 1024 || (long long)d.kH * d.dil_h > 1 << 20 || (long long)d.pad_h + oH > 1 << 28 || (long long)d.pad_w + oW > 1 << 28) return p;
   // Bands for two blocks an SM, as far as the rows go: what a block costs beside its sums is its start (64 images, 32 -> 16 channels: 4 bands an image 11.5 us, 6 15.1, 12 19.3, 2 16.6).
   // Of the outputs a thread can take the most that leave every warp some.
   const int steps = ceil_div(oH, d.stride_h);
   const long long wanted = 2 * kNumSMs / ((long long)d.N * p.groups);
   p.per = ceil_div(steps, (int)(wanted < 1 ? 1 : (wanted > steps ? steps : wanted)));
   auto units = [&](int q) { return (long long)d.stride_h * d.stride_w * ceil_div((long long)p.per * p.columns, 128ll / p.OC * q); };
   p.PX = units(4) >= kSumThreads / 32 ? 4 : units(2) >= kSumThreads / 32 ? 2 : 1;
   const int fit = (int)((kSumBytes - p.filters) / p.row) - p.halo;
   if (p.per > fit) p.per = fit;
   p.bands = ceil_div(steps, p.per);
   p.fits = (long long)d.N * p.bands < 1ll << 31 && (long long)p.per * p.columns < 1 << 30;
   return p;
}

template <int OC, int PX>
int launch_sum(cudaStream_t s, const sofie_conv_transpose2d_desc &d, int oH, int oW, const SumPlan &p, const float *X, const float *W, const float *bias, float *Y)
{
   const SumGeom g = {d, oH, oW, p.bands, p.per, p.per + p.halo};
   const size_t smem = p.filters + p.row * g.lines + (d.kH + d.kW) * sizeof(int2);
   auto kern = conv_transpose_sum_kernel<OC, PX>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), (int)smem));
   SOFIE_CUDA_TRY(launch_dependent(kern, dim3((unsigned)(d.N * (long long)g.bands), p.groups), dim3(kSumThreads), smem, s, g, FastDiv(g.bands), FastDiv(p.columns), FastDiv(d.kH * d.kW), FastDiv(ceil_div(p.per * p.columns, 128 / OC * PX)),
                                   FastDiv(d.stride_w), g.lines * d.W, X, W, bias, Y));
   SOFIE_LAUNCH_CHECK("conv_transpose_sum_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// Layers of up to 48 products an output, counted without borders: sums in 64 bits, by the kernel above or by the direct form, whichever takes less time by an estimate. -1 where an output has more, where
// neither can, and (product_form) where the product form is the faster one.
int launch_few_products(cudaStream_t s, const sofie_conv_transpose2d_desc &d, int oH, int oW, bool product_form, const float *X, const float *W, const float *bias, float *Y)
{
   // 64 -> 32 channels, 2 x 2 / 2 (64 products) on 256 images of 8 x 8: 44 us here, 30 in the product form; 32 -> 16, 4 x 4 / 2 (128) on 64 of 16 x 16: 29 and 31; 16 -> 16, 3 x 3 / 1 (144) on
   // 64 of 64 x 64: 101 here, 84 in the direct form.
   if ((long long)d.C * d.kH * d.kW > 48ll * d.stride_h * d.stride_w || forced_engine() == SOFIE_ENGINE_TCGEN05) return -1;
   // Times in us, fitted to 8900 layers of 1 to 4096 images (to 13, 20 and 19 %): blocks beyond what is resident at a time count, the first round's round trips do not shrink. Many small images, few products and large
   // strides are the direct form's (1 x 1 images, 4 x 4 / 2, 2 -> 49 channels, 3899 of them 8.5 us against 167), longer sums this kernel's. Of 2500 other layers the choice takes 0.77 of the time of the direct form with sums in
   // 32 bits in the mean, 2.7 % of them above 1.2 (with this kernel for all of them 0.88, 20 % above 1.2, up to 28 times the time); against the product form 0.70, one of 172 above 1.2.
   const int taps = d.kH * d.kW;
   const double outputs = 1e-4 * d.N * d.Cout * oH * oW, products = std::min((double)taps / (d.stride_h * d.stride_w), (double)d.H * d.W * taps / ((double)oH * oW)) * d.C; // of an output
   const SumPlan p = plan_sum(d, oH, oW);
   double sum = 1e30;
   if (p.fits) {
      const double blocks = (double)d.N * p.bands * p.groups, rounds = std::max(1.0, blocks / (2 * kNumSMs));
      const double units = std::max(1.0, (double)d.stride_h * d.stride_w * ceil_div((long long)p.per * p.columns, 128ll / p.OC * p.PX) / (kSumThreads / 32)); // a warp's
      const double walk = ceil_div(d.C, 4) * std::max(ceil_div(taps * std::min(d.Cout, p.OC), 32), ceil_div(std::min(p.per + p.halo, d.H) * d.W, 32)) / 8.0;
      sum = 0.98 + rounds * (1.88 + 1.2 * walk + units * (0.042 * taps + 0.0196 * products * (p.PX + 1) + 0.097 * p.PX)) + 0.029 * outputs;
   }
   double phase;
   {
      const int OC = phase_channels(d, oH, oW);
      const double blocks = (double)ceil_div<size_t>((size_t)d.N * oH * d.stride_w * p.columns, kPhaseThreads) * ceil_div(d.Cout, OC), share = blocks / kNumSMs;
      const size_t channel = (size_t)taps * OC * sizeof(double);
      const int fit = (int)(kPhaseFilterBytes / channel), CK = fit >= d.C ? d.C : fit / 4 * 4;
      const double rounds = std::max(1.0, share / std::min<size_t>(12, 227 * 1024 / (CK * channel + 1024)));
      const double stage = (double)d.C * taps * OC / kPhaseThreads, tests = d.kH + (double)d.kH / d.stride_h * d.kW;
      const double trips = (double)ceil_div(d.kH, d.stride_h) * ceil_div(d.kW, d.stride_w) * (d.C / 16 + d.C % 16 / 4 + d.C % 4);
      phase = 2.82 + rounds * (0.868 * stage + 0.103 * tests + 0.069 * trips) + share * (0.107 + 0.0123 * stage + 0.0185 * tests + 0.0032 * products * OC) + 0.0115 * outputs;
      if (CK < 1) phase = 1e30;
   }
   const bool here = sum < phase;
   if (product_form) {
      const double pixels = 1e-5 * d.N * d.H * d.W, columns = (double)taps * d.Cout;
      if (std::min(sum, phase) >= 0.85 * (10.2 + pixels * (0.413 * d.C + 0.721 * columns + 0.00407 * columns * d.C) + 0.0313 * outputs)) return -1;
   }
   if (!here) return launch_phase_exact(s, d, oH, oW, X, W, bias, Y);
#define SOFIE_SUM(C, P) return launch_sum<C, P>(s, d, oH, oW, p, X, W, bias, Y)
#define SOFIE_SUM_OC(P) \
   if (p.OC == 4) SOFIE_SUM(4, P); \
   if (p.OC == 8) SOFIE_SUM(8, P); \
   SOFIE_SUM(16, P)
   if (p.PX == 1) { SOFIE_SUM_OC(1); }
   if (p.PX == 2) { SOFIE_SUM_OC(2); }
   SOFIE_SUM_OC(4);
#undef SOFIE_SUM_OC
#undef SOFIE_SUM
}

// ---- the product form: one GEMM over all images on the tensor cores, then a gather -------------------------------
// The reference computes, per image, filter^T [Cout*kH*kW, C] x image [C, H*W] with sgemm_ and scatters the columns
// into the output (col2im). Here the images are brought to channel-last once, so ALL of them are one K-major operand:
//     P [N*H*W, kH*kW*Cout] = Xt [N*H*W, C] x Wt [kH*kW*Cout, C]^T        (sofie_cuda_gemm_f32: tcgen05, 3xTF32)
// and an output pixel gathers its taps' products from P (the gather form of col2im: no atomics, no zero fill), adds the
// bias and applies Relu. Column order (tap, output channel) makes four output channels of a tap 16 contiguous bytes.
__global__ void conv_transpose_weights_kernel(const float *__restrict__ W, float *__restrict__ Wt, int C, int Cout, int taps)
{
   const size_t total = (size_t)C * Cout * taps;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
      const int ic = (int)(i % C);
      const size_t row = i / C; // (tap, co)
      const int co = (int)(row % Cout), tap = (int)(row / Cout);
      Wt[i] = __ldg(W + ((size_t)ic * Cout + co) * taps + tap);
   }
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads)
conv_transpose_gather_kernel(sofie_conv_transpose2d_desc d, int oH, int oW, size_t total, const float *__restrict__ P,
                             const float *__restrict__ bias, float *__restrict__ Y)
{
   const int ocg = (d.Cout + kOcPerThread - 1) / kOcPerThread;
   const size_t in_hw = (size_t)d.H * d.W, out_hw = (size_t)oH * oW;
   const size_t ncol = (size_t)d.kH * d.kW * d.Cout;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
      const int ow = (int)(i % oW);
      size_t t = i / oW;
      const int oh = (int)(t % oH);
      t /= oH;
      const int oc0 = (int)(t % ocg) * kOcPerThread;
      const int n = (int)(t / ocg);
      float acc[kOcPerThread] = {0.f, 0.f, 0.f, 0.f};
      for (int r = 0; r < d.kH; r++) {
         const int th = oh + d.pad_h - r * d.dil_h;
         if (th < 0 || th % d.stride_h) continue;
         const int ih = th / d.stride_h;
         if (ih >= d.H) continue;
         for (int s = 0; s < d.kW; s++) {
            const int tw = ow + d.pad_w - s * d.dil_w;
            if (tw < 0 || tw % d.stride_w) continue;
            const int iw = tw / d.stride_w;
            if (iw >= d.W) continue;
            const float *p = P + ((size_t)n * in_hw + (size_t)ih * d.W + iw) * ncol + (size_t)(r * d.kW + s) * d.Cout + oc0;
            if (VEC) {
               const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
               acc[0] += v.x;
               acc[1] += v.y;
               acc[2] += v.z;
               acc[3] += v.w;
            } else {
#pragma unroll
               for (int j = 0; j < kOcPerThread; j++)
                  if (oc0 + j < d.Cout) acc[j] += __ldg(p + j);
            }
         }
      }
#pragma unroll
      for (int j = 0; j < kOcPerThread; j++) {
         if (oc0 + j < d.Cout) {
            float v = acc[j] + (bias ? __ldg(bias + oc0 + j) : 0.f);
            if (d.relu) v = relu_ref(v);
            Y[((size_t)n * d.Cout + oc0 + j) * out_hw + (size_t)oh * oW + ow] = v;
         }
      }
   }
}

// shape checks shared by the two entry points; the output extent on success
int check_conv_transpose(const sofie_conv_transpose2d_desc *d, long &oH, long &oW)
{
   SOFIE_REQUIRE(d != nullptr, "NULL descriptor");
   SOFIE_REQUIRE(d->N >= 0 && d->C > 0 && d->H > 0 && d->W > 0 && d->Cout > 0 && d->kH > 0 && d->kW > 0, "bad ConvTranspose shape");
   SOFIE_REQUIRE(d->stride_h > 0 && d->stride_w > 0 && d->dil_h > 0 && d->dil_w > 0 && d->pad_h >= 0 && d->pad_w >= 0 &&
                    d->out_pad_h >= 0 && d->out_pad_w >= 0,
                 "bad ConvTranspose strides, dilations or pads");
   // output_padding only makes sense below the stride (ONNX); larger values would leave rows nothing writes to
   SOFIE_REQUIRE(d->out_pad_h < d->stride_h || d->out_pad_h < d->dil_h, "output_padding must be smaller than the stride or the dilation");
   SOFIE_REQUIRE(d->out_pad_w < d->stride_w || d->out_pad_w < d->dil_w, "output_padding must be smaller than the stride or the dilation");
   oH = (long)d->stride_h * (d->H - 1) + (long)d->dil_h * (d->kH - 1) + 1 + d->out_pad_h - 2L * d->pad_h;
   oW = (long)d->stride_w * (d->W - 1) + (long)d->dil_w * (d->kW - 1) + 1 + d->out_pad_w - 2L * d->pad_w;
   SOFIE_REQUIRE(oH > 0 && oW > 0 && oH < (1L << 30) && oW < (1L << 30), "ConvTranspose output would be empty");
   return SOFIE_CUDA_OK;
}

} // namespace
} // namespace sofie

using namespace sofie;

extern "C" size_t sofie_cuda_conv_transpose2d_f32_gemm_scratch(const sofie_conv_transpose2d_desc *d)
{
   return d ? sofie_conv_transpose2d_gemm_scratch_bytes(d) : 0;
}

extern "C" int sofie_cuda_conv_transpose2d_f32_gemm(void *stream, const sofie_conv_transpose2d_desc *d, const float *X, const float *W,
                                                    const float *bias, float *Y, void *scratch, size_t scratch_bytes)
{
   long oH, oW;
   const int rc = check_conv_transpose(d, oH, oW);
   if (rc) return rc;
   const size_t need = sofie_conv_transpose2d_gemm_scratch_bytes(d);
   if (need == 0) return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "this ConvTranspose shape is served by sofie_cuda_conv_transpose2d_f32 only");
   if (d->N == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(X && W && Y && scratch, "NULL tensor");
   SOFIE_REQUIRE(scratch_bytes >= need, "scratch of %zu bytes, %zu needed", scratch_bytes, need);
   SOFIE_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255) == 0, "scratch must be 256-byte aligned");
   cudaStream_t s = as_stream(stream);
   const int few = launch_few_products(s, *d, (int)oH, (int)oW, true, X, W, bias, Y);
   if (few >= 0) return few;
   const size_t pixels = (size_t)d->N * d->H * d->W;
   const int taps = d->kH * d->kW;
   float *Xt = static_cast<float *>(scratch);
   float *Wt = Xt + sofie_round_up_floats(pixels * d->C);
   float *P = Wt + sofie_round_up_floats((size_t)taps * d->Cout * d->C);
   int st = sofie_cuda_nchw_to_nhwc_f32(stream, X, Xt, d->N, d->C, d->H, d->W);
   if (st) return st;
   conv_transpose_weights_kernel<<<grid_for((size_t)taps * d->Cout * d->C), kThreads, 0, s>>>(W, Wt, d->C, d->Cout, taps);
   SOFIE_LAUNCH_CHECK("conv_transpose_weights_kernel");
   SOFIE_REQUIRE(pixels < (1u << 31) && (size_t)taps * d->Cout < (1u << 31), "ConvTranspose too large for the product form");
   const sofie_gemm_f32_desc g = {(int32_t)pixels, (int32_t)(taps * d->Cout), d->C, 0, 1, 1.f, 0.f, 0, 0};
   st = sofie_cuda_gemm_f32(stream, &g, Xt, Wt, nullptr, P); // records the engine that ran
   if (st) return st;
   const size_t total = (size_t)d->N * ((d->Cout + kOcPerThread - 1) / kOcPerThread) * oH * oW;
   if (d->Cout % 4 == 0)
      conv_transpose_gather_kernel<true><<<grid_for(total), kThreads, 0, s>>>(*d, (int)oH, (int)oW, total, P, bias, Y);
   else
      conv_transpose_gather_kernel<false><<<grid_for(total), kThreads, 0, s>>>(*d, (int)oH, (int)oW, total, P, bias, Y);
   SOFIE_LAUNCH_CHECK("conv_transpose_gather_kernel");
   return SOFIE_CUDA_OK;
}

extern "C" int sofie_cuda_conv_transpose2d_f32(void *stream, const sofie_conv_transpose2d_desc *d, const float *X, const float *W,
                                               const float *bias, float *Y)
{
   long oH, oW;
   const int rc = check_conv_transpose(d, oH, oW);
   if (rc) return rc;
   if (d->N == 0) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(X && W && Y, "NULL tensor");
   const int few = launch_few_products(as_stream(stream), *d, (int)oH, (int)oW, false, X, W, bias, Y);
   if (few >= 0) return few;
   return launch_direct(as_stream(stream), *d, (int)oH, (int)oW, X, W, bias, Y);
}
