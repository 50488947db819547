// CUDA-core contraction kernels. They serve every shape the tensor-core (tcgen05) kernels do not
// take -- transposed A, K not a multiple of the TMA alignment, grouped / strided / dilated
// convolutions, the K=27 and K=9 first convolution layers -- and they are the numerical cross-check
// of the tensor-core kernels in the GPU tests. They run on the GPU; there is no CPU path.
#include "contract.cuh"

#include <cuda_fp8.h>
#include <type_traits>

using namespace sofie;

namespace sofie {

// ------------------------------------------------------------------------------------------------
// fp32 GEMM: 64x64 tile, 256 threads, 4x4 outputs per thread, K step 16.
// ------------------------------------------------------------------------------------------------
template <bool TA, bool TB>
__global__ void __launch_bounds__(256)
gemm_f32_simt_kernel(sofie_gemm_f32_desc d, const float *__restrict__ A, const float *__restrict__ B,
                     const float *__restrict__ C, float *__restrict__ Y)
{
   constexpr int BM = 64, BN = 64, BK = 16;
   __shared__ float As[BK][BM + 4];
   __shared__ float Bs[BK][BN + 4];
   const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
   const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
   float acc[4][4] = {};
   for (int k0 = 0; k0 < d.K; k0 += BK) {
      for (int i = tid; i < BM * BK; i += 256) {
         int m, k;
         if (TA) { m = i % BM; k = i / BM; } else { k = i % BK; m = i / BK; }
         int gm = m0 + m, gk = k0 + k;
         float v = 0.f;
         if (gm < d.M && gk < d.K) v = TA ? A[(size_t)gk * d.M + gm] : A[(size_t)gm * d.K + gk];
         As[k][m] = v;
      }
      for (int i = tid; i < BN * BK; i += 256) {
         int n, k;
         if (TB) { k = i % BK; n = i / BK; } else { n = i % BN; k = i / BN; }
         int gn = n0 + n, gk = k0 + k;
         float v = 0.f;
         if (gn < d.N && gk < d.K) v = TB ? B[(size_t)gn * d.K + gk] : B[(size_t)gk * d.N + gn];
         Bs[k][n] = v;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < BK; k++) {
         float a[4], b[4];
#pragma unroll
         for (int i = 0; i < 4; i++) a[i] = As[k][ty * 4 + i];
#pragma unroll
         for (int j = 0; j < 4; j++) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
         for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
   }
#pragma unroll
   for (int i = 0; i < 4; i++) {
      int gm = m0 + ty * 4 + i;
      if (gm >= d.M) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
         int gn = n0 + tx * 4 + j;
         if (gn >= d.N) continue;
         float y = d.alpha * acc[i][j];
         if (d.bias_kind == 1) y += d.beta * C[gn];
         else if (d.bias_kind == 2) y += d.beta * C[(size_t)gm * d.N + gn];
         if (d.relu) y = relu_ref(y);
         Y[(size_t)gm * d.N + gn] = y;
      }
   }
}

// ---- outputs of few terms (K <= 32) --------------------------------------------------------------
// What the kernel above spends on a large output of few terms is instructions: it walks K in steps of 16 between barriers for 64 x 64 outputs, and each staged value and
// each stored one has its own indexes. Here a block keeps its BN columns of B, all K of them, and walks tiles of BM rows, the next tile's A on its way under this one; a warp's
// BM / 8 rows read A as broadcasts of four rows and feed packed FMAs (two rows each, in the order of k and rounded as the scalar ones: the same sums), and a lane's columns are
// 32 apart, so that a warp stores whole lines of any alignment. Bound by issue slots still (20 instructions for 32 outputs of 9 terms, 63 % of the slots). Against the kernel
// above: 9602 x 3820 x 9 83 -> 38 us (its bytes take 23), 16384 x 4093 x 8 with a full C 169 -> 106 (83), 13028 x 2481 x 14 73 -> 42, 12399 x 459 x 23 28 -> 20, 728 x 2032 x 10 7.7 -> 6.1.
// Tiles of 128 rows: 41, 119, 45, 19, 6.8.
constexpr int kFewThreads = 256, kFewK = 32, kFewRows = 64;
template <int BN, int BIAS>
__global__ void __launch_bounds__(kFewThreads, 3)
gemm_f32_few_terms_kernel(sofie_gemm_f32_desc d, const float *__restrict__ A, const float *__restrict__ B, const float *C, float *Y, uint32_t tiles_m, uint32_t sharers, FastDiv columns,
                          FastDiv terms)
{
   constexpr int BM = kFewRows, ROWS = BM / 8, COLS = BN / 32, PA = BM + 4, PB = BN + 1, BATCH = 4; // rows of C under way
   extern __shared__ __align__(16) float few[];
   float *Bs = few + 2 * d.K * PA; // [k][column]; few: two tiles [k][row]
   const int tid = threadIdx.x, lane = tid & 31, row0 = (tid >> 5) * ROWS, K = d.K;
   uint32_t tn;
   const uint32_t sharer = columns.divmod(blockIdx.x, tn);
   const int n0 = (int)tn * BN;
   // EXTENT rows or columns from `first` on, of `count`, into [k][extent]; threads along what is contiguous in memory
   auto stage = [&](float *dst, int pitch, int extent, const float *src, bool k_contiguous, int first, int count) {
      for (int i = tid; i < extent * K; i += kFewThreads) {
         uint32_t k, e;
         if (k_contiguous) e = terms.divmod((uint32_t)i, k);
         else k = (uint32_t)i / (uint32_t)extent, e = (uint32_t)i % (uint32_t)extent; // a power of two
         const bool in = first + (int)e < count;
         const float *from = src + (in ? (k_contiguous ? (size_t)first * K + i : (size_t)k * count + first + e) : 0);
         asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + k * pitch + e)), "l"(from), "r"(in ? 4 : 0) : "memory");
      }
   };
   stage(Bs, PB, BN, B, d.transB, n0, d.N);
   stage(few, PA, BM, A, !d.transA, (int)sharer * BM, d.M);
   asm volatile("cp.async.commit_group;" ::: "memory");
   bool in[COLS];
   float bias[COLS];
#pragma unroll
   for (int j = 0; j < COLS; j++) {
      in[j] = n0 + lane + 32 * j < d.N;
      bias[j] = BIAS == 1 && in[j] ? d.beta * C[n0 + lane + 32 * j] : 0.f;
   }
   int buf = 0;
   for (uint32_t t = sharer; t < tiles_m; t += sharers, buf ^= 1) {
      const int m0 = (int)t * BM;
      __syncthreads(); // the tile before this one is no longer read
      if (t + sharers < tiles_m) stage(few + (buf ^ 1) * K * PA, PA, BM, A, !d.transA, (int)(t + sharers) * BM, d.M);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      uint64_t acc[ROWS / 2][COLS]; // two rows each
#pragma unroll
      for (int i = 0; i < ROWS / 2; i++)
#pragma unroll
         for (int j = 0; j < COLS; j++) acc[i][j] = 0;
      const float *a_k = few + buf * K * PA + row0, *b_k = Bs + lane;
#pragma unroll 2
      for (int k = 0; k < K; k++, a_k += PA, b_k += PB) {
         uint64_t b[COLS];
#pragma unroll
         for (int j = 0; j < COLS; j++) b[j] = pack_f32x2(b_k[32 * j], b_k[32 * j]);
#pragma unroll
         for (int i = 0; i < ROWS / 4; i++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(a_k + 4 * i);
#pragma unroll
            for (int j = 0; j < COLS; j++) {
               acc[2 * i][j] = fma_f32x2(a.x, b[j], acc[2 * i][j]);
               acc[2 * i + 1][j] = fma_f32x2(a.y, b[j], acc[2 * i + 1][j]);
            }
         }
      }
      const int rows = min(ROWS, d.M - m0 - row0);
      size_t at = (size_t)(m0 + row0) * d.N + n0 + lane;
#pragma unroll
      for (int i = 0; i < ROWS; i += BATCH) {
         float c[BATCH][COLS]; // read before the first of them is written: Y may be C
         if (BIAS == 2) {
#pragma unroll
            for (int r = 0; r < BATCH; r++)
#pragma unroll
               for (int j = 0; j < COLS; j++) c[r][j] = i + r < rows && in[j] ? C[at + (size_t)r * d.N + 32 * j] : 0.f;
         }
#pragma unroll
         for (int r = 0; r < BATCH; r++, at += d.N) {
            if (i + r >= rows) break;
#pragma unroll
            for (int j = 0; j < COLS; j++) {
               float lo, hi;
               unpack_f32x2(acc[(i + r) / 2][j], lo, hi);
               float y = d.alpha * ((i + r) % 2 ? hi : lo);
               if (BIAS == 1) y += bias[j];
               if (BIAS == 2) y = fmaf(d.beta, c[r][j], y);
               if (d.relu) y = relu_ref(y);
               if (in[j]) Y[at + 32 * j] = y;
            }
         }
      }
   }
}

template <int BN>
int launch_few_terms(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y)
{
   constexpr int BM = kFewRows;
   const int tiles_n = ceil_div(d.N, BN), tiles_m = ceil_div(d.M, BM), smem = d.K * (2 * (BM + 4) + BN + 1) * (int)sizeof(float);
   long long sharers = 3ll * kNumSMs / tiles_n; // blocks that share a column of tiles: three an SM are resident
   sharers = sharers < 1 ? 1 : (sharers > tiles_m ? tiles_m : sharers);
   auto go = [&](auto kind) -> int {
      auto kern = gemm_f32_few_terms_kernel<BN, decltype(kind)::value>;
      SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), smem));
      kern<<<(unsigned)(sharers * tiles_n), kFewThreads, smem, s>>>(d, A, B, C, Y, (uint32_t)tiles_m, (uint32_t)sharers, FastDiv(tiles_n), FastDiv(d.K));
      SOFIE_LAUNCH_CHECK("gemm_f32_few_terms_kernel");
      set_last_engine(SOFIE_ENGINE_SIMT);
      return SOFIE_CUDA_OK;
   };
   return d.bias_kind == 0 ? go(std::integral_constant<int, 0>{}) : d.bias_kind == 1 ? go(std::integral_constant<int, 1>{}) : go(std::integral_constant<int, 2>{});
}

static int launch_gemm_f32_few_terms(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y)
{
   // the widest tile that still gives every SM one; 64 x 64 against 64 x 32: 287 x 1457 x 8 (115 tiles) 3.5 us both, 78 x 1574 x 16 (50) 4.2 against 3.6
   // and of which no more than half is padding: 11732 x 19 x 14 (A transposed) 5.3 us at 128 columns, 3.7 at 32, 60000 x 9 x 4 6.5 and 4.5
   const long long tall = ceil_div(d.M, kFewRows);
   if (d.N > 64 && tall * ceil_div(d.N, 128) >= kNumSMs) return launch_few_terms<128>(s, d, A, B, C, Y);
   if (d.N > 32 && tall * ceil_div(d.N, 64) >= 64) return launch_few_terms<64>(s, d, A, B, C, Y);
   return launch_few_terms<32>(s, d, A, B, C, Y);
}

// Products of few FMAs, whatever the layout: what bounds them is latency. The kernel above walks K in steps of 16 with a round trip to memory
// and two barriers each (2 x 1 x 427 34 us), the tensor-core kernels set themselves up (6 to 8 us). Here T lanes share an output, each with every
// T-th term of K, all loads of eight terms issued together, and add up their sums in pairs: 2 x 1 x 427 2.7 us, 5 x 2 x 166 21.7 -> 2.3,
// 2 x 119 x 66 12.1 -> 2.6. From 1024 terms on a lane of 32 would have more than four such batches, 0.3 us each one after the other, and the split-K
// kernel would be the faster one: a block of 256 shares the output (3 x 6 x 7858 11.5 -> 5.1 us, split-K 5.9; 1 x 2 x 5995 8.7 -> 4.1, split-K 4.3). Sums carry what products and additions round off in a second
// word (T. Ogita, S. M. Rump and S. Oishi, "Accurate sum and dot product", 2005), which costs nothing here: no other kernel's are closer. (In 64 bits
// the same took 71 us for 1 x 1 x 16384.)
struct TwoSum {
   float s = 0.f, c = 0.f; // s is the ordinary sum
   __device__ __forceinline__ void add(float x)
   {
      const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
      c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z)));
      s = t;
   }
   __device__ __forceinline__ void add_product(float x, float y)
   {
      const float p = __fmul_rn(x, y);
      add(p);
      c = __fadd_rn(c, __fmaf_rn(x, y, -p));
   }
};
template <int T>
__global__ void __launch_bounds__(T > 128 ? T : 128)
gemm_f32_tiny_kernel(sofie_gemm_f32_desc d, const float *__restrict__ A, const float *__restrict__ B, const float *C, float *Y)
{
   griddep_launch_dependents();
   griddep_wait(A, B); // the operands may be the previous kernel's output
   const int i = (blockIdx.x * (T > 128 ? T : 128) + threadIdx.x) / T, t = threadIdx.x % T;
   const bool live = i < d.M * d.N;
   const int m = live ? i / d.N : 0, n = live ? i - m * d.N : 0;
   const long long as = d.transA ? d.M : 1, bs = d.transB ? 1 : d.N;
   const float *a = A + (d.transA ? m : (long long)m * d.K) + t * as, *b = B + (d.transB ? (long long)n * d.K : n) + t * bs;
   const float c = d.bias_kind == 0 || !live ? 0.f : C[d.bias_kind == 1 ? n : i];
   TwoSum acc;
   for (int k = t; k < d.K; k += 8 * T, a += 8 * T * as, b += 8 * T * bs) {
      float x[8], y[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
         const bool in = k + j * T < d.K;
         x[j] = in ? a[j * T * as] : 0.f;
         y[j] = in ? b[j * T * bs] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; j++) acc.add_product(x[j], y[j]);
   }
   auto add_up = [&](int lanes) { // of a group of lanes, into its first
      for (int o = lanes / 2; o > 0; o /= 2) {
         const float s = __shfl_down_sync(0xFFFFFFFFu, acc.s, o, lanes), r = __shfl_down_sync(0xFFFFFFFFu, acc.c, o, lanes);
         acc.add(s);
         acc.c += r;
      }
   };
   add_up(T > 32 ? 32 : T);
   if constexpr (T > 32) { // an output is a block's: the sums of its warps
      __shared__ float2 warps[T / 32];
      if (t % 32 == 0) warps[t / 32] = make_float2(acc.s, acc.c);
      __syncthreads();
      if (t >= 32) return;
      acc.s = warps[t % (T / 32)].x, acc.c = warps[t % (T / 32)].y;
      add_up(T / 32);
   }
   if (t == 0 && live) {
      float sum = acc.s + acc.c;
      if (!(fabsf(sum) < __uint_as_float(0x7F800000u))) { // infinities, NaNs, and what overflows: as the chain of FMAs
         sum = 0.f;
         a = A + (d.transA ? m : (long long)m * d.K), b = B + (d.transB ? (long long)n * d.K : n);
         for (int k = 0; k < d.K; k++, a += as, b += bs) sum = fmaf(*a, *b, sum);
      }
      float y = d.alpha * sum;
      if (d.bias_kind) y += d.beta * c;
      Y[i] = d.relu ? relu_ref(y) : y;
   }
}

// Up to 2^18 FMAs, of 8192 terms at most: from there on the loads count, which are not shared (2^19: 1.4 to 1.7 times as fast in the mean, but
// half as fast in the worst case; up to 2^18 1.2 to 4 times, 2.4 in the mean, over 420 products of every layout). A longer K is taken where the
// kernel above would.
bool gemm_f32_tiny_ok(const sofie_gemm_f32_desc &d)
{
   const long long fmas = (long long)d.M * d.N * d.K;
   return (long long)d.M * d.N <= 1 << 18 && fmas <= 1 << 18 && (d.K <= 8192 || fmas <= 32768);
}

int launch_gemm_f32_tiny(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y)
{
   const int outputs = d.M * d.N;
   auto launch = [&](auto lanes) {
      constexpr int T = decltype(lanes)::value, threads = T > 128 ? T : 128;
      return launch_dependent(gemm_f32_tiny_kernel<T>, dim3(ceil_div(outputs * T, threads)), dim3(threads), 0, s, d, A, B, C, Y);
   };
   // as many lanes as keep a lane's terms to one batch of loads; 256 for 740 to 1024 terms of a hundred outputs and more are up to 10 % slower than 32
   SOFIE_CUDA_TRY(d.K <= 8 ? launch(std::integral_constant<int, 1>{}) : d.K <= 32 ? launch(std::integral_constant<int, 4>{}) :
                  d.K <= 128 ? launch(std::integral_constant<int, 16>{}) : d.K <= 1024 ? launch(std::integral_constant<int, 32>{}) : launch(std::integral_constant<int, 256>{}));
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

int launch_gemm_f32_simt(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C,
                         float *Y)
{
   // (up to eight columns a block of one step is as soon done: 16377 x 2 x 10 4.8 us against 5.3)
   if (d.K <= kFewK && d.M > 8 && d.N > 8) return launch_gemm_f32_few_terms(s, d, A, B, C, Y);
   dim3 grid(ceil_div(d.N, 64), ceil_div(d.M, 64));
   if (d.transA && d.transB) gemm_f32_simt_kernel<true, true><<<grid, 256, 0, s>>>(d, A, B, C, Y);
   else if (d.transA) gemm_f32_simt_kernel<true, false><<<grid, 256, 0, s>>>(d, A, B, C, Y);
   else if (d.transB) gemm_f32_simt_kernel<false, true><<<grid, 256, 0, s>>>(d, A, B, C, Y);
   else gemm_f32_simt_kernel<false, false><<<grid, 256, 0, s>>>(d, A, B, C, Y);
   SOFIE_LAUNCH_CHECK("gemm_f32_simt_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// ------------------------------------------------------------------------------------------------
// Direct convolution, fp32 and uint8/int8. One thread = one (pooled) output position x OCB output
// channels; the weights of those channels sit in shared memory and are read as broadcasts.
// ------------------------------------------------------------------------------------------------
constexpr int kConvOCB = 16;     // output channels per block
constexpr int kConvThreads = 128;

template <typename TX, typename TW, typename TACC>
__device__ __forceinline__ void conv_accumulate(const ConvGeom &g, const TX *__restrict__ X, const TW *__restrict__ ws,
                                                int n, int cbase, int cg, int oh, int ow, int x_zp, TACC *acc)
{
   for (int c = 0; c < cg; c++) {
      for (int r = 0; r < g.kH; r++) {
         int ih = oh * g.sh - g.pad_h + r * g.dh;
         if (ih < 0 || ih >= g.H) continue;
         for (int t = 0; t < g.kW; t++) {
            int iw = ow * g.sw - g.pad_w + t * g.dw;
            if (iw < 0 || iw >= g.W) continue;
            int cc = cbase + c;
            size_t xi = g.x_nhwc ? (((size_t)n * g.H + ih) * g.W + iw) * g.C + cc
                                 : (((size_t)n * g.C + cc) * g.H + ih) * g.W + iw;
            TACC xv = (TACC)X[xi] - (TACC)x_zp;
            const TW *w = ws + ((c * g.kH + r) * g.kW + t) * kConvOCB;
#pragma unroll
            for (int o = 0; o < kConvOCB; o++) {
               if constexpr (std::is_integral_v<TACC>) acc[o] += xv * (TACC)w[o];
               else acc[o] = fmaf(xv, (TACC)w[o], acc[o]);
            }
         }
      }
   }
}

// Epilogue functors turn the accumulators of one output position into stored values.
struct EpiF32 {
   const float *bias;
   __device__ float operator()(float acc, int oc, int relu) const
   {
      float v = bias ? acc + bias[oc] : acc;
      return relu ? relu_ref(v) : v;
   }
};
struct EpiU8 {
   const float *mult;
   const int32_t *bias;
   int y_zp;
   __device__ uint8_t operator()(int acc, int oc, int relu) const
   {
      if (bias) acc += bias[oc];
      return (uint8_t)requant_u8(acc, mult[oc], y_zp, relu);
   }
};

template <typename TX, typename TW, typename TACC, typename TY, typename Epi>
__global__ void __launch_bounds__(kConvThreads)
conv2d_direct_kernel(ConvGeom g, const TX *__restrict__ X, const TW *__restrict__ Wt, Epi epi, int x_zp,
                     TY *__restrict__ Y)
{
   extern __shared__ __align__(16) unsigned char smem_raw[];
   TW *ws = reinterpret_cast<TW *>(smem_raw);
   const int cg = g.C / g.group, og = g.Cout / g.group;
   const int ocb_per_group = ceil_div(og, kConvOCB);
   const int grp = blockIdx.y / ocb_per_group;
   const int oc0 = grp * og + (blockIdx.y % ocb_per_group) * kConvOCB; // first output channel of this block
   const int oc_end = (grp + 1) * og;
   const int kk = cg * g.kH * g.kW;
   // stage weights as ws[(c,r,t)][o]
   for (int i = threadIdx.x; i < kk * kConvOCB; i += kConvThreads) {
      int o = i % kConvOCB, k = i / kConvOCB;
      int oc = oc0 + o;
      TW v = 0;
      if (oc < oc_end) {
         int t = k % g.kW, r = (k / g.kW) % g.kH, c = k / (g.kW * g.kH);
         size_t wi = g.w_packed ? (((size_t)oc * g.kH + r) * g.kW + t) * cg + c
                                : (((size_t)oc * cg + c) * g.kH + r) * g.kW + t;
         v = Wt[wi];
      }
      ws[i] = v;
   }
   __syncthreads();
   const size_t positions = (size_t)g.N * g.pH * g.pW;
   for (size_t p = blockIdx.x * (size_t)kConvThreads + threadIdx.x; p < positions;
        p += (size_t)gridDim.x * kConvThreads) {
      int pw = p % g.pW, ph = (p / g.pW) % g.pH, n = p / ((size_t)g.pW * g.pH);
      TY best[kConvOCB];
      const int taps = g.pool == 2 ? 4 : 1;
      for (int q = 0; q < taps; q++) {
         int oh = g.pool == 2 ? ph * 2 + (q >> 1) : ph, ow = g.pool == 2 ? pw * 2 + (q & 1) : pw;
         TACC acc[kConvOCB];
#pragma unroll
         for (int o = 0; o < kConvOCB; o++) acc[o] = 0;
         conv_accumulate<TX, TW, TACC>(g, X, ws, n, grp * cg, cg, oh, ow, x_zp, acc);
#pragma unroll
         for (int o = 0; o < kConvOCB; o++) {
            TY v = epi(acc[o], min(oc0 + o, g.Cout - 1), g.relu);
            best[o] = (q == 0 || v > best[o]) ? v : best[o];
         }
      }
#pragma unroll
      for (int o = 0; o < kConvOCB; o++) {
         int oc = oc0 + o;
         if (oc >= oc_end) break;
         size_t yi = g.y_nhwc ? (((size_t)n * g.pH + ph) * g.pW + pw) * g.Cout + oc
                              : (((size_t)n * g.Cout + oc) * g.pH + ph) * g.pW + pw;
         Y[yi] = best[o];
      }
   }
}

template <typename TX, typename TW, typename TACC, typename TY, typename Epi>
int launch_conv_direct(cudaStream_t s, const ConvGeom &g, const TX *X, const TW *Wt, Epi epi, int x_zp, TY *Y)
{
   const int cg = g.C / g.group, og = g.Cout / g.group;
   size_t smem = (size_t)cg * g.kH * g.kW * kConvOCB * sizeof(TW);
   if (smem > 200 * 1024) return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "convolution weights slice of %zu bytes exceeds shared memory", smem);
   auto kern = conv2d_direct_kernel<TX, TW, TACC, TY, Epi>;
   if (smem > 48 * 1024) SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), (int)smem));
   size_t positions = (size_t)g.N * g.pH * g.pW;
   if (positions == 0) return SOFIE_CUDA_OK;
   int gy = g.group * ceil_div(og, kConvOCB);
   size_t gx = ceil_div<size_t>(positions, kConvThreads);
   size_t cap = (size_t)kNumSMs * 16;
   if (gx > cap) gx = cap;
   kern<<<dim3((unsigned)gx, gy), kConvThreads, smem, s>>>(g, X, Wt, epi, x_zp, Y);
   SOFIE_LAUNCH_CHECK("conv2d_direct_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

int launch_conv2d_f32_simt(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias,
                           float *Y)
{
   int rc = launch_conv2d_f32_first(s, g, X, W, bias, Y);
   if (rc < 0) rc = launch_conv2d_f32_direct3x3(s, g, X, W, bias, Y);
   if (rc >= 0) return rc;
   return launch_conv_direct<float, float, float, float, EpiF32>(s, g, X, W, EpiF32{bias}, 0, Y);
}
int launch_qconv2d_simt(cudaStream_t s, const ConvGeom &g, const uint8_t *X, const int8_t *W, const float *mult,
                        const int32_t *bias, int x_zp, int y_zp, uint8_t *Y)
{
   const int rc = launch_qconv2d_first(s, g, X, W, mult, bias, x_zp, y_zp, Y);
   if (rc >= 0) return rc;
   return launch_conv_direct<uint8_t, int8_t, int, uint8_t, EpiU8>(s, g, X, W, EpiU8{mult, bias, y_zp}, x_zp, Y);
}

// ------------------------------------------------------------------------------------------------
// uint8 x int8 GEMM with int32 accumulation (dp4a), W as [N,K]. 64x64 tile, K step 64 bytes.
// Computes sum_k a*w (a unsigned); the zero-point term arrives through corr[n].
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ int dp4a_u8s8(unsigned a, int b, int c)
{
   int d;
   asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
   return d;
}

template <bool WNK>
__global__ void __launch_bounds__(256)
qgemm_simt_kernel(sofie_qgemm_desc d, const uint8_t *__restrict__ A, const int8_t *__restrict__ W,
                  const float *__restrict__ mult, const int32_t *__restrict__ corr, uint8_t *__restrict__ Y, float *__restrict__ Yf32,
                  float dq_scale)
{
   constexpr int BM = 64, BN = 64, BK = 64;
   __shared__ unsigned As[BM][BK / 4 + 1];
   __shared__ int Ws[BN][BK / 4 + 1];
   const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
   const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
   int acc[4][4] = {};
   for (int k0 = 0; k0 < d.K; k0 += BK) {
      for (int i = tid; i < BM * BK; i += 256) {
         int k = i % BK, m = i / BK;
         int gm = m0 + m, gk = k0 + k;
         uint8_t v = (gm < d.M && gk < d.K) ? A[(size_t)gm * d.K + gk] : 0;
         reinterpret_cast<uint8_t *>(&As[m][0])[k] = v;
      }
      for (int i = tid; i < BN * BK; i += 256) {
         int n, k;
         if (WNK) { k = i % BK; n = i / BK; } else { n = i % BN; k = i / BN; }
         int gn = n0 + n, gk = k0 + k;
         int8_t v = 0;
         if (gn < d.N && gk < d.K) v = WNK ? W[(size_t)gn * d.K + gk] : W[(size_t)gk * d.N + gn];
         reinterpret_cast<int8_t *>(&Ws[n][0])[k] = v;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < BK / 4; k++) {
         unsigned a[4];
         int b[4];
#pragma unroll
         for (int i = 0; i < 4; i++) a[i] = As[ty * 4 + i][k];
#pragma unroll
         for (int j = 0; j < 4; j++) b[j] = Ws[tx * 4 + j][k];
#pragma unroll
         for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = dp4a_u8s8(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
   }
#pragma unroll
   for (int i = 0; i < 4; i++) {
      int gm = m0 + ty * 4 + i;
      if (gm >= d.M) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
         int gn = n0 + tx * 4 + j;
         if (gn >= d.N) continue;
         int a = acc[i][j] + (corr ? corr[gn] : 0);
         const int q = requant_u8(a, mult[gn], d.y_zp, d.relu);
         if (Yf32) Yf32[(size_t)gm * d.N + gn] = __fmul_rn((float)(q - d.y_zp), dq_scale);
         else Y[(size_t)gm * d.N + gn] = (uint8_t)q;
      }
   }
}

int launch_qgemm_simt(cudaStream_t s, const sofie_qgemm_desc &d, const uint8_t *A, const int8_t *W, const float *mult,
                      const int32_t *corr, uint8_t *Y, float *Yf32, float dq_scale)
{
   dim3 grid(ceil_div(d.N, 64), ceil_div(d.M, 64));
   if (d.w_is_nk) qgemm_simt_kernel<true><<<grid, 256, 0, s>>>(d, A, W, mult, corr, Y, Yf32, dq_scale);
   else qgemm_simt_kernel<false><<<grid, 256, 0, s>>>(d, A, W, mult, corr, Y, Yf32, dq_scale);
   SOFIE_LAUNCH_CHECK("qgemm_simt_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// ------------------------------------------------------------------------------------------------
// E4M3 x E4M3 GEMM on CUDA cores: decode through a 256-entry table, fp32 FMA accumulation.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float e4m3_decode(unsigned v)
{
   unsigned e = (v >> 3) & 0xF, m = v & 7;
   float r;
   if (e == 0) r = (float)m * 0.001953125f; // m * 2^-9
   else r = __uint_as_float(((e + 120u) << 23) | (m << 20));
   if (e == 0xF && m == 7) r = __uint_as_float(0x7FC00000u);
   return (v & 0x80) ? -r : r;
}

__global__ void __launch_bounds__(256)
gemm_e4m3_simt_kernel(sofie_fp8_gemm_desc d, const uint8_t *__restrict__ A, const uint8_t *__restrict__ W,
                      const float *__restrict__ bias, uint16_t *__restrict__ Ybf16, uint8_t *__restrict__ Yq, float *__restrict__ Yf32,
                      const float *__restrict__ a_scale_dev)
{
   constexpr int BM = 64, BN = 64, BK = 16;
   __shared__ float lut[256];
   __shared__ float As[BK][BM + 4];
   __shared__ float Bs[BK][BN + 4];
   const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
   lut[tid] = e4m3_decode(tid);
   __syncthreads();
   const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
   float acc[4][4] = {};
   for (int k0 = 0; k0 < d.K; k0 += BK) {
      for (int i = tid; i < BM * BK; i += 256) {
         int k = i % BK, m = i / BK, gm = m0 + m, gk = k0 + k;
         As[k][m] = (gm < d.M && gk < d.K) ? lut[A[(size_t)gm * d.K + gk]] : 0.f;
      }
      for (int i = tid; i < BN * BK; i += 256) {
         int k = i % BK, n = i / BK, gn = n0 + n, gk = k0 + k;
         Bs[k][n] = (gn < d.N && gk < d.K) ? lut[W[(size_t)gn * d.K + gk]] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < BK; k++) {
         float a[4], b[4];
#pragma unroll
         for (int i = 0; i < 4; i++) a[i] = As[k][ty * 4 + i];
#pragma unroll
         for (int j = 0; j < 4; j++) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
         for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
      __syncthreads();
   }
   const float scale = __fmul_rn(a_scale_dev ? *a_scale_dev : d.a_scale, d.w_scale);
#pragma unroll
   for (int i = 0; i < 4; i++) {
      int gm = m0 + ty * 4 + i;
      if (gm >= d.M) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
         int gn = n0 + tx * 4 + j;
         if (gn >= d.N) continue;
         float y = __fmul_rn(acc[i][j], scale);
         if (bias) y = __fadd_rn(y, bias[gn]);
         if (d.relu) y = relu_ref(y);
         uint16_t h = f32_to_bf16_rne(y);
         if (Ybf16) Ybf16[(size_t)gm * d.N + gn] = h;
         if (Yf32) Yf32[(size_t)gm * d.N + gn] = bf16_to_f32(h);
         if (Yq) Yq[(size_t)gm * d.N + gn] =
            (uint8_t)__nv_cvt_float_to_fp8(__fdiv_rn(bf16_to_f32(h), d.q_scale), __NV_SATFINITE, __NV_E4M3);
      }
   }
}

int launch_gemm_e4m3_simt(cudaStream_t s, const sofie_fp8_gemm_desc &d, const uint8_t *A, const uint8_t *W,
                          const float *bias, uint16_t *Ybf16, uint8_t *Yq, float *Yf32, const float *a_scale_dev)
{
   dim3 grid(ceil_div(d.N, 64), ceil_div(d.M, 64));
   gemm_e4m3_simt_kernel<<<grid, 256, 0, s>>>(d, A, W, bias, Ybf16, Yq, Yf32, a_scale_dev);
   SOFIE_LAUNCH_CHECK("gemm_e4m3_simt_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

// Weight repack [Cout, C, kH, kW] -> [Cout, kH, kW, C].
template <typename T>
__global__ void pack_ohwi_kernel(const T *__restrict__ W, T *__restrict__ P, int Cout, int C, int kH, int kW)
{
   size_t total = (size_t)Cout * C * kH * kW;
   for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
      int c = i % C;
      size_t t = i / C;
      int s = t % kW; t /= kW;
      int r = t % kH;
      int oc = t / kH;
      P[i] = W[(((size_t)oc * C + c) * kH + r) * kW + s];
   }
}
template <typename T>
int launch_pack_ohwi(cudaStream_t s, const T *W, T *P, int Cout, int C, int kH, int kW)
{
   size_t total = (size_t)Cout * C * kH * kW;
   if (!total) return SOFIE_CUDA_OK;
   int blocks = (int)(ceil_div<size_t>(total, 256) < 1184 ? ceil_div<size_t>(total, 256) : 1184);
   pack_ohwi_kernel<T><<<blocks, 256, 0, s>>>(W, P, Cout, C, kH, kW);
   SOFIE_LAUNCH_CHECK("pack_ohwi_kernel");
   return SOFIE_CUDA_OK;
}
template int launch_pack_ohwi<float>(cudaStream_t, const float *, float *, int, int, int, int);
template int launch_pack_ohwi<int8_t>(cudaStream_t, const int8_t *, int8_t *, int, int, int, int);

} // namespace sofie
