// fp32 products with at most 8 rows or columns (from 64 terms on, of more FMAs than gemm_f32_tiny_kernel's), any layout.
//
// One operand is long (R rows), the other short (S <= 8). What bounds such a product is the long operand's way out of memory, as long as enough of it is asked for at
// once; the tile kernels leave most SMs idle or pad S to their tile, and the split-K pair are two launches. Every value of the long operand is one thread's alone here, so it comes
// straight into registers, sixteen loads under way, whole lines a warp whatever the alignment; the short operand's slice is staged in shared memory.
//   neighbouring rows are neighbours in memory: a lane owns RT rows, the warps take k in turn, the short operand is read as broadcasts (packed FMAs of two columns)
//   rows contiguous in k: the lanes take k in turn, a warp owns RT rows, its sums are added up by a butterfly that leaves each lane some of them
// K is cut over a cluster of up to eight blocks, whose sums meet through distributed shared memory: each block adds up and writes its share of the outputs. Chains are
// 16 or 32 terms long, a chunk's are added up before they join the sum of the chunks, and the last additions (of the lanes that hold a row's terms, of the blocks) are in 64 bits and rounded once: of 160 drawn products none was
// further from float64 than on the kernels that took them before (0.70 of their error in the mean, 0.31 with operands of one sign); with all of it in 32 bits some were by a tenth, and the chains of rows contiguous in k
// grew with K. It costs 2 % of the time in the mean, 15 % at most (6 x 1069 x 820, B stored [N,K]: 5.3 -> 6.1 us).
// The drawn products take 0.69 of those kernels' time in the mean; 2 x 3731 x 2897 31 -> 10.3 us, 6317 x 2 x 3797 (A transposed) 45 -> 23 (its bytes take 15), 5 x 2378 x 2513 27 -> 12.6 (B stored [N,K] 30 -> 15.0),
// 9640 x 7 x 1000 24 -> 17.4, 3027 x 4 x 108 6.3 -> 3.2. 9 to 16 columns are no faster (1.0 in the mean: the short operand's reads), nor are tiles of the long operand in shared memory.
#include "contract.cuh"

namespace sofie {
namespace {

constexpr int kSkThreads = 256, kSkWarps = kSkThreads / 32, kSkLoads = 16;

struct SkinnyArgs {
   const float *P, *Q, *C;
   float *Y;
   long long q_s, q_k; // strides of the short operand
   long long y_r, y_s; // of the result (and a C of its shape)
   int R, S, K, per;   // per: K a block
   float alpha, beta;
   int bias_kind, bias_long, relu; // bias_long: a C of one row runs along the long operand
};

// Rows r0 .. r0 + rows of the result out of the blocks' sums [row][SP + 1], threads along what is contiguous in Y.
template <int SP>
__device__ __forceinline__ void skinny_output(const SkinnyArgs &g, const double *sums, int r0, int rows, uint32_t rank, uint32_t ranks)
{
   if (ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
   else __syncthreads();
   const int total = rows * g.S;
   for (int i = threadIdx.x + (int)rank * kSkThreads; i < total; i += (int)ranks * kSkThreads) {
      const bool along_s = g.y_s == 1;
      const int r = along_s ? i / g.S : i % rows, s = along_s ? i - r * g.S : i / rows;
      const double *at = sums + r * (SP + 1) + s;
      double sum = 0.0; // over the blocks that share K
      const uint32_t local = (uint32_t)__cvta_generic_to_shared(at);
#pragma unroll
      for (uint32_t c = 0; c < 8; c++) {
         uint32_t remote;
         double part = 0.0;
         if (c < ranks) {
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(c));
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(part) : "r"(remote) : "memory");
         }
         sum += part;
      }
      const long long y = (r0 + r) * g.y_r + s * g.y_s;
      double full = g.alpha * sum;
      if (g.bias_kind == 1) full += (double)g.beta * g.C[g.bias_long ? r0 + r : s];
      else if (g.bias_kind == 2) full += (double)g.beta * g.C[y];
      const float out = (float)full;
      g.Y[y] = g.relu ? relu_ref(out) : out;
   }
   if (ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory"); // no block ends while its sums are read
}

// COUNT k of the short operand from k0 on into shared memory, [k][SP] or [s][pitch], zeros behind k_end and S
template <int SP, bool K_FIRST>
__device__ __forceinline__ void skinny_stage(const SkinnyArgs &g, float *dst, int pitch, int count, int k0, int k_end)
{
   auto copy = [&](int k, int s) {
      const bool in = s < g.S && k0 + k < k_end;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + (K_FIRST ? k * pitch + s : s * pitch + k))),
                   "l"(in ? g.Q + s * g.q_s + (k0 + k) * g.q_k : g.Q), "r"(in ? 4 : 0)
                   : "memory");
   };
   // threads along what is contiguous in memory
   if (g.q_k == 1) {
      for (int s = threadIdx.x >> 5; s < SP; s += kSkWarps)
         for (int k = threadIdx.x & 31; k < count; k += 32) copy(k, s);
   } else {
      for (int k = threadIdx.x / SP; k < count; k += kSkThreads / SP) copy(k, threadIdx.x % SP);
   }
   asm volatile("cp.async.wait_all;" ::: "memory");
}

__device__ __forceinline__ void skinny_ranks(uint32_t &rank, uint32_t &ranks)
{
   asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
   asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
}

constexpr int kSkChunk = 512; // k of the short operand in shared memory at a time

template <int SP, int RT>
__global__ void __launch_bounds__(kSkThreads, 2) gemm_f32_skinny_lanes_kernel(SkinnyArgs g)
{
   constexpr int U = kSkLoads / RT, ROWS = 32 * RT, CHAINS = 16 / SP; // k under way; sums of every CHAINS-th of them
   __shared__ __align__(16) float q[kSkChunk * SP > kSkWarps / 2 * RT * SP * 32 ? kSkChunk * SP : kSkWarps / 2 * RT * SP * 32]; // later: half of the warps' sums
   __shared__ double sums[ROWS * (SP + 1)];
   griddep_launch_dependents();
   griddep_wait(); // the operands may be the previous kernel's output
   uint32_t rank, ranks;
   skinny_ranks(rank, ranks);
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = (int)(blockIdx.x / ranks) * ROWS, k_begin = (int)rank * g.per, k_end = min(g.K, k_begin + g.per);
   const float *p = g.P + r0 + lane;
   bool in[RT];
#pragma unroll
   for (int i = 0; i < RT; i++) in[i] = r0 + lane + 32 * i < g.R;
   auto load = [&](float(&v)[U][RT], int k) {
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
         for (int i = 0; i < RT; i++) v[u][i] = k + kSkWarps * u < k_end && in[i] ? load_dependent(p + (size_t)(k + kSkWarps * u) * g.R + 32 * i) : 0.f;
   };
   uint64_t chain[CHAINS][RT][SP / 2]; // two columns each
#pragma unroll
   for (int c = 0; c < CHAINS; c++)
#pragma unroll
      for (int i = 0; i < RT; i++)
#pragma unroll
         for (int j = 0; j < SP / 2; j++) chain[c][i][j] = 0;
   float acc[RT][SP] = {};
   float v[2][U][RT];
   load(v[0], k_begin + warp);
   for (int c0 = k_begin; c0 < k_end; c0 += kSkChunk) {
      if (c0 != k_begin) __syncthreads();
      skinny_stage<SP, true>(g, q, SP, min(kSkChunk, k_end - c0 + 2 * kSkWarps * U), c0, k_end);
      __syncthreads();
      const int end = min(k_end, c0 + kSkChunk);
      auto step = [&](float(&now)[U][RT], float(&next)[U][RT], int k) {
         load(next, k + kSkWarps * U);
#pragma unroll
         for (int u = 0; u < U; u++) {
            const float *w = q + (k + kSkWarps * u - c0) * SP;
#pragma unroll
            for (int j = 0; j < SP / 4; j++) {
               const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(w + 4 * j);
#pragma unroll
               for (int i = 0; i < RT; i++) {
                  const uint64_t x = pack_f32x2(now[u][i], now[u][i]);
                  chain[u % CHAINS][i][2 * j] = fma_f32x2(x, b.x, chain[u % CHAINS][i][2 * j]);
                  chain[u % CHAINS][i][2 * j + 1] = fma_f32x2(x, b.y, chain[u % CHAINS][i][2 * j + 1]);
               }
            }
         }
      };
      static_assert(kSkChunk % (2 * kSkWarps * U) == 0, "two steps at a time");
      for (int k = c0 + warp; k < end; k += 2 * kSkWarps * U) {
         step(v[0], v[1], k);
         step(v[1], v[0], k + kSkWarps * U); // zeros behind k_end
      }
      // the chains of these k join the thread's sums
#pragma unroll
      for (int i = 0; i < RT; i++)
#pragma unroll
         for (int j = 0; j < SP / 2; j++) {
            float lo[CHAINS], hi[CHAINS];
#pragma unroll
            for (int c = 0; c < CHAINS; c++) {
               unpack_f32x2(chain[c][i][j], lo[c], hi[c]);
               chain[c][i][j] = 0;
            }
            acc[i][2 * j] += CHAINS == 4 ? (lo[0] + lo[1]) + (lo[2 % CHAINS] + lo[3 % CHAINS]) : lo[0] + lo[1];
            acc[i][2 * j + 1] += CHAINS == 4 ? (hi[0] + hi[1]) + (hi[2 % CHAINS] + hi[3 % CHAINS]) : hi[0] + hi[1];
         }
   }
   // the warps' sums, half of them to the other half, three times
#pragma unroll
   for (int half = kSkWarps / 2; half >= 1; half /= 2) {
      __syncthreads(); // the short operand, or the sums before these, are no longer read
      float *mine = q + (warp % half) * RT * SP * 32 + lane;
      if (warp >= half && warp < 2 * half) {
#pragma unroll
         for (int i = 0; i < RT; i++)
#pragma unroll
            for (int j = 0; j < SP; j++) mine[(i * SP + j) * 32] = acc[i][j];
      }
      __syncthreads();
      if (warp < half) {
#pragma unroll
         for (int i = 0; i < RT; i++)
#pragma unroll
            for (int j = 0; j < SP; j++) acc[i][j] += mine[(i * SP + j) * 32];
      }
   }
   if (warp == 0) {
#pragma unroll
      for (int i = 0; i < RT; i++)
#pragma unroll
         for (int j = 0; j < SP; j++) sums[(lane + 32 * i) * (SP + 1) + j] = acc[i][j];
   }
   skinny_output<SP>(g, sums, r0, min(ROWS, g.R - r0), rank, ranks);
}

// W: consecutive k a lane loads at once (rows of whole 16-byte words: 4)
template <int SP, int RT, int W>
__global__ void __launch_bounds__(kSkThreads, 2) gemm_f32_skinny_rows_kernel(SkinnyArgs g)
{
   constexpr int U = kSkLoads / RT / W, STEP = 32 * W, STRIDE = U * STEP, CHUNK = kSkChunk, PITCH = CHUNK + 4, N = RT * SP, ROWS = kSkWarps * RT;
   __shared__ __align__(16) float q[SP * PITCH]; // [s][k]
   __shared__ double sums[ROWS * (SP + 1)];
   griddep_launch_dependents();
   griddep_wait();
   uint32_t rank, ranks;
   skinny_ranks(rank, ranks);
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = (int)(blockIdx.x / ranks) * ROWS, k_begin = (int)rank * g.per, k_end = min(g.K, k_begin + g.per), first = warp * RT;
   const float *p[RT];
   bool in[RT];
#pragma unroll
   for (int i = 0; i < RT; i++) {
      in[i] = r0 + first + i < g.R;
      p[i] = g.P + (size_t)(in[i] ? r0 + first + i : 0) * g.K;
   }
   auto load = [&](float(&v)[U][RT][W], int k0) {
#pragma unroll
      for (int u = 0; u < U; u++) {
         const int k = k0 + u * STEP + lane * W;
#pragma unroll
         for (int i = 0; i < RT; i++) {
            const bool ok = k < k_end && in[i];
            if constexpr (W == 4) {
               if (ok) asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[u][i][0]), "=f"(v[u][i][1]), "=f"(v[u][i][2]), "=f"(v[u][i][3]) : "l"(p[i] + k) : "memory");
               else v[u][i][0] = v[u][i][1] = v[u][i][2] = v[u][i][3] = 0.f;
            } else {
               v[u][i][0] = ok ? load_dependent(p[i] + k) : 0.f;
            }
         }
      }
   };
   float chain[N], sum[N]; // of this chunk's terms; of the chunks before it
#pragma unroll
   for (int j = 0; j < N; j++) chain[j] = sum[j] = 0.f;
   float v[2][U][RT][W];
   static_assert(CHUNK % (2 * STRIDE) == 0, "two steps at a time");
   load(v[0], k_begin);
   for (int c0 = k_begin; c0 < k_end; c0 += CHUNK) {
      if (c0 != k_begin) __syncthreads();
      skinny_stage<SP, false>(g, q, PITCH, min(CHUNK, k_end - c0 + 2 * STRIDE), c0, k_end);
      __syncthreads();
      auto step = [&](float(&now)[U][RT][W], float(&next)[U][RT][W], int k0) {
         load(next, k0 + STRIDE);
#pragma unroll
         for (int u = 0; u < U; u++) {
            const int k = k0 + u * STEP + lane * W - c0;
#pragma unroll
            for (int s = 0; s < SP; s++) {
               float w[W];
               if constexpr (W == 4) {
                  const float4 x = *reinterpret_cast<const float4 *>(q + s * PITCH + k);
                  w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
               } else {
                  w[0] = q[s * PITCH + k];
               }
#pragma unroll
               for (int i = 0; i < RT; i++)
#pragma unroll
                  for (int e = 0; e < W; e++) chain[i * SP + s] = fmaf(now[u][i][e], w[e], chain[i * SP + s]);
            }
         }
      };
      const int end = min(k_end, c0 + CHUNK);
      for (int k0 = c0; k0 < end; k0 += 2 * STRIDE) {
         step(v[0], v[1], k0);
         step(v[1], v[0], k0 + STRIDE); // zeros behind k_end
      }
#pragma unroll
      for (int j = 0; j < N; j++) {
         sum[j] += chain[j];
         chain[j] = 0.f;
      }
   }
   // a butterfly over the lanes: while a lane has several sums it sends half of them and keeps the other half; the last three steps, where a rounding counts most, in 64 bits
   int kept = N, at = 0;
   auto halve = [&](auto *v, int o) {
      const bool up = lane & o;
      if (kept > 1) {
         kept >>= 1;
#pragma unroll
         for (int j = 0; j < N / 2; j++)
            if (j < kept) {
               const auto send = up ? v[j] : v[j + kept], keep = up ? v[j + kept] : v[j];
               v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
         at += up ? kept : 0;
      } else {
         v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      }
   };
   halve(sum, 16);
   halve(sum, 8);
   double acc[N / 4];
#pragma unroll
   for (int j = 0; j < N / 4; j++) acc[j] = sum[j];
   static_assert(N == 16 || N == 32, "four sums a lane after the first steps, or eight");
   halve(acc, 4);
   halve(acc, 2);
   halve(acc, 1);
   sums[(first + at / SP) * (SP + 1) + at % SP] = acc[0];
   skinny_output<SP>(g, sums, r0, min(ROWS, g.R - r0), rank, ranks);
}

int launch_clustered(cudaStream_t s, void (*kern)(SkinnyArgs), SkinnyArgs &g, int rows, int slice)
{
   // As many blocks to a K as leave under 300 of them (two an SM are resident) and slices of `slice` at least. Of 160 drawn products 27 take another cut with 150, 1.24 of the time in their mean (0.79 to 1.64),
   // 23 with 600, 1.25 (0.85 to 2.06).
   const int groups = ceil_div(g.R, rows);
   int ranks = 1;
   while (ranks < 8 && (long long)groups * ranks * 2 < 300 && g.K / (ranks * 2) >= slice) ranks *= 2;
   g.per = (ceil_div(g.K, ranks) + 3) & ~3; // slices start on 16-byte words
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3((unsigned)(groups * ranks));
   cfg.blockDim = dim3(kSkThreads);
   cfg.stream = s;
   cudaLaunchAttribute attr[2];
   attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
   attr[1].id = cudaLaunchAttributeClusterDimension;
   attr[1].val.clusterDim = {(unsigned)ranks, 1, 1};
   cfg.attrs = attr;
   cfg.numAttrs = ranks > 1 ? 2 : 1;
   SOFIE_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, g));
   SOFIE_LAUNCH_CHECK("gemm_f32_skinny_kernel");
   set_last_engine(SOFIE_ENGINE_SIMT);
   return SOFIE_CUDA_OK;
}

template <int SP>
int launch_skinny(cudaStream_t s, SkinnyArgs &g, bool k_contiguous)
{
   if (!k_contiguous) {
      const int pairs = ceil_div(g.R, 64); // of rows a lane: one where a whole cluster on each would leave most SMs idle
      if (pairs < 5) return launch_clustered(s, gemm_f32_skinny_lanes_kernel<SP, 1>, g, 32, 64);
      return launch_clustered(s, gemm_f32_skinny_lanes_kernel<SP, 2>, g, 64, pairs < 16 ? 64 : (pairs < 48 ? 128 : 256));
   }
   const bool vec = (reinterpret_cast<uintptr_t>(g.P) & 15) == 0 && g.K % 4 == 0;
   return launch_clustered(s, vec ? gemm_f32_skinny_rows_kernel<SP, 4, 4> : gemm_f32_skinny_rows_kernel<SP, 4, 1>, g, kSkWarps * 4, 128);
}

} // namespace

bool gemm_f32_skinny_ok(const sofie_gemm_f32_desc &d)
{
   // from 64 terms on: below, the adding up of the partial sums is most of the error (9750 x 1 x 35 5.5e-8 from float64 against 4.0e-8). Up to 2^20: a sum is of K / 4096 chunks' sums then,
   // and no more have been compared with the other kernels' (at 262144 terms 0.5 to 0.6 of their error)
   if ((d.M > 8 && d.N > 8) || d.K < 64 || d.K > 1 << 20) return false;
   // Of five to eight columns, 12000 rows and more and up to 300 terms the kernel of two TF32 parts took less time (16384 x 8 x 92 5.9 us, 8.6 here; 16384 x 5 x 272 10.3 and 11.9) with 1.2 to 1.7 times the error: they stay.
   // K is shared by eight blocks at most, which leaves most SMs idle where the long side is not long: split-K, whose slabs are 64, keeps what it is faster at. 8 x 8 x 65536 15.6 us there, 46 here, 1 x 4 x 16385
   // 6.5 and 12, 100 x 8 x 32768 20.5 and 25.7, but 250 x 8 x 32768 32.6 and 27.8, 100 x 8 x 8192 12.1 and 8.8; rows read value by value turn earlier: 8 x 8 x 8193 8.6 and 10.9, 32 x 8 x 3001
   // 5.3 and 5.7, 250 x 8 x 16385 (B stored [N,K]) 16.2 and 16.7.
   if (!splitk_shape_ok(d)) return true;
   const bool long_a = d.M >= d.N, k_contiguous = long_a ? !d.transA : d.transB, by_value = k_contiguous && d.K % 4 != 0;
   const int longer = long_a ? d.M : d.N;
   return d.K <= (by_value && longer <= 64 ? 2560 : 8192) || longer > (by_value ? 256 : 160);
}

int launch_gemm_f32_skinny(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y)
{
   const bool long_a = d.M >= d.N;
   SkinnyArgs g = {};
   g.P = long_a ? A : B, g.Q = long_a ? B : A, g.C = C, g.Y = Y;
   const bool k_contiguous = long_a ? !d.transA : d.transB;
   if (long_a) g.q_s = d.transB ? d.K : 1, g.q_k = d.transB ? 1 : d.N;
   else g.q_s = d.transA ? 1 : d.K, g.q_k = d.transA ? d.M : 1;
   g.y_r = long_a ? d.N : 1, g.y_s = long_a ? 1 : d.N;
   g.R = long_a ? d.M : d.N, g.S = long_a ? d.N : d.M, g.K = d.K;
   g.alpha = d.alpha, g.beta = d.beta, g.bias_kind = d.bias_kind, g.bias_long = !long_a, g.relu = d.relu;
   if (g.S <= 4) return launch_skinny<4>(s, g, k_contiguous);
   return launch_skinny<8>(s, g, k_contiguous);
}

} // namespace sofie
