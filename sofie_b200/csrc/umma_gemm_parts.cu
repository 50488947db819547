// fp32 tensor-core GEMM out of operands that were split beforehand: a first kernel writes the three bfloat16 parts of every value of A
// and B (gemm_parts.cuh) to a workspace of the caller, a second one multiplies them. The products, their order and the error are those
// of umma_gemm_any.cu, whose CTAs each split their own copy of both operands: there a stage of 32 K at 128 columns takes 1.2 us, bound by
// the workers' chain of loading, splitting and storing, here 0.5, for one pass over the operands more (1.8 us per million values) and a
// launch. What bounds it: the MMAs (64 clocks each at 128 columns, 768 a stage; 950 with the partial sums read out of the same tensor
// memory), on large products the power limit (4096 x 4096 x 2048 278 us of 302, 1.48 PFLOP/s in bfloat16 products).
//   * The workspace holds the parts in the shape in which a stage of the second kernel wants them: for every 32 elements of K and every
//     tile of rows, [part][row][32 K] with 64-byte rows, swizzled. A stage is one contiguous copy per operand (cp.async.bulk), whatever
//     layout and alignment the operand has.
//   * One warp copies, one issues the MMAs, eight to sixteen add the partial sums up in registers (the tensor core's sums truncate) and
//     write the tile through a staging buffer of their own, so that the next tile's MMAs run under it.
//   * Few tiles: a cluster of S CTAs shares a tile's K, as in umma_gemm_any.cu.
#include "gemm_parts.cuh"
#include "contract.cuh"

#include <type_traits>

namespace sofie {
namespace umma {
namespace {

// ---------------------------------------------------------------------------------- the split
constexpr int kSplitThreads = 256, kSplitRows = 32, kSplitStages = 4; // a block splits 32 rows x 128 K

// Where the parts of row `row`, stage `kb` start: tiles of `tile` rows, `tiles` of them.
struct PartsLayout {
   unsigned char *p;
   int tile, tiles;
   __device__ __forceinline__ unsigned char *at(int kb, int t) const { return p + ((size_t)kb * tiles + t) * (size_t)(3 * kAnyRow) * tile; }
};

__device__ __forceinline__ void split8(const float (&v)[8], uint4 (&w)[3])
{
   uint32_t p[3][4];
#pragma unroll
   for (int j = 0; j < 4; j++) any_split(v[2 * j], v[2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
   for (int q = 0; q < 3; q++) w[q] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
}

// 32 rows x 128 K of one operand. What bounds it is memory (4 bytes in, 6 out per value); both sides of every copy are whole sectors:
//   rows contiguous: a lane has 16 consecutive K of one row, read 128 bytes of 32 rows at a time and written as 32 bytes per part;
//   K contiguous: a warp has 16 rows of one stage; four lanes write the 64 bytes of a row. Rows that are not 16-byte multiples are read
//   32 floats at a time and turned round in shared memory.
__device__ __forceinline__ void split_block(const AnyOperand &o, const PartsLayout &out, int K, int nkb, int row0, int kb0, float *buf)
{
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kb = kb0 + (warp >> 1), half = warp & 1;
   if (kb >= nkb) return;
   const int tile = row0 / out.tile, in_tile = row0 - tile * out.tile; // tiles are multiples of 32 rows
   unsigned char *dst = out.at(kb, tile);
   const size_t part = (size_t)out.tile * kAnyRow;
   if (o.mode == kRowsContiguous) {
      const int row = row0 + lane, k0 = kb * kAnyKE + 16 * half;
      float v[2][8];
      const float *p = o.p + (long long)k0 * o.ld + row;
#pragma unroll
      for (int j = 0; j < 16; j++, p += o.ld) v[j >> 3][j & 7] = row < o.rows && k0 + j < K ? __ldg(p) : 0.f;
      uint4 w[2][3];
      split8(v[0], w[0]);
      split8(v[1], w[1]);
      const int r = in_tile + lane, s = (r >> 1) & 3; // chunks 2 half and 2 half + 1 lie side by side, in the order the swizzle gives
      unsigned char *q = dst + r * kAnyRow + (((2 * half) ^ (s & 2)) << 4);
#pragma unroll
      for (int i = 0; i < 3; i++) {
         const uint4 a = s & 1 ? w[1][i] : w[0][i], b = s & 1 ? w[0][i] : w[1][i];
         asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(q + i * part), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x),
                      "r"(b.y), "r"(b.z), "r"(b.w)
                      : "memory");
      }
      return;
   }
   const int r = lane >> 2, c = lane & 3, k0 = kb * kAnyKE;
   float v[2][8];
   if (o.mode == kVecK) { // K % 4 == 0
#pragma unroll
      for (int i = 0; i < 2; i++) {
         const int row = row0 + 16 * half + 8 * i + r;
         const float *p = o.p + (long long)row * o.ld + k0 + 8 * c;
#pragma unroll
         for (int h = 0; h < 8; h += 4) {
            const float4 x = row < o.rows && k0 + 8 * c + h < K ? __ldg(reinterpret_cast<const float4 *>(p + h)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i][h] = x.x, v[i][h + 1] = x.y, v[i][h + 2] = x.z, v[i][h + 3] = x.w;
         }
      }
   } else {
      float *mine = buf + warp * 16 * 33;
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; i++) {
         const int row = row0 + 16 * half + i;
         x[i] = row < o.rows && k0 + lane < K ? __ldg(o.p + (long long)row * o.ld + k0 + lane) : 0.f;
      }
#pragma unroll
      for (int i = 0; i < 16; i++) mine[i * 33 + lane] = x[i];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
         for (int j = 0; j < 8; j++) v[i][j] = mine[(8 * i + r) * 33 + 8 * c + j];
   }
#pragma unroll
   for (int i = 0; i < 2; i++) {
      uint4 w[3];
      split8(v[i], w);
      const int rt = in_tile + 16 * half + 8 * i + r;
      unsigned char *q = dst + rt * kAnyRow + ((c ^ ((rt >> 1) & 3)) << 4);
#pragma unroll
      for (int j = 0; j < 3; j++) *reinterpret_cast<uint4 *>(q + j * part) = w[j];
   }
}

// Grid: (groups of 32 rows of A and then of B, blocks of 128 K).
__global__ void __launch_bounds__(kSplitThreads)
split_parts_kernel(AnyOperand A, AnyOperand B, PartsLayout pa, PartsLayout pb, int K, int nkb, int groups_a)
{
   __shared__ float buf[kSplitThreads / 32 * 16 * 33];
   griddep_launch_dependents();
   griddep_wait(A.p, B.p); // the operands may be the previous kernel's output, the workspace may still be read by it
   const int g = blockIdx.x, kb0 = blockIdx.y * kSplitStages;
   if (g < groups_a) split_block(A, pa, K, nkb, g * kSplitRows, kb0, buf);
   else split_block(B, pb, K, nkb, (g - groups_a) * kSplitRows, kb0, buf);
}

// ---------------------------------------------------------------------------------- the product
constexpr int kPartsMaxStages = 6;
constexpr unsigned long long kPartsMaxBytes = 1ull << 30; // of workspace; what needs more is split by every tile for itself

template <int BN>
struct PartsSmem {
   static constexpr int kA = kAnyBM * kAnyRow, kB = BN * kAnyRow;
   static constexpr int kStage = 3 * (kA + kB);
   static constexpr int kWarps = BN == 96 ? 12 : (BN == 32 ? 8 : 16);  // writer warps: kWarps / 4 share the rows of a lane quarter
   static constexpr int kCols = BN / (kWarps / 4);                    // columns of the tile one of them has: 32 or 16
   static constexpr int kWriters = kWarps * 32, kThreads = kWriters + 64; // and the warps that copy and that issue the MMAs
   static constexpr int kStaging = kWarps * 32 * 16 * 4;              // a writer warp's rows leave sixteen columns at a time
   static constexpr int kStages = BN >= 96 ? 4 : (BN == 64 ? 5 : 6);
   static constexpr int kTilePitch = BN + 4;                          // of a partial tile that a cluster adds up
   static_assert(kAnyBM * kTilePitch * 4 <= kStages * kStage, "a partial tile fits in the stages");
   static_assert(kB % 512 == 0, "parts start on whole swizzle atoms");
   static constexpr int kBytes = kStages * kStage + kStaging + 1024;
   static_assert(kBytes <= 232448 - 256, "fits beside the barriers");
};

// A doubtful sum again, as the chain of FMAs.
__device__ __noinline__ float parts_chain(const AnyOperand &A, const AnyOperand &B, int K, int row, int col)
{
   const bool ac = A.mode == kRowsContiguous, bc = B.mode == kRowsContiguous;
   const long long as = ac ? A.ld : 1, bs = bc ? B.ld : 1;
   const float *a = A.p + row * (ac ? 1 : A.ld), *b = B.p + col * (bc ? 1 : B.ld);
   float v = 0.f;
#pragma unroll 1
   for (int k = 0; k < K; k++, a += as, b += bs) v = fmaf(*a, *b, v);
   return v;
}

// any_doubtful() of one or more of N sums, in three instructions each: an infinity or NaN times 0 stays, 2e - 1 leaves the zeros out.
template <int N>
__device__ __forceinline__ bool parts_doubtful(const float (&acc)[N])
{
   float finite = 0.f;
   uint32_t least = 0xFFFFFFFFu;
#pragma unroll
   for (int j = 0; j < N; j++) {
      finite = fmaf(acc[j], 0.f, finite);
      least = min(least, 2 * __float_as_uint(acc[j]) - 1);
   }
   return finite != 0.f || least < 2 * (31u << 23) - 1;
}

// 32 rows of 16 sums in shared memory, 64 bytes a row, the 16-byte words of a row in the order that makes a column of words (written by
// the threads that have the rows) and a row of them (read on the way out) both free of bank conflicts.
__device__ __forceinline__ uint32_t parts_word(int r, int q) { return (uint32_t)(r * 16 + 4 * (q ^ ((r >> 1) & 3))); } // in floats

// Such a block, whose upper left corner is (m0, n0), to global memory: 64 bytes of two rows, or of eight, at a time. What bounds it is
// instruction issue, so what does not change along the rows is decided outside. Loads of C are issued together: as far as the compiler
// knows, a store may change what they read.
template <bool FULL, bool VEC>
__device__ __forceinline__ void parts_write_as(const AnyEpilogue &ep, const float *sums, int m0, int n0, int M, int N, int lane)
{
   constexpr int LANES = VEC ? 4 : 16, STEP = 32 / LANES, BATCH = VEC ? 4 : 8;
   const int q = lane % LANES, r0 = lane / LANES, col = n0 + (VEC ? 4 * q : q);
   if (!FULL && col >= N) return;
   using T = std::conditional_t<VEC, float4, float>;
   auto finish = [&](T v, T c) {
      if constexpr (VEC) return make_float4(any_finish(ep, v.x, c.x), any_finish(ep, v.y, c.y), any_finish(ep, v.z, c.z), any_finish(ep, v.w, c.w));
      else return any_finish(ep, v, c);
   };
   T one{};
   if (ep.bias_kind == 1) {
      if constexpr (VEC) one = make_float4(ep.C[col], ep.C[col + 1], ep.C[col + 2], ep.C[col + 3]);
      else one = ep.C[col];
   }
   const size_t at = (size_t)(m0 + r0) * N + col, step = (size_t)STEP * N;
   float *y = ep.Y + at;
   const float *c = ep.C + at;
#pragma unroll
   for (int i0 = 0; i0 < LANES; i0 += BATCH, y += BATCH * step, c += BATCH * step) {
      T b[BATCH];
#pragma unroll
      for (int i = 0; i < BATCH; i++)
         b[i] = ep.bias_kind == 2 && (FULL || m0 + r0 + (i0 + i) * STEP < M) ? *reinterpret_cast<const T *>(c + i * step) : one;
#pragma unroll
      for (int i = 0; i < BATCH; i++) {
         const int r = r0 + (i0 + i) * STEP;
         const T v = *reinterpret_cast<const T *>(sums + (VEC ? parts_word(r, q) : parts_word(r, q >> 2) + (q & 3)));
         if (FULL || m0 + r < M) *reinterpret_cast<T *>(y + i * step) = finish(v, b[i]);
      }
   }
}
__device__ __forceinline__ void parts_write(const AnyEpilogue &ep, const float *sums, int m0, int n0, int M, int N, int lane)
{
   const bool full = m0 + 32 <= M && n0 + 16 <= N;
   if (ep.vec) {
      if (full) parts_write_as<true, true>(ep, sums, m0, n0, M, N, lane);
      else parts_write_as<false, true>(ep, sums, m0, n0, M, N, lane);
   } else {
      if (full) parts_write_as<true, false>(ep, sums, m0, n0, M, N, lane);
      else parts_write_as<false, false>(ep, sums, m0, n0, M, N, lane);
   }
}

// A full C is read once, at the end of a tile, from memory: its lines are asked for when the tile begins (1000 x 777 x 1333 with new inputs every
// pass 27.1 -> 25.7 us).
__device__ __forceinline__ void parts_prefetch(const float *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The end of a tile that a cluster shares: every rank adds up and writes its rows out of all partial tiles (distributed shared memory, in the
// order of the ranks). With the loads of a thread's whole share issued together, as for a tile of one CTA, it took longer (320 x 1239 x 2149 26.0
// instead of 23.8 us).
template <int BN, bool VEC>
__device__ __forceinline__ void parts_cluster_write(const AnyOperand &A, const AnyOperand &B, const AnyEpilogue &ep, int K, int S, int rank, const unsigned char *smem,
                                                    volatile uint32_t *abort_flag, volatile uint32_t *doubt_flag, int m_tile, int n0, bool writer)
{
   using L = PartsSmem<BN>;
   using T = std::conditional_t<VEC, float4, float>;
   constexpr int W = VEC ? 4 : 1, ROW = BN / W;
   const int rows = kAnyBM / S, r0 = rank * rows, m0 = m_tile + r0, M = A.rows, N = B.rows;
   __syncwarp();
   cluster_sync_all(); // every rank's partial tile is complete
   if (writer && !*abort_flag) {
      const uint32_t base = smem_u32(smem);
      uint32_t doubt = 0;
      for (int q = 0; q < S; q++) doubt |= __float_as_uint(ld_cluster_f1(mapa_shared(smem_u32(const_cast<uint32_t *>(doubt_flag)), (uint32_t)q)));
      auto sums = [&](auto checked) {
#pragma unroll(VEC ? 2 : 4)
         for (int i = threadIdx.x; i < rows * ROW; i += L::kWriters) {
            const int r = i / ROW, c = i % ROW * W, row = m0 + r, col = n0 + c;
            if (row >= M || col >= N) continue;
            T b{}, v{};
            if (ep.bias_kind == 2) b = *reinterpret_cast<const T *>(ep.C + (size_t)row * N + col);
            else if (ep.bias_kind == 1) {
               if constexpr (VEC) b = make_float4(ep.C[col], ep.C[col + 1], ep.C[col + 2], ep.C[col + 3]);
               else b = ep.C[col];
            }
            const uint32_t at = base + (uint32_t)((r0 + r) * L::kTilePitch + c) * 4;
            for (int q = 0; q < S; q++) {
               if constexpr (VEC) {
                  const float4 w = ld_cluster_f4(mapa_shared(at, (uint32_t)q));
                  v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
               } else v += ld_cluster_f1(mapa_shared(at, (uint32_t)q));
            }
            auto sure = [&](float x, int cc) {
               if constexpr (decltype(checked)::value) return any_doubtful(x) ? parts_chain(A, B, K, row, cc) : x;
               else return x;
            };
            if constexpr (VEC)
               *reinterpret_cast<float4 *>(ep.Y + (size_t)row * N + col) = make_float4(any_finish(ep, sure(v.x, col), b.x), any_finish(ep, sure(v.y, col + 1), b.y),
                                                                                       any_finish(ep, sure(v.z, col + 2), b.z), any_finish(ep, sure(v.w, col + 3), b.w));
            else ep.Y[(size_t)row * N + col] = any_finish(ep, sure(v, col), b);
         }
      };
      if (doubt) sums(std::true_type{});
      else sums(std::false_type{});
   }
   __syncwarp();
   cluster_sync_all(); // nobody leaves while its tile is still read
}

// Grid: S x min(tiles, SMs / S) CTAs in clusters of S; with S = 1 a CTA walks tiles (N fastest), with S > 1 it has one.
template <int BN>
__global__ void __launch_bounds__(PartsSmem<BN>::kThreads, 1)
umma_gemm_parts_kernel(AnyOperand A, AnyOperand B, PartsLayout pa, PartsLayout pb, AnyEpilogue ep, int K, int S, uint32_t *status)
{
   using L = PartsSmem<BN>;
   constexpr int COLS = L::kCols;
   constexpr uint32_t TMEM_COLS = 4 * BN <= 128 ? 128 : (4 * BN <= 256 ? 256 : 512); // two buffers of [the leading products | the smaller ones]
   extern __shared__ unsigned char smem_raw[];
   unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
   __shared__ uint64_t full_bar[kPartsMaxStages], empty_bar[kPartsMaxStages], tmem_full[2], tmem_empty[2], drain_bar;
   __shared__ uint32_t tmem_base_holder;
   __shared__ volatile uint32_t abort_flag, doubt_flag; // doubt_flag: a sum of this rank's partial tile is doubtful

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   SOFIE_PROF_DECL
   griddep_launch_dependents();
   const int rank = S > 1 ? (int)cluster_ctarank() : 0;
   const int M = A.rows, N = B.rows;
   const int tiles_n = pb.tiles, num_tiles = pa.tiles * tiles_n;
   const int nkb = (K + kAnyKE - 1) / kAnyKE;
   const int kb0 = (int)((long long)nkb * rank / S), kbn = (int)((long long)nkb * (rank + 1) / S) - kb0; // this rank's stages of a tile
   const int units = (kbn + ep.unit - 1) / ep.unit;
   const int tile0 = blockIdx.x / S, tile_step = gridDim.x / S;

   if (threadIdx.x == 0) {
      for (int s = 0; s < L::kStages; s++) {
         mbar_init(&full_bar[s], 1);
         mbar_init(&empty_bar[s], 1);
      }
      for (int b = 0; b < 2; b++) {
         mbar_init(&tmem_full[b], 1);
         mbar_init(&tmem_empty[b], L::kWriters / 32);
      }
      mbar_init(&drain_bar, 1);
      abort_flag = 0;
      doubt_flag = 0;
      fence_mbar_init();
   }
   if (warp == L::kWriters / 32 + 1) {
      tmem_alloc(&tmem_base_holder, TMEM_COLS);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = tmem_base_holder;
   griddep_wait(); // the parts are the previous kernel's output

   if (warp < L::kWriters / 32) {
      // ---------------- writers ----------------
      const int lane_base = (warp & 3) * 32, col_base = (warp >> 2) * COLS;
      const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)col_base;
      float *staging = reinterpret_cast<float *>(smem + L::kStages * L::kStage) + warp * 32 * 16;
      int u = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
         if (ep.bias_kind == 2) { // the 32 rows and COLS columns that this warp has, or its share of the rank's rows
            const int m0 = (tile / tiles_n) * kAnyBM, n0 = (tile % tiles_n) * BN;
            if (S == 1) {
               const int row = min(m0 + lane_base + lane, M - 1), col = min(n0 + col_base, N - 1);
               parts_prefetch(ep.C + (size_t)row * N + col);
               parts_prefetch(ep.C + (size_t)row * N + min(col + COLS - 1, N - 1));
            } else {
               constexpr int LINES = BN / 32 + 1;
               for (int i = threadIdx.x; i < kAnyBM / S * LINES; i += L::kWriters)
                  parts_prefetch(ep.C + (size_t)min(m0 + rank * (kAnyBM / S) + i / LINES, M - 1) * N + min(n0 + min(i % LINES * 32, BN - 1), N - 1));
            }
         }
         float acc[COLS];
#pragma unroll
         for (int j = 0; j < COLS; j++) acc[j] = 0.f;
         for (int unit = 0; unit < units; unit++, u++) {
            const int buf = u & 1;
            ok = SOFIE_PROF_WAIT(mbar_wait(&tmem_full[buf], (u >> 1) & 1, &abort_flag, status, kStatusWaitAccum, 0x3000 + u));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 8) {
               uint32_t r[8], x[8];
               tmem_ld_32x8(t_row + (uint32_t)(buf * 2 * BN + c0), r);
               tmem_ld_32x8(t_row + (uint32_t)(buf * 2 * BN + BN + c0), x);
               tmem_ld_wait();
#pragma unroll
               for (int j = 0; j < 8; j++) acc[c0 + j] += __uint_as_float(r[j]) + __uint_as_float(x[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
         }
         if (!ok) break;
         if (S > 1) { // the MMAs are done, and with them the copies: the partial tile takes the place of the stages
            float *mine = reinterpret_cast<float *>(smem) + (lane_base + lane) * L::kTilePitch + col_base;
#pragma unroll
            for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4 *>(mine + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
            if (parts_doubtful<COLS>(acc)) doubt_flag = 1;
            break; // one tile per cluster
         }
         const int m0 = (tile / tiles_n) * kAnyBM + lane_base, n0 = (tile % tiles_n) * BN + col_base;
         if (m0 >= M) continue;
         const bool doubt = __any_sync(0xFFFFFFFFu, parts_doubtful<COLS>(acc));
#pragma unroll
         for (int c0 = 0; c0 < COLS; c0 += 16) {
            if (n0 + c0 < N) {
#pragma unroll
               for (int q = 0; q < 4; q++)
                  *reinterpret_cast<float4 *>(staging + parts_word(lane, q)) = make_float4(acc[c0 + 4 * q], acc[c0 + 4 * q + 1], acc[c0 + 4 * q + 2], acc[c0 + 4 * q + 3]);
               if (doubt && m0 + lane < M)
#pragma unroll 1
                  for (int j = 0; j < 16 && n0 + c0 + j < N; j++) {
                     float *v = staging + parts_word(lane, j >> 2) + (j & 3);
                     if (any_doubtful(*v)) *v = parts_chain(A, B, K, m0 + lane, n0 + c0 + j);
                  }
               __syncwarp();
               parts_write(ep, staging, m0, n0 + c0, M, N, lane);
               __syncwarp();
            }
         }
      }
   } else if (warp == L::kWriters / 32) {
      // ---------------- copies ----------------
      int g = 0, s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
         const unsigned char *a = pa.at(kb0, tile / tiles_n), *b = pb.at(kb0, tile % tiles_n);
         const size_t da = (size_t)pa.tiles * 3 * L::kA, db = (size_t)pb.tiles * 3 * L::kB;
         for (int kb = 0; kb < kbn; kb++, g++, a += da, b += db, ring_next(s, ph, L::kStages)) {
            ok = SOFIE_PROF_WAIT(mbar_wait_warp(&empty_bar[s], ph ^ 1, &abort_flag, status, kStatusWaitEmpty, g));
            if (!ok) break;
            warp_expect_tx(&full_bar[s], L::kStage);
            warp_bulk_load(smem + s * L::kStage, a, 3 * L::kA, &full_bar[s]);
            warp_bulk_load(smem + s * L::kStage + 3 * L::kA, b, 3 * L::kB, &full_bar[s]);
         }
      }
      drain_copies(full_bar, s, ph, g, L::kStages);
   } else {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc_wide = make_idesc<kBF16>(kAnyBM, 2 * BN), idesc = make_idesc<kBF16>(kAnyBM, BN);
      int s = 0, u = 0;
      uint32_t ph = 0;
      WarpWait wait;
      for (int tile = tile0; tile < num_tiles; tile += tile_step) {
         for (int kc = 0; kc < kbn; kc += ep.unit, u++) {
            const int buf = u & 1;
            wait(&tmem_empty[buf], ((u >> 1) & 1) ^ 1);
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 2 * BN);
            const int kce = min(kbn, kc + ep.unit);
            for (int kb = kc; kb < kce; kb++, ring_next(s, ph, L::kStages)) {
               wait(&full_bar[s], ph);
               tc_fence_after();
               const uint32_t base = smem_u32(smem + s * L::kStage);
               const uint64_t da0 = make_smem_desc(base, kAnyRow), da1 = make_smem_desc(base + L::kA, kAnyRow), da2 = make_smem_desc(base + 2 * L::kA, kAnyRow);
               const uint64_t db0 = make_smem_desc(base + 3 * L::kA, kAnyRow), db1 = make_smem_desc(base + 3 * L::kA + L::kB, kAnyRow),
                              db2 = make_smem_desc(base + 3 * L::kA + 2 * L::kB, kAnyRow);
#pragma unroll
               for (int k = 0; k < 2; k++) {
                  const uint64_t koff = (uint64_t)(2 * k);
                  warp_mma<kBF16>(d_tmem, da0 + koff, db0 + koff, idesc_wide, (kb == kc && k == 0) ? 0u : 1u); // and the second part of B behind it
                  warp_mma<kBF16>(d_tmem + BN, da1 + koff, db0 + koff, idesc, 1);
                  warp_mma<kBF16>(d_tmem + BN, da1 + koff, db1 + koff, idesc, 1);
                  warp_mma<kBF16>(d_tmem + BN, da0 + koff, db2 + koff, idesc, 1);
                  warp_mma<kBF16>(d_tmem + BN, da2 + koff, db0 + koff, idesc, 1);
               }
               wait.commit(&empty_bar[s]);
            }
            wait.commit(&tmem_full[buf]);
         }
      }
      wait.finish(&drain_bar, &abort_flag, status, kStatusWaitFull, u);
   }
   SOFIE_PROF_REPORT(warp < L::kWriters / 32 ? "writer" : (warp == L::kWriters / 32 ? "copy" : "mma"));
   if (S > 1) {
      const int m0 = (tile0 / tiles_n) * kAnyBM, n0 = (tile0 % tiles_n) * BN;
      const bool writer = warp < L::kWriters / 32;
      if (ep.vec) parts_cluster_write<BN, true>(A, B, ep, K, S, rank, smem, &abort_flag, &doubt_flag, m0, n0, writer);
      else parts_cluster_write<BN, false>(A, B, ep, K, S, rank, smem, &abort_flag, &doubt_flag, m0, n0, writer);
   }
   tc_fence_before();
   __syncthreads();
   if (warp == L::kWriters / 32 + 1) {
      __syncwarp();
      tc_fence_after();
      tmem_dealloc(tmem_base, TMEM_COLS);
   }
}

template <int BN>
int launch_parts(cudaStream_t s, const AnyOperand &A, const AnyOperand &B, const AnyEpilogue &ep, int K, int S, unsigned char *scratch)
{
   using L = PartsSmem<BN>;
   auto kern = umma_gemm_parts_kernel<BN>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), L::kBytes));
   uint32_t *status = device_status_word(s);
   if (!status) return fail(SOFIE_CUDA_ERR_CUDA, "cannot allocate the device status word");
   const int nkb = ceil_div(K, kAnyKE);
   const PartsLayout pa{scratch, kAnyBM, ceil_div(A.rows, kAnyBM)};
   const PartsLayout pb{scratch + (size_t)nkb * pa.tiles * 3 * L::kA, BN, ceil_div(B.rows, BN)};
   const int ga = ceil_div(A.rows, kSplitRows), gb = ceil_div(B.rows, kSplitRows);
   SOFIE_CUDA_TRY(launch_dependent(split_parts_kernel, dim3(ga + gb, ceil_div(nkb, kSplitStages)), dim3(kSplitThreads), 0, s, A, B, pa, pb, K, nkb, ga));
   const int tiles = pa.tiles * pb.tiles, grid = S > 1 ? tiles * S : (tiles < kNumSMs ? tiles : kNumSMs);
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(grid);
   cfg.blockDim = dim3(L::kThreads);
   cfg.dynamicSmemBytes = L::kBytes;
   cfg.stream = s;
   cudaLaunchAttribute attr[2];
   attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
   attr[1].id = cudaLaunchAttributeClusterDimension;
   attr[1].val.clusterDim.x = (unsigned)S;
   attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
   cfg.attrs = attr;
   cfg.numAttrs = S > 1 ? 2 : 1;
   SOFIE_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, A, B, pa, pb, ep, K, S, status));
   set_last_engine(SOFIE_ENGINE_TCGEN05);
   return SOFIE_CUDA_OK;
}

struct PartsPlan {
   int BN = 0, S = 1; // BN = 0: the product is faster on the other kernels
   size_t bytes = 0;
};

// Tile width and clusters along K by the time they take, in ns, fitted to 22700 runs of 2800 products (each at every width and cluster size; the
// choice is 1.2 % above the best of them in the mean): both launches, the split of (M + N) x K values, a stage of 32 K, a tile's end (longer
// where rows of Y are not whole 16-byte words and where C is of Y's shape), under which the next tile's stages run, or the exchange within
// a cluster; at least the writes of Y. `room` is what clusters of 1 / 2 / 4 / 8 found at the time of the fit, the same on every card as kClusterRoom is.
// Against the other kernels' estimate, which is 20 % low in the mean: the split pays from about 2^20 outputs or 2^24 FMAs a tile on. 1000 x 777 x
// 1333 with A transposed and a full bias 39 -> 25.7 us, 4096 x 4096 x 2048 522 -> 302, 785 x 2853 x 683 64 -> 35, 16384 x 777 x 64 59 -> 32; of the 2800
// (M and N from 48 on) it takes three in five, and 0.3 % of them are more than 3 % slower. With 32 to 47 rows
// or columns it takes a fifth of 260, 0.84 of the other kernels' time in the mean, but below K = 256 six of 12 took 3 to 15 % longer (41 x 17142 x 180 14.6 us
// without, 16.7 with): those are left to the others.
PartsPlan parts_plan(const sofie_gemm_f32_desc &d)
{
   static const int widths[4] = {128, 96, 64, 32}, stage[4] = {505, 441, 404, 347}, end[4] = {1908, 1421, 586, 214}, room[4] = {kNumSMs, kNumSMs, 132, 96};
   PartsPlan p;
   const int tm = ceil_div(d.M, kAnyBM), nkb = ceil_div(d.K, kAnyKE);
   const bool full = d.bias_kind == 2, tma = !d.transA && d.transB && d.K % 4 == 0;
   if (d.M < 32 || d.N < 32 || (!forced_engine() && gemm_f32_tiny_ok(d))) return p;  // hardly a tile: not measured, and the skinny products have more precise kernels
   if (d.K < 256 && (d.M < 48 || d.N < 48)) return p;
   if (d.K < 48) return p; // the writes of Y count, and short K leaves the split little to save: 16384 x 4093 x 8 169 us either way
   const long long split = 4560 + 1817 * (((long long)d.M + d.N) * nkb * kAnyKE) / 1000000, out = 1361 * ((long long)d.M * d.N * (full ? 2 : 1)) / 1000000;
   long long best = -1;
   for (int w = 0; w < 4; w++) {
      if (widths[w] > 32 && widths[w] / 2 >= d.N) continue; // more than half of the tile would be padding
      const long long tiles = (long long)tm * ceil_div(d.N, widths[w]);
      const long long tail = (long long)end[w] * (d.N % 4 ? 167 : 100) / 100 * (full ? 135 : 100) / 100;
      for (int i = 0, q = 1; i < 4 && (q == 1 || (nkb >= 2 * q && tiles * q <= 3 * kNumSMs)); i++, q *= 2) {
         const long long waves = (tiles * q + room[i] - 1) / room[i], work = (long long)ceil_div(nkb, q) * stage[w];
         const long long main = q == 1 ? waves * (1082 + (work > tail ? work : tail)) + (work > tail ? tail : work) : waves * (work + tail + 3414 + 152 * q);
         const long long time = split + (main > out ? main : out);
         if (best < 0 || time < best) best = time, p.BN = widths[w], p.S = q;
      }
   }
   const unsigned long long tiles_n = ceil_div(d.N, p.BN);
   const unsigned long long bytes = (unsigned long long)nkb * 3 * kAnyRow * ((unsigned long long)tm * kAnyBM + tiles_n * p.BN);
   if (best * 100 >= gemm_f32_whole_ns(d, tma) * 105 || bytes > kPartsMaxBytes || tm * tiles_n > 0x7FFFFFFF / 8 || ceil_div(nkb, kSplitStages) > 65535) p.BN = 0;
   else p.bytes = (size_t)bytes;
   return p;
}

} // namespace
} // namespace umma

size_t gemm_f32_parts_bytes(const sofie_gemm_f32_desc &d) { return umma::parts_plan(d).bytes; }

int launch_gemm_f32_parts(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y, void *scratch, size_t bytes)
{
   using namespace umma;
   const PartsPlan p = parts_plan(d);
   if (!p.BN || bytes < p.bytes || (reinterpret_cast<uintptr_t>(scratch) & 127)) return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "not a product of split operands");
   auto aligned = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
   const bool vec_k = d.K % 4 == 0;
   const AnyOperand a{A, d.transA ? d.M : d.K, d.M, d.transA ? kRowsContiguous : (vec_k && aligned(A) ? kVecK : kScalarK)};
   const AnyOperand b{B, d.transB ? d.K : d.N, d.N, !d.transB ? kRowsContiguous : (vec_k && aligned(B) ? kVecK : kScalarK)};
   const AnyEpilogue ep{d.alpha, d.beta, C, Y, d.bias_kind, d.relu, d.N % 4 == 0 && aligned(Y) && (d.bias_kind != 2 || aligned(C)), d.K >= 1024 ? 8 : (d.K >= 256 ? 4 : 3)};
   unsigned char *w = static_cast<unsigned char *>(scratch);
   switch (p.BN) {
   case 128: return launch_parts<128>(s, a, b, ep, d.K, p.S, w);
   case 96: return launch_parts<96>(s, a, b, ep, d.K, p.S, w);
   case 64: return launch_parts<64>(s, a, b, ep, d.K, p.S, w);
   default: return launch_parts<32>(s, a, b, ep, d.K, p.S, w);
   }
}

} // namespace sofie
