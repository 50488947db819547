// fp32 tensor-core GEMM for the operands TMA cannot fetch -- a transposed A, B stored [K,N], rows that are not multiples of 16
// bytes, unaligned bases -- and for few tiles with a long K. Without it these products are chains of fp32 FMAs on the CUDA cores, and
// its results are no further from the exact ones than theirs: every value is split into three bfloat16 parts that add up to it (8 + 8 + 8
// bits), and the six products of parts that reach into 24 bits are summed by the tensor core, the leading ones apart from the others
// (what is dropped is below 2^-25 of a product). The tensor core's sums truncate, so they are added to fp32 registers every few stages:
// every 96 elements of K below K = 256, where a chain of FMAs has made few roundings too, every 128 up to K = 1023, every 256 from there.
// Error against float64 over that of the chain of FMAs, N(0,1) operands: at most 0.57 below K = 32, 0.62 below 96, 0.55 below 256, 0.44 below
// 1024, 0.39 beyond; operands of one sign: 0.68, 0.95, 0.84, 0.72, 0.71. (Two TF32 parts, 22 bits, and sums of 256, N(0,1): 1.7 up to K = 256.)
// Infinities, NaNs and the ends of fp32's range give what the chain gives (any_doubtful below).
//   * sixteen worker warps read the operands themselves, split them in registers and write the parts where the MMA's swizzled K-major
//     descriptors expect them. A unit of work is eight consecutive K of one row: two 16-byte loads, eight scalar loads (rows that are
//     not 16-byte multiples), or eight loads of consecutive rows (K is not the contiguous dimension), always one conflict-free
//     16-byte store per part. Groups of them take the stages in turn: while one splits and stores, the others' loads are in flight
//     (one group with two stages of loads in flight was bound by their latency). The same warps add the partial sums up in registers
//     and write the tile.
//   * B's parts lie one behind the other, so that the first instruction of a K step multiplies A's first part with two of B's at once,
//     into neighbouring columns of the accumulator.
//   * a cluster of S CTAs shares one output tile: each takes a S-th of K, leaves its partial tile in shared memory, and adds up and
//     writes a S-th of the rows out of all of them (distributed shared memory, fixed order). No scratch buffer, one launch.
// What bounds it is the workers' chain of loading, splitting and storing; the MMAs of a stage take 770 clocks at 128 columns.
// The tile goes out through shared memory, so stores (and a bias of the output's shape) are contiguous along rows for every N.
#include "gemm_parts.cuh"
#include "contract.cuh"

namespace sofie {
namespace umma {
namespace {

constexpr int kAnyWorkers = 16 * 32;
// Groups of worker warps that take the stages in turn. Four were 5 to 10 % faster at 32 columns with a long K and as much slower with a
// short one (the pipeline takes longer to start), and spilled at 64 columns. Turned tiles (K >= 512, below) have four: 27 x 2512 x 3682 28.1 -> 26.2 us, 13 x 1652 x 2420 13.6 -> 12.9,
// 15 x 1446 x 1006 10.4 -> 10.7.
constexpr int kAnyGroups = 2, kAnyTurnedGroups = 4;
constexpr int kAnyThreads = kAnyWorkers + 32; // and the warp that issues the MMAs
constexpr int kAnyMaxStages = 5;

template <int BN>
struct AnySmem {
   static constexpr int kA = kAnyBM * kAnyRow, kB = BN * kAnyRow;
   static constexpr int kStage = 3 * (kA + kB);                       // the three parts of both operands
   static constexpr int kPitch = BN + 4;                              // floats per row of the outgoing tile, which takes the
   static constexpr int kTile = kAnyBM * kPitch * 4;                  // place of the stages when their MMAs are done
   static constexpr int kStages = BN == 128 ? 4 : 5;
   static_assert(kTile <= kStages * kStage, "the tile fits in the stages");
   static_assert(kB % 512 == 0, "parts start on whole swizzle atoms");
   static constexpr int kBytes = kStages * kStage + 1024;
};

// One thread's share of the tiles of an operand with R rows: U units, a unit being K chunk `c` (eight floats) of row `r`.
//   K contiguous: four lanes cover the 128 bytes of one row; the thread's units are T / 4 rows apart, in the same chunk.
//   Rows contiguous: lanes cover consecutive rows; the thread's units are in one row, T / R chunks apart (T threads per group).
// Either way the 16-byte stores of eight lanes fall into eight different bank groups, and everything that depends on the thread is
// worked out once per tile: the loops below are the loads, an addition and the split per unit (with the addresses taken from the unit
// number the loaders were bound by instruction issue). With 32 rows half of the threads have no unit.
template <int R, int T>
struct AnyLoader {
   static constexpr int U = R * 4 / T > 0 ? R * 4 / T : 1;
   static constexpr bool kAll = R * 4 >= T;                       // every thread has a unit
   static constexpr int kRowStep = T / 4, kChunkStep = T / R;     // between the units of a thread
   const float *p = nullptr; // the thread's first element at K = 0 of the tile
   uint32_t at = 0;          // byte offset of its first unit in the tile
   uint32_t ok = 0;          // bit i: the row of unit i exists
   float v[U][8];

   __device__ __forceinline__ void place(const AnyOperand &o, int t)
   {
      const int r = o.mode == kRowsContiguous ? (t & (R - 1)) : (t >> 2), c = o.mode == kRowsContiguous ? t / R : (t & 3);
      at = (uint32_t)(r * kAnyRow + ((c ^ ((r >> 1) & 3)) << 4)); // the 64-byte swizzle the descriptors name
   }
   __device__ __forceinline__ void tile(const AnyOperand &o, int row0, int t)
   {
      if (o.mode == kRowsContiguous) {
         const int r = row0 + (t & (R - 1));
         ok = r < o.rows && (kAll || t < R * 4) ? ~0u : 0u;
         p = o.p + r + (long long)(8 * (t / R)) * o.ld;
      } else {
         const int r = row0 + (t >> 2);
         ok = 0;
#pragma unroll
         for (int i = 0; i < U; i++) ok |= (r + kRowStep * i < o.rows && (kAll || t < R * 4) ? 1u : 0u) << i;
         p = o.p + (long long)r * o.ld + 8 * (t & 3);
      }
   }
   // the units of the stage that starts at element k0 of K; K ends at kend
   __device__ __forceinline__ void load(const AnyOperand &o, int k0, int kend, int t)
   {
#pragma unroll
      for (int i = 0; i < U; i++)
#pragma unroll
         for (int j = 0; j < 8; j++) v[i][j] = 0.f;
      if (o.mode == kRowsContiguous) {
         const float *q = p + (long long)k0 * o.ld;
         int left = ok ? kend - k0 - 8 * (t / R) : 0; // elements of K from the thread's first chunk on
#pragma unroll
         for (int i = 0; i < U; i++, left -= 8 * kChunkStep) {
            const float *e = q + (long long)(8 * kChunkStep * i) * o.ld;
#pragma unroll
            for (int j = 0; j < 8; j++, e += o.ld)
               if (left > j) v[i][j] = *e;
         }
      } else {
         const float *q = p + k0;
         const long long step = kRowStep * o.ld;
         const int left = kend - k0 - 8 * (t & 3);
         if (o.mode == kVecK) { // K % 4 == 0 and kend % 4 == 0
#pragma unroll
            for (int i = 0; i < U; i++, q += step)
#pragma unroll
               for (int h = 0; h < 8; h += 4)
                  if (((ok >> i) & 1) && left > h) {
                     const float4 w = *reinterpret_cast<const float4 *>(q + h);
                     v[i][h] = w.x, v[i][h + 1] = w.y, v[i][h + 2] = w.z, v[i][h + 3] = w.w;
                  }
         } else {
#pragma unroll
            for (int i = 0; i < U; i++, q += step)
#pragma unroll
               for (int j = 0; j < 8; j++)
                  if (((ok >> i) & 1) && left > j) v[i][j] = q[j];
         }
      }
   }
   // the parts lie `part` bytes apart
   __device__ __forceinline__ void store(const AnyOperand &o, unsigned char *p0, int part, int t)
   {
      if (!kAll && t >= R * 4) return;
#pragma unroll
      for (int i = 0; i < U; i++) {
         // units a multiple of 8 rows apart keep their place in the swizzle pattern; chunks kChunkStep apart flip its upper bit
         const uint32_t off = o.mode == kRowsContiguous ? (at ^ (uint32_t)(i * kChunkStep * 16)) : (at + (uint32_t)(i * kRowStep * kAnyRow));
         uint32_t w[3][4];
#pragma unroll
         for (int j = 0; j < 4; j++) any_split(v[i][2 * j], v[i][2 * j + 1], w[0][j], w[1][j], w[2][j]);
#pragma unroll
         for (int q = 0; q < 3; q++) *reinterpret_cast<uint4 *>(p0 + q * part + off) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
      }
   }
};

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kAnyWorkers) : "memory"); }

// any_write below for a tile with doubtful sums.
template <int BN, bool TURNED>
__device__ __forceinline__ void any_write_checked(const AnyOperand &A, const AnyOperand &B, int K, const AnyEpilogue &ep, const float *tile, int S, int r0, int rows, int m0, int n0)
{
   constexpr int P = AnySmem<BN>::kPitch;
   const uint32_t base = smem_u32(tile);
   const long long as = A.mode == kRowsContiguous ? A.ld : 1, ar = A.mode == kRowsContiguous ? 1 : A.ld;
   const long long bs = B.mode == kRowsContiguous ? B.ld : 1, br = B.mode == kRowsContiguous ? 1 : B.ld;
#pragma unroll 1
   for (int i = threadIdx.x; i < rows * BN; i += kAnyWorkers) {
      const int r = r0 + i / BN, c = i % BN, row = m0 + r, col = n0 + c;
      if (row >= A.rows || col >= B.rows) continue;
      float v = 0.f;
      for (int q = 0; q < S; q++) v += S == 1 ? tile[r * P + c] : ld_cluster_f1(mapa_shared(base + (uint32_t)(r * P + c) * 4, (uint32_t)q));
      if (any_doubtful(v)) {
         const float *a = A.p + row * ar, *b = B.p + col * br;
         v = 0.f;
#pragma unroll 1
         for (int k = 0; k < K; k++, a += as, b += bs) v = fmaf(*a, *b, v);
      }
      const size_t y = TURNED ? (size_t)col * A.rows + row : (size_t)row * B.rows + col;
      const float bias = ep.bias_kind == 1 ? ep.C[TURNED ? row : col] : (ep.bias_kind == 2 ? ep.C[y] : 0.f);
      ep.Y[y] = any_finish(ep, v, bias);
   }
}

// Rows [r0, r0 + rows) of the tile at (m0, n0), the sum of the S partial tiles, to global memory. TURNED: the operands have changed places, the tile's rows are Y's columns;
// a flag in the place of the template's cost every other product 0.2 us.
template <int BN, bool TURNED>
__device__ __forceinline__ void any_write(const AnyEpilogue &ep, const float *tile, int S, int r0, int rows, int m0, int n0, int M, int N)
{
   constexpr int P = AnySmem<BN>::kPitch;
   const uint32_t base = smem_u32(tile);
   if (!TURNED && ep.vec) {
#pragma unroll 2
      for (int i = threadIdx.x; i < rows * (BN / 4); i += kAnyWorkers) {
         const int r = r0 + i / (BN / 4), c = (i % (BN / 4)) * 4, row = m0 + r, col = n0 + c;
         if (row >= M || col >= N) continue;
         float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
         if (ep.bias_kind == 1) b = make_float4(ep.C[col], ep.C[col + 1], ep.C[col + 2], ep.C[col + 3]);
         else if (ep.bias_kind == 2) b = *reinterpret_cast<const float4 *>(ep.C + (size_t)row * N + col);
         float4 v;
         if (S == 1) {
            v = *reinterpret_cast<const float4 *>(tile + r * P + c);
         } else {
            v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int q = 0; q < S; q++) {
               const float4 w = ld_cluster_f4(mapa_shared(base + (uint32_t)(r * P + c) * 4, (uint32_t)q));
               v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
            }
         }
         *reinterpret_cast<float4 *>(ep.Y + (size_t)row * N + col) =
            make_float4(any_finish(ep, v.x, b.x), any_finish(ep, v.y, b.y), any_finish(ep, v.z, b.z), any_finish(ep, v.w, b.w));
      }
   } else {
      const int log_rows = __ffs(rows) - 1; // a power of two
#pragma unroll 4
      for (int i = threadIdx.x; i < rows * BN; i += kAnyWorkers) {
         // threads along what is contiguous in Y
         const int r = r0 + (TURNED ? i & (rows - 1) : i / BN), c = TURNED ? i >> log_rows : i % BN, row = m0 + r, col = n0 + c;
         if (row >= M || col >= N) continue;
         const size_t y = TURNED ? (size_t)col * M + row : (size_t)row * N + col;
         const float b = ep.bias_kind == 1 ? ep.C[TURNED ? row : col] : (ep.bias_kind == 2 ? ep.C[y] : 0.f);
         float v = 0.f;
         if (S == 1) v = tile[r * P + c];
         else
            for (int q = 0; q < S; q++) v += ld_cluster_f1(mapa_shared(base + (uint32_t)(r * P + c) * 4, (uint32_t)q));
         ep.Y[y] = any_finish(ep, v, b);
      }
   }
}

// Grid: S x min(tiles, SMs / S) CTAs in clusters of S; with S = 1 a CTA walks tiles (N fastest), with S > 1 it has one.
template <int BN, bool TURNED>
__global__ void __launch_bounds__(kAnyThreads, 1)
umma_gemm_any_kernel(AnyOperand A, AnyOperand B, AnyEpilogue ep, int K, int S, uint32_t *status)
{
   using L = AnySmem<BN>;
   constexpr int G = TURNED ? kAnyTurnedGroups : kAnyGroups, GT = kAnyWorkers / G; // groups and their threads
   constexpr int QUARTER = BN / 4;       // columns of the tile a worker warp adds up
   constexpr uint32_t TMEM_COLS = 4 * BN; // two buffers of [the leading products | the smaller ones]
   extern __shared__ unsigned char smem_raw[];
   unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
   float *tile_out = reinterpret_cast<float *>(smem);
   __shared__ uint64_t full_bar[kAnyMaxStages], empty_bar[kAnyMaxStages], tmem_full[2], tmem_empty[2], drain_bar;
   __shared__ uint32_t tmem_base_holder;
   __shared__ volatile uint32_t abort_flag, doubt_flag; // doubt_flag: a sum of this CTA's tile is doubtful

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   SOFIE_PROF_DECL
   griddep_launch_dependents();
   const int rank = S > 1 ? (int)cluster_ctarank() : 0;
   const int M = A.rows, N = B.rows;
   const int tiles_n = (N + BN - 1) / BN, num_tiles = ((M + kAnyBM - 1) / kAnyBM) * tiles_n;
   const int nkb = (K + kAnyKE - 1) / kAnyKE;
   const int kb0 = (int)((long long)nkb * rank / S), kbn = (int)((long long)nkb * (rank + 1) / S) - kb0; // this rank's stages of a tile
   const int kend = min(K, (kb0 + kbn) * kAnyKE);
   const int unit_stages = ep.unit, units = (kbn + unit_stages - 1) / unit_stages;
   const int tile0 = blockIdx.x / S, tile_step = gridDim.x / S;
   auto a_part = [&](int s, int q) { return smem + s * L::kStage + q * L::kA; };
   auto b_part = [&](int s, int q) { return smem + s * L::kStage + 3 * L::kA + q * L::kB; };

   if (threadIdx.x == 0) {
      for (int s = 0; s < L::kStages; s++) {
         mbar_init(&full_bar[s], GT / 32);
         mbar_init(&empty_bar[s], 1);
      }
      for (int b = 0; b < 2; b++) {
         mbar_init(&tmem_full[b], 1);
         mbar_init(&tmem_empty[b], kAnyWorkers / 32);
      }
      mbar_init(&drain_bar, 1);
      abort_flag = 0;
      doubt_flag = 0;
      fence_mbar_init();
   }
   if (warp == kAnyWorkers / 32) {
      tmem_alloc(&tmem_base_holder, TMEM_COLS);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = tmem_base_holder;
   griddep_wait(); // any of the operands may be the previous kernel's output

   if (warp < kAnyWorkers / 32) {
      // ---------------- workers ----------------
      const int group = threadIdx.x / GT, t = threadIdx.x % GT;
      const int lane_base = (warp & 3) * 32, col_base = (warp >> 2) * QUARTER;
      const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)col_base;
      AnyLoader<kAnyBM, GT> la;
      AnyLoader<BN, GT> lb;
      la.place(A, t);
      lb.place(B, t);
      // Stages are numbered through all tiles of this CTA; the group's own are every G-th. `lt`, `lk`: the stage whose loads are
      // issued next; g: the stage the group stores next.
      int lt = tile0, lk = group, placed = -1;
      auto load = [&] {
         while (lk >= kbn) {
            lk -= kbn;
            lt += tile_step;
         }
         if (lt >= num_tiles) return;
         if (lt != placed) {
            placed = lt;
            la.tile(A, (lt / tiles_n) * kAnyBM, t);
            lb.tile(B, (lt % tiles_n) * BN, t);
         }
         la.load(A, (kb0 + lk) * kAnyKE, kend, t);
         lb.load(B, (kb0 + lk) * kAnyKE, kend, t);
         lk += G;
      };
      load();
      int g = group, s = group % L::kStages, u = 0, first = 0; // first: number of the current tile's first stage
      uint32_t ph = (uint32_t)(group / L::kStages) & 1u;
      // a warp whose wait gave up goes on to the end with the others (their barriers count it); its later waits return at once
      for (int tile = tile0; tile < num_tiles; tile += tile_step, first += kbn) {
         const int m0 = (tile / tiles_n) * kAnyBM, n0 = (tile % tiles_n) * BN;
         float acc[QUARTER];
#pragma unroll
         for (int j = 0; j < QUARTER; j++) acc[j] = 0.f;
         auto promote = [&] {
            const int buf = u & 1;
            if (SOFIE_PROF_WAIT(mbar_wait(&tmem_full[buf], (u >> 1) & 1, &abort_flag, status, kStatusWaitAccum, 0x3000 + u))) {
               tc_fence_after();
#pragma unroll
               for (int c0 = 0; c0 < QUARTER; c0 += 8) {
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
            u++;
         };
         int unit = 0; // units of this tile already added up
         for (; g < first + kbn; g += G) {
            // the partial sum of a unit is collected a ring's length after its last stage was stored: its MMAs are done by then
            if (g - first >= (unit + 1) * unit_stages + L::kStages) {
               promote();
               unit++;
            }
            if (SOFIE_PROF_WAIT(mbar_wait(&empty_bar[s], ph ^ 1, &abort_flag, status, kStatusWaitEmpty, g))) {
               la.store(A, a_part(s, 0), L::kA, t);
               lb.store(B, b_part(s, 0), L::kB, t);
               // visible to the tensor core: before the next loads are issued, because the fence would wait for them
               fence_proxy_async();
               __syncwarp();
               if (lane == 0) mbar_arrive(&full_bar[s]);
            }
            load();
            for (int i = 0; i < G; i++) ring_next(s, ph, L::kStages);
         }
         for (; unit < units; unit++) promote();
         workers_sync(); // all units added up: the tile's MMAs are done and its stages free
         float *mine = tile_out + (lane_base + lane) * L::kPitch + col_base;
#pragma unroll
         for (int j = 0; j < QUARTER; j += 4) *reinterpret_cast<float4 *>(mine + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
         // any_doubtful() of all of them in three instructions each: an infinity or NaN times 0 stays, 2e - 1 leaves the zeros out
         float finite = 0.f;
         uint32_t least = 0xFFFFFFFFu;
#pragma unroll
         for (int j = 0; j < QUARTER; j++) {
            finite = fmaf(acc[j], 0.f, finite);
            least = min(least, 2 * __float_as_uint(acc[j]) - 1);
         }
         if (finite != 0.f || least < 2 * (31u << 23) - 1) doubt_flag = 1;
         workers_sync();
         if (S > 1) break; // one tile per cluster: it is summed up below
         if (!abort_flag) {
            if (doubt_flag) any_write_checked<BN, TURNED>(A, B, K, ep, tile_out, 1, 0, kAnyBM, m0, n0);
            else any_write<BN, TURNED>(ep, tile_out, 1, 0, kAnyBM, m0, n0, M, N);
         }
         workers_sync(); // the tile has been read: its place is the stages' again
         if (threadIdx.x == 0) doubt_flag = 0; // set again behind the next tile's first workers_sync
      }
   } else {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc_wide = make_idesc<kBF16>(kAnyBM, 2 * BN), idesc = make_idesc<kBF16>(kAnyBM, BN);
      int s = 0, u = 0;
      uint32_t ph = 0;
      WarpWait wait;
      for (int tile = tile0; tile < num_tiles; tile += tile_step) {
         for (int kc = 0; kc < kbn; kc += unit_stages, u++) {
            const int buf = u & 1;
            wait(&tmem_empty[buf], ((u >> 1) & 1) ^ 1);
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 2 * BN);
            const int kce = min(kbn, kc + unit_stages);
            for (int kb = kc; kb < kce; kb++, ring_next(s, ph, L::kStages)) {
               wait(&full_bar[s], ph);
               tc_fence_after();
               const uint64_t da0 = make_smem_desc(smem_u32(a_part(s, 0)), kAnyRow), da1 = make_smem_desc(smem_u32(a_part(s, 1)), kAnyRow);
               const uint64_t da2 = make_smem_desc(smem_u32(a_part(s, 2)), kAnyRow), db0 = make_smem_desc(smem_u32(b_part(s, 0)), kAnyRow);
               const uint64_t db1 = make_smem_desc(smem_u32(b_part(s, 1)), kAnyRow), db2 = make_smem_desc(smem_u32(b_part(s, 2)), kAnyRow);
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
      wait.finish(&drain_bar, &abort_flag, status, kStatusWaitConv, u);
   }
   SOFIE_PROF_REPORT(warp < kAnyWorkers / 32 ? "worker" : "mma");
   if (S > 1) {
      // every rank's partial tile is complete; each sums up and writes its share of the rows
      __syncwarp();
      cluster_sync_all();
      if (warp < kAnyWorkers / 32 && !abort_flag) {
         uint32_t doubt = 0;
         for (int q = 0; q < S; q++) doubt |= __float_as_uint(ld_cluster_f1(mapa_shared(smem_u32(const_cast<uint32_t *>(&doubt_flag)), (uint32_t)q)));
         const int r0 = rank * (kAnyBM / S), m0 = (tile0 / tiles_n) * kAnyBM, n0 = (tile0 % tiles_n) * BN;
         if (doubt) any_write_checked<BN, TURNED>(A, B, K, ep, tile_out, S, r0, kAnyBM / S, m0, n0);
         else any_write<BN, TURNED>(ep, tile_out, S, r0, kAnyBM / S, m0, n0, M, N);
      }
      __syncwarp();
      cluster_sync_all(); // nobody leaves while its tile is still read
   }
   tc_fence_before();
   __syncthreads();
   if (warp == kAnyWorkers / 32) {
      __syncwarp();
      tc_fence_after();
      tmem_dealloc(tmem_base, TMEM_COLS);
   }
}

template <int BN, bool TURNED = false>
int launch_any(cudaStream_t s, const AnyOperand &A, const AnyOperand &B, const AnyEpilogue &ep, int K, int S)
{
   using L = AnySmem<BN>;
   auto kern = umma_gemm_any_kernel<BN, TURNED>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), L::kBytes));
   uint32_t *status = device_status_word(s);
   if (!status) return fail(SOFIE_CUDA_ERR_CUDA, "cannot allocate the device status word");
   const int tiles = ceil_div(A.rows, kAnyBM) * ceil_div(B.rows, BN);
   const int grid = S > 1 ? tiles * S : (tiles < kNumSMs ? tiles : kNumSMs);
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = dim3(grid);
   cfg.blockDim = dim3(kAnyThreads);
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
   SOFIE_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, A, B, ep, K, S, status));
   set_last_engine(SOFIE_ENGINE_TCGEN05);
   return SOFIE_CUDA_OK;
}

// Time of a product on this kernel in ns, at its best tile width and cluster size.
long long any_ns(const sofie_gemm_f32_desc &desc, bool turned, int &BN, int &S)
{
   sofie_gemm_f32_desc d = desc;
   if (turned) d.M = desc.N, d.N = desc.M;
   const int tm = ceil_div(d.M, kAnyBM), nkb = ceil_div(d.K, kAnyKE);
   // Tile width and clusters along K by the time they take, in ns (fitted to 450 products, each at every width and cluster size): a stage
   // of 32 K, a tile's start and end, the exchange within a cluster, and what the write-out takes more where rows of Y are not whole
   // 16-byte words and where a bias of Y's shape is read. Nothing overlaps a CTA's write-out. Clusters that the card has no room for wait for a
   // round to end: with 140 CTAs taken for granted at four, where it has 132, 14 x 2144 x 1368 took 22.6 us (13.4 turned) and 19 x 2227 x 740 19.9 (12.1).
   static const int widths[3] = {128, 64, 32}, stage[3] = {1210, 700, 750}, tile[3] = {4100, 2300, 1500}, scalar[3] = {2000, 1000, 470}, scalar_full[3] = {3500, 1600, 950};
   const bool vec = d.N % 4 == 0 && !turned, full = d.bias_kind == 2;
   const long long bias = full ? (long long)d.M * d.N / 750 : 0;
   BN = 32, S = 1;
   long long best = -1;
   for (int w = 0; w < 3; w++) {
      if (widths[w] > 32 && widths[w] / 2 >= d.N) continue; // more than half of the tile would be padding
      const long long tiles = (long long)tm * ceil_div(d.N, widths[w]);
      const int out = vec ? 0 : scalar[w] + (full ? scalar_full[w] : 0);
      for (int i = 0, q = 1; i < 4 && (q == 1 || (nkb >= 2 * q && tiles * q <= 3 * kNumSMs)); i++, q *= 2) {
         const long long waves = (tiles * q + kClusterRoom[i] - 1) / kClusterRoom[i];
         const long long time = 1400 + bias + waves * ((long long)ceil_div(nkb, q) * stage[w] + tile[w] + out / q + (q > 1 ? 2100 : 0));
         if (best < 0 || time < best) best = time, BN = widths[w], S = q;
      }
   }
   return best;
}
// Up to 31 rows fill a quarter of a tile of 128; the rest of it is zeros that are loaded, split and multiplied too. As the columns of a tile they fill it, and the long side makes the rows:
// the same parts and products, written along the tile's rows. 30 x 1109 x 1819 28.3 -> 13.1 us, 18 x 2378 x 2513 32.7 -> 23.1, 9 x 2327 x 1695 24.2 -> 16.7. Taken where the estimate
// says 0.8 of the time: of 148 products timed each way the 44 below it took 0.65 to 1.00, the others 0.91 to 1.47 (but for four). From K = 512 on, since these write word by word
// (31 x 3359 x 472 12.5 -> 13.3 us). From 32 rows on operands split beforehand are the faster ones (64 x 2533 x 3026 31 us, turned 41).
long long any_best_ns(const sofie_gemm_f32_desc &d, bool &turned, int &BN, int &S)
{
   int other_BN, other_S;
   const long long straight = any_ns(d, false, BN, S), other = d.M < 32 && d.K >= 512 ? any_ns(d, true, other_BN, other_S) : straight;
   turned = 10 * other < 8 * straight;
   if (!turned) return straight;
   BN = other_BN, S = other_S;
   return other;
}
// ... and on the CUDA-core kernel.
long long simt_ns(const sofie_gemm_f32_desc &d)
{
   const long long blocks = (long long)ceil_div(d.M, 64) * ceil_div(d.N, 64), steps = ceil_div(d.K, 16);
   const long long alone = 1900 * steps * ((blocks + 3 * kNumSMs - 1) / (3 * kNumSMs));
   const long long filled = ((d.transB ? 645 : 445) * steps + 800 + (d.bias_kind == 2 ? 330 : 0)) * blocks / kNumSMs;
   return 2200 + (alone > filled ? alone : filled);
}

} // namespace
} // namespace umma

long long gemm_f32_whole_ns(const sofie_gemm_f32_desc &d, bool tma)
{
   int BN, S;
   bool turned;
   const long long any = umma::any_best_ns(d, turned, BN, S), simt = umma::simt_ns(d);
   return tma || simt > any ? any : simt;
}

int launch_gemm_f32_any(cudaStream_t s, const sofie_gemm_f32_desc &d, bool tma, const float *A, const float *B, const float *C, float *Y)
{
   using namespace umma;
   auto aligned = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
   const bool vec_k = d.K % 4 == 0;
   const AnyOperand a{A, d.transA ? d.M : d.K, d.M, d.transA ? kRowsContiguous : (vec_k && aligned(A) ? kVecK : kScalarK)};
   const AnyOperand b{B, d.transB ? d.K : d.N, d.N, !d.transB ? kRowsContiguous : (vec_k && aligned(B) ? kVecK : kScalarK)};
   const AnyEpilogue ep{d.alpha, d.beta, C, Y, d.bias_kind, d.relu, d.N % 4 == 0 && aligned(Y) && (d.bias_kind != 2 || aligned(C)), d.K >= 1024 ? 8 : (d.K >= 256 ? 4 : 3)};
   int BN, S;
   bool turned;
   const long long best = any_best_ns(d, turned, BN, S);
   // What TMA cannot fetch has the CUDA-core kernel beside it: blocks of 64 x 64, steps of 16 K that take 1.9 us alone and 0.45 us (0.65 with
   // B stored [N,K]) apart on an SM full of them, whose outputs leave while other blocks compute. It wins where the output is what
   // counts: 16384 x 777 x 64 81 us against 144; 1000 x 777 x 1333 211 against 38. Over
   // 620 products the choice is 0.9 % above the faster of the two in the mean, and never more than 5 % above the CUDA-core kernel. Up to 32 terms the CUDA cores' kernel is another and up to 1.9 times as fast
   // as estimated (16384 x 4093 x 8 with a full bias 106 us, 580 here; 2310 x 3543 x 17 15 and 28): what the estimate leaves on this kernel stays here all the same, where its error is half (0.4 to 0.8) of a chain's.
   if (!tma && forced_engine() != SOFIE_ENGINE_TCGEN05) {
      if (simt_ns(d) < best) return fail(SOFIE_CUDA_ERR_UNSUPPORTED, "faster on the CUDA cores");
   }
   if (turned) return launch_any<32, true>(s, b, a, ep, d.K, S); // (a wider tile would be half padding)
   if (BN == 128) return launch_any<128>(s, a, b, ep, d.K, S);
   if (BN == 64) return launch_any<64>(s, a, b, ep, d.K, S);
   return launch_any<32>(s, a, b, ep, d.K, S);
}

} // namespace sofie
