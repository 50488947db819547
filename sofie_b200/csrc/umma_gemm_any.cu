// fp32 tensor-core GEMM for the operands TMA cannot fetch -- a transposed A, B stored [K,N], rows that are not multiples of 16
// bytes, unaligned bases -- and for few tiles with a long K. The same arithmetic as the TMA kernel of umma_gemm.cu (3xTF32: every
// value split into hi = tf32(x) and lo = x - hi, lo*hi + hi*lo + hi*hi into a TMEM accumulator, promoted to fp32 registers every 256
// elements of K), with two differences:
//   * sixteen worker warps read the operands themselves, split them in registers and write the hi / lo tiles where the MMA's
//     swizzled K-major descriptors expect them. A unit of work is four consecutive K of one row: one 16-byte load, four scalar loads
//     (rows that are not 16-byte multiples), or four loads of consecutive rows (K is not the contiguous dimension), always one
//     conflict-free 16-byte store per tile. Groups of them take the stages in turn: while one splits and stores, the others' loads
//     are in flight (one group with two stages of loads in flight was bound by their latency: 2500 clocks a stage). The same warps
//     add the partial sums up in registers and write the tile.
//   * B's hi and lo tiles lie side by side as one operand of twice the width: A_hi x [B_hi | B_lo] and A_lo x B_hi are two MMAs per
//     K step instead of three, with a sixth less shared memory read.
//   * a cluster of S CTAs shares one output tile: each takes a S-th of K, leaves its partial tile in shared memory, and adds up and
//     writes a S-th of the rows out of all of them (distributed shared memory, fixed order). No scratch buffer, one launch.
// Measured on B200 (in a graph, back to back): 1000 x 777 x 1333 with A transposed 211 us on the CUDA cores, 35 here; 200 x 200 x 4000
// 85 us on one CTA per 128 x 64 tile, 15 here; 4096 x 4096 x 2048 603 us by the TMA kernel (128 x 64 tiles), 440 here (157 TFLOP/s of
// the 273 that bf16 / 6 leaves): what bounds it is the workers' chain of loading, splitting and storing (1860 clocks a stage, of which
// the MMAs take 770 and their issue 700).
// The tile goes out through shared memory, so stores (and a bias of the output's shape) are contiguous along rows for every N.
#include "umma.cuh"
#include "contract.cuh"

namespace sofie {
namespace umma {
namespace {

constexpr int kAnyBM = 128;             // rows of the tile = TMEM lanes
constexpr int kAnyKE = 32;              // floats of K per stage = one 128-byte swizzle row
constexpr int kAnyWorkers = 16 * 32;
// Groups of worker warps that take the stages in turn. Four were 5 to 10 % faster at 32 columns with a long K and as much slower with a
// short one (the pipeline takes longer to start), and spilled at 64 columns.
constexpr int kAnyGroups = 2;
constexpr int kAnyThreads = kAnyWorkers + 32; // and the warp that issues the MMAs
constexpr int kAnyPromote = 8;          // stages accumulated in one TMEM buffer: 256 elements of K
constexpr int kAnyMaxStages = 5;

template <int BN>
struct AnySmem {
   static constexpr int kA = kAnyBM * 128, kB = BN * 128;
   static constexpr int kStage = 2 * (kA + kB);                       // hi and lo
   static constexpr int kPitch = BN + 4;                              // floats per row of the outgoing tile, which takes the
   static constexpr int kTile = kAnyBM * kPitch * 4;                  // place of the stages when their MMAs are done
   static constexpr int kStages = BN == 128 ? 3 : (BN == 64 ? 4 : 5);
   static_assert(kTile <= kStages * kStage, "the tile fits in the stages");
   static constexpr int kBytes = kStages * kStage + 1024;
};

// How an operand of `rows` x K is read.
enum AnyMode { kVecK = 0, kScalarK = 1, kRowsContiguous = 2 };
struct AnyOperand {
   const float *p;
   long long ld; // distance of rows (kVecK, kScalarK) or of consecutive K (kRowsContiguous)
   int rows, mode;
};

__device__ __forceinline__ void any_split(float x, float &h, float &l)
{
   uint32_t w;
   asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(w) : "f"(x));
   h = __uint_as_float(w);
   l = x - h;
}

// One thread's share of the tiles of an operand with R rows: U units, a unit being K chunk `c` (four floats) of row `r`.
//   K contiguous: eight lanes cover the 128 bytes of one row; the thread's units are T / 8 rows apart, in the same chunk.
//   Rows contiguous: lanes cover consecutive rows; the thread's units are in one row, T / R chunks apart (T threads per group).
// Either way the 16-byte stores of eight lanes fall into eight different bank groups, and everything that depends on the thread is
// worked out once per tile: the loops below are a load, an addition and the split per unit (with the addresses taken from the unit
// number the loaders were bound by instruction issue).
template <int R, int T>
struct AnyLoader {
   static constexpr int U = R * 8 / T;
   static constexpr int kRowStep = T / 8, kChunkStep = T / R; // between the units of a thread
   const float *p = nullptr; // the thread's first element at K = 0 of the tile
   uint32_t at = 0;          // byte offset of its first unit in the tile
   uint32_t ok = 0;          // bit i: the row of unit i exists
   float4 v[U];

   __device__ __forceinline__ void place(const AnyOperand &o, int t)
   {
      const int r = o.mode == kRowsContiguous ? (t & (R - 1)) : (t >> 3), c = o.mode == kRowsContiguous ? t / R : (t & 7);
      at = (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); // the 128-byte swizzle the descriptors name
   }
   __device__ __forceinline__ void tile(const AnyOperand &o, int row0, int t)
   {
      if (o.mode == kRowsContiguous) {
         const int r = row0 + (t & (R - 1));
         ok = r < o.rows ? ~0u : 0u;
         p = o.p + r + (long long)(4 * (t / R)) * o.ld;
      } else {
         const int r = row0 + (t >> 3);
         ok = 0;
#pragma unroll
         for (int i = 0; i < U; i++) ok |= (r + kRowStep * i < o.rows ? 1u : 0u) << i;
         p = o.p + (long long)r * o.ld + 4 * (t & 7);
      }
   }
   // the units of the stage that starts at element k0 of K; K ends at kend
   __device__ __forceinline__ void load(const AnyOperand &o, int k0, int kend, int t)
   {
      if (o.mode == kRowsContiguous) {
         const float *q = p + (long long)k0 * o.ld;
         const long long step = (long long)(4 * kChunkStep) * o.ld;
         int left = kend - k0 - 4 * (t / R); // elements of K from the thread's first chunk on
#pragma unroll
         for (int i = 0; i < U; i++, q += step, left -= 4 * kChunkStep) {
            const float *q1 = q + o.ld, *q2 = q1 + o.ld, *q3 = q2 + o.ld;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ok && left > 0) v[i].x = *q;
            if (ok && left > 1) v[i].y = *q1;
            if (ok && left > 2) v[i].z = *q2;
            if (ok && left > 3) v[i].w = *q3;
         }
      } else {
         const float *q = p + k0;
         const long long step = kRowStep * o.ld;
         const int left = kend - k0 - 4 * (t & 7);
         if (o.mode == kVecK) { // K % 4 == 0 and kend % 4 == 0
#pragma unroll
            for (int i = 0; i < U; i++, q += step) {
               v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
               if (((ok >> i) & 1) && left > 0) v[i] = *reinterpret_cast<const float4 *>(q);
            }
         } else {
#pragma unroll
            for (int i = 0; i < U; i++, q += step) {
               const bool row = (ok >> i) & 1;
               v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
               if (row && left > 0) v[i].x = q[0];
               if (row && left > 1) v[i].y = q[1];
               if (row && left > 2) v[i].z = q[2];
               if (row && left > 3) v[i].w = q[3];
            }
         }
      }
   }
   __device__ __forceinline__ void store(const AnyOperand &o, unsigned char *hi, unsigned char *lo)
   {
#pragma unroll
      for (int i = 0; i < U; i++) {
         // units a multiple of 8 rows apart keep their place in the swizzle pattern; chunks kChunkStep apart flip its upper bits
         const uint32_t off = o.mode == kRowsContiguous ? (at ^ (uint32_t)(i * kChunkStep * 16)) : (at + (uint32_t)(i * kRowStep * 128));
         float4 h, l;
         any_split(v[i].x, h.x, l.x);
         any_split(v[i].y, h.y, l.y);
         any_split(v[i].z, h.z, l.z);
         any_split(v[i].w, h.w, l.w);
         *reinterpret_cast<float4 *>(hi + off) = h;
         *reinterpret_cast<float4 *>(lo + off) = l;
      }
   }
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
   float4 v;
   asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
   return v;
}
__device__ __forceinline__ float ld_cluster_f1(uint32_t addr)
{
   float v;
   asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
   return v;
}
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kAnyWorkers) : "memory"); }

struct AnyEpilogue {
   float alpha, beta;
   const float *C;
   float *Y;
   int bias_kind, relu, vec; // vec: rows of Y (and of a full C) start on 16-byte boundaries
};

__device__ __forceinline__ float any_finish(const AnyEpilogue &ep, float v, float c)
{
   v = ep.alpha * v;
   if (ep.bias_kind) v += ep.beta * c;
   return ep.relu ? relu_ref(v) : v;
}

// Rows [r0, r0 + rows) of the tile at (m0, n0), the sum of the S partial tiles, to global memory.
template <int BN>
__device__ __forceinline__ void any_write(const AnyEpilogue &ep, const float *tile, int S, int r0, int rows, int m0, int n0, int M, int N)
{
   constexpr int P = AnySmem<BN>::kPitch;
   const uint32_t base = smem_u32(tile);
   if (ep.vec) {
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
#pragma unroll 4
      for (int i = threadIdx.x; i < rows * BN; i += kAnyWorkers) {
         const int r = r0 + i / BN, c = i % BN, row = m0 + r, col = n0 + c;
         if (row >= M || col >= N) continue;
         const float b = ep.bias_kind == 1 ? ep.C[col] : (ep.bias_kind == 2 ? ep.C[(size_t)row * N + col] : 0.f);
         float v = 0.f;
         if (S == 1) v = tile[r * P + c];
         else
            for (int q = 0; q < S; q++) v += ld_cluster_f1(mapa_shared(base + (uint32_t)(r * P + c) * 4, (uint32_t)q));
         ep.Y[(size_t)row * N + col] = any_finish(ep, v, b);
      }
   }
}

// Grid: S x min(tiles, SMs / S) CTAs in clusters of S; with S = 1 a CTA walks tiles (N fastest), with S > 1 it has one.
template <int BN>
__global__ void __launch_bounds__(kAnyThreads, 1)
umma_gemm_any_kernel(AnyOperand A, AnyOperand B, AnyEpilogue ep, int K, int S, uint32_t *status)
{
   using L = AnySmem<BN>;
   constexpr int G = kAnyGroups, GT = kAnyWorkers / G; // groups and their threads
   constexpr int QUARTER = BN / 4;       // columns of the tile a worker warp adds up
   constexpr uint32_t TMEM_COLS = 4 * BN; // two buffers of [hi x hi | the cross terms]
   extern __shared__ unsigned char smem_raw[];
   unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
   float *tile_out = reinterpret_cast<float *>(smem);
   __shared__ uint64_t full_bar[kAnyMaxStages], empty_bar[kAnyMaxStages], tmem_full[2], tmem_empty[2];
   __shared__ uint32_t tmem_base_holder;
   __shared__ volatile uint32_t abort_flag;

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   SOFIE_PROF_DECL
   griddep_launch_dependents();
   const int rank = S > 1 ? (int)cluster_ctarank() : 0;
   const int M = A.rows, N = B.rows;
   const int tiles_n = (N + BN - 1) / BN, num_tiles = ((M + kAnyBM - 1) / kAnyBM) * tiles_n;
   const int nkb = (K + kAnyKE - 1) / kAnyKE;
   const int kb0 = (int)((long long)nkb * rank / S), kbn = (int)((long long)nkb * (rank + 1) / S) - kb0; // this rank's stages of a tile
   const int kend = min(K, (kb0 + kbn) * kAnyKE);
   const int units = (kbn + kAnyPromote - 1) / kAnyPromote;
   const int tile0 = blockIdx.x / S, tile_step = gridDim.x / S;
   auto a_hi = [&](int s) { return smem + s * L::kStage; };
   auto a_lo = [&](int s) { return smem + s * L::kStage + L::kA; };
   auto b_hi = [&](int s) { return smem + s * L::kStage + 2 * L::kA; };
   auto b_lo = [&](int s) { return smem + s * L::kStage + 2 * L::kA + L::kB; };

   if (threadIdx.x == 0) {
      for (int s = 0; s < L::kStages; s++) {
         mbar_init(&full_bar[s], GT / 32);
         mbar_init(&empty_bar[s], 1);
      }
      for (int b = 0; b < 2; b++) {
         mbar_init(&tmem_full[b], 1);
         mbar_init(&tmem_empty[b], kAnyWorkers / 32);
      }
      abort_flag = 0;
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
            if (g - first >= (unit + 1) * kAnyPromote + L::kStages) {
               promote();
               unit++;
            }
            if (SOFIE_PROF_WAIT(mbar_wait(&empty_bar[s], ph ^ 1, &abort_flag, status, kStatusWaitEmpty, g))) {
               la.store(A, a_hi(s), a_lo(s));
               lb.store(B, b_hi(s), b_lo(s));
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
         workers_sync();
         if (S > 1) break; // one tile per cluster: it is summed up below
         if (!abort_flag) any_write<BN>(ep, tile_out, 1, 0, kAnyBM, m0, n0, M, N);
         workers_sync(); // the tile has been read: its place is the stages' again
      }
   } else if (lane == 0) {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc_wide = make_idesc<kTF32>(kAnyBM, 2 * BN), idesc = make_idesc<kTF32>(kAnyBM, BN);
      int s = 0, u = 0, g = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
         for (int kc = 0; kc < kbn && ok; kc += kAnyPromote, u++) {
            const int buf = u & 1;
            if (!SOFIE_PROF_WAIT(mbar_wait(&tmem_empty[buf], ((u >> 1) & 1) ^ 1, &abort_flag, status, kStatusWaitAccum, 0x1000 + u))) {
               ok = false;
               break;
            }
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 2 * BN);
            const int kce = min(kbn, kc + kAnyPromote);
            for (int kb = kc; kb < kce; kb++, g++, ring_next(s, ph, L::kStages)) {
               ok = SOFIE_PROF_WAIT(mbar_wait(&full_bar[s], ph, &abort_flag, status, kStatusWaitConv, g));
               if (!ok) break;
               tc_fence_after();
               const uint64_t da = make_smem_desc(smem_u32(a_hi(s)), 128), dal = make_smem_desc(smem_u32(a_lo(s)), 128);
               const uint64_t db = make_smem_desc(smem_u32(b_hi(s)), 128);
#pragma unroll
               for (int k = 0; k < 4; k++) {
                  const uint64_t koff = (uint64_t)(2 * k);
                  tc_mma<kTF32>(d_tmem, da + koff, db + koff, idesc_wide, (kb == kc && k == 0) ? 0u : 1u);
                  tc_mma<kTF32>(d_tmem + BN, dal + koff, db + koff, idesc, 1);
               }
               tc_commit(&empty_bar[s]);
            }
            if (ok) tc_commit(&tmem_full[buf]);
         }
      }
   }
   SOFIE_PROF_REPORT(warp < kAnyWorkers / 32 ? "worker" : "mma");
   if (S > 1) {
      // every rank's partial tile is complete; each sums up and writes its share of the rows
      __syncwarp();
      cluster_sync_all();
      if (warp < kAnyWorkers / 32 && !abort_flag)
         any_write<BN>(ep, tile_out, S, rank * (kAnyBM / S), kAnyBM / S, (tile0 / tiles_n) * kAnyBM, (tile0 % tiles_n) * BN, M, N);
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

template <int BN>
int launch_any(cudaStream_t s, const AnyOperand &A, const AnyOperand &B, const AnyEpilogue &ep, int K, int S)
{
   using L = AnySmem<BN>;
   auto kern = umma_gemm_any_kernel<BN>;
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

} // namespace
} // namespace umma

int launch_gemm_f32_any(cudaStream_t s, const sofie_gemm_f32_desc &d, const float *A, const float *B, const float *C, float *Y)
{
   using namespace umma;
   auto aligned = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
   const bool vec_k = d.K % 4 == 0;
   const AnyOperand a{A, d.transA ? d.M : d.K, d.M, d.transA ? kRowsContiguous : (vec_k && aligned(A) ? kVecK : kScalarK)};
   const AnyOperand b{B, d.transB ? d.K : d.N, d.N, !d.transB ? kRowsContiguous : (vec_k && aligned(B) ? kVecK : kScalarK)};
   const AnyEpilogue ep{d.alpha, d.beta, C, Y, d.bias_kind, d.relu, d.N % 4 == 0 && aligned(Y) && (d.bias_kind != 2 || aligned(C))};
   const int tm = ceil_div(d.M, kAnyBM), nkb = ceil_div(d.K, kAnyKE);
   // Tile width and clusters along K by the time they take: a stage of 32 K costs about 1800 / 1150 / 900 clocks at 128 / 64 / 32
   // columns, a tile's start and end about 6000, the exchange within a cluster 2500 more; clusters of 2 / 4 / 8 found room for
   // 148 / 140 / 104 CTAs at a time.
   static const int widths[3] = {128, 64, 32}, cost[3] = {1800, 1150, 900}, room[4] = {kNumSMs, kNumSMs, 140, 104};
   int BN = 32, S = 1;
   long long best = -1;
   for (int w = 0; w < 3; w++) {
      if (widths[w] > 32 && widths[w] / 2 >= d.N) continue; // more than half of the tile would be padding
      const long long tiles = (long long)tm * ceil_div(d.N, widths[w]);
      for (int i = 0, q = 1; i < 4 && (q == 1 || (nkb >= 2 * q && tiles * q <= 3 * kNumSMs)); i++, q *= 2) {
         const long long waves = (tiles * q + room[i] - 1) / room[i];
         const long long time = waves * ((long long)ceil_div(nkb, q) * cost[w] + 6000 + (q > 1 ? 2500 : 0));
         if (best < 0 || time < best) best = time, BN = widths[w], S = q;
      }
   }
   if (BN == 128) return launch_any<128>(s, a, b, ep, d.K, S);
   if (BN == 64) return launch_any<64>(s, a, b, ep, d.K, S);
   return launch_any<32>(s, a, b, ep, d.K, S);
}

} // namespace sofie
