// fp32 3x3 convolution (stride 1, pad 1, NHWC, 16 or 32 input channels) with its operands split into two HALF-precision parts.
//
// The haloed-patch kernel of umma_conv.cu splits fp32 values into two TF32 parts: eight bytes a value, eight values of K per MMA. What
// bounds it is the shared memory between the roles: the MMAs' reads of the 128-row patch operand, the weights beside it and the
// converters' own traffic, 260 KB (16 -> 32 channels) and 608 KB (32 -> 64) a tile at 128 bytes a clock. Two half-precision parts of
// a value hold the same 22 bits in four bytes, and an MMA takes sixteen of them: 136 and 326 KB a tile.
//
// Half precision has 5 bits of exponent, so the parts are formed of SCALED values: a patch is multiplied by the power of two that brings
// its largest magnitude into [2^14, 2^15), every output channel's weights by one of their own, and the epilogue multiplies the sums by the
// product of the inverse powers (exact). A trailing part is multiplied by another 2^11 before it is rounded, so that it lies where its leading part
// does and not 2^11 below, at the end of half precision's range (the scaled residual of H. Ootomo and R. Yokota, "Recovering single precision accuracy
// from Tensor Cores while surpassing the FP32 theoretical peak performance", 2022); the products with one trailing factor have sums of their own, which
// the epilogue multiplies by 2^-11. A value whose scaled magnitude is 2^-14 or more is then held to 2^-22 of itself, as two TF32 parts hold it; a
// smaller one to 2^-36 after scaling. The converters look for a value as small as that, at EVERY value of the patch and not at the largest of
// a pixel or a channel: its neighbours may meet weights that are zero. A tile that has one, and any with an infinity or a NaN, is computed
// by the epilogue warps as chains of fp32 FMAs from global memory; all tiles are when the weights of an output channel span more than that, or when the
// two scales together leave fp32's range. The largest of a patch may be 2^28 times its smallest, beside zeros, before any of this happens.
// Error against float64 (2-norm), N(0,1) operands: 2.1e-7 at 16 and 3.7e-7 at 32 channels, where TF32 parts gave 7.0e-7 and 1.28e-6 (their trailing
// part is truncated, these are rounded, and the sums take half as many steps); operands of one sign 6.1e-7 and 1.4e-6 (1.05e-6 and 2.4e-6).
// 8192 images 16 -> 32 at 32 x 32 with MaxPool 490 -> 332 us, 32 -> 64 at 16 x 16 367 -> 205 us; unpooled 2048 x 16 -> 32 172 -> 143 us. A tile taken
// as FMA chains costs about sixty of the others (45 us).
//
// A tile is 16 x 8 pixels of one image; one TMA box brings its 18 x 10 patch (zero fill outside the image) as fp32 rows; two groups of four
// converter warps take the patches in turn, find the largest magnitude, split the values and write both parts as K-major swizzled
// rows, from which each of the 9 taps is a start address (see the haloed-patch kernel). One MMA multiplies the leading parts of the
// pixels with [leading | trailing] weights (2 * BN columns), one the trailing parts with the leading weights, into the second BN columns. A TMEM buffer goes back to the issuers as soon as it has been read, before pooling and stores. Pooled tiles are
// read in the shape that puts a pixel and the one below it in one thread: a third of the shuffles, which wait for the shared-memory
// pipe the MMAs keep busy (the epilogue set the kernel's time with them: 375 instead of 326 us).
// Waiting with one lane and a vote, or with test_wait, instead of whole warps on try_wait: 5 to 25 % slower.
#include "umma.cuh"
#include "contract.cuh"
#include <cuda_fp16.h>

namespace sofie {
namespace umma {
namespace {

constexpr int kHalfTileH = 16, kHalfTileW = 8;
constexpr int kHalfPatchH = kHalfTileH + 2, kHalfPatchW = kHalfTileW + 2;
constexpr int kHalfPatchPixels = kHalfPatchH * kHalfPatchW;
constexpr int kHalfEpiWarps = 8, kHalfConvGroups = 2, kHalfConvGroupWarps = 4;
constexpr int kHalfConvWarps = kHalfConvGroups * kHalfConvGroupWarps;
constexpr int kHalfIssuerB = 2 + kHalfEpiWarps + kHalfConvWarps;
constexpr int kHalfThreads = (kHalfIssuerB + 1) * 32;
constexpr int kHalfMaxSlots = 4;
constexpr int kHalfScales = 16;       // ring of tile scales: more than the tiles between a converter and the epilogue (slots + TMEM buffers)
constexpr uint32_t kHalfSpread = 28;  // a value may be 2^-28 of the patch's largest (see above)
constexpr float kHalfTrailing = 2048.f; // trailing parts are held times 2^11

__host__ __device__ constexpr int half_part_bytes(int C) { return (kHalfPatchPixels * 2 * C + 1023) / 1024 * 1024; } // a patch's leading or trailing parts
__host__ __device__ constexpr int half_raw_bytes(int C) { return kHalfPatchPixels * 4 * C; }
__host__ __device__ constexpr int half_weight_bytes(int BN, int C) { return 9 * 2 * BN * 2 * C; }
// patches in flight as fp32, and as many as parts: four or two, so that a slot always meets the same converter group and the same issuer
__host__ __device__ constexpr int half_slots(int BN, int C)
{
   return 220 * 1024 - half_weight_bytes(BN, C) >= 4 * (half_raw_bytes(C) + 2 * half_part_bytes(C)) ? 4 : 2;
}

struct HalfConvParams {
   const float *X, *W, *bias; // NHWC, [Cout][3][3][C], [Cout] or nullptr
   float *Y;                  // NHWC, pooled or not
   int N, H, W_, Cout;
   int tilesH, tilesW, num_tiles;
   int relu;
};

// Offset of a 16-byte piece in rows of RB bytes as the MMA's swizzle expects it (the region starts on a 1024-byte boundary).
template <int RB>
__device__ __forceinline__ uint32_t half_swizzled(uint32_t off)
{
   static_assert(RB == 32 || RB == 64, "rows of 16 or 32 halves");
   return off ^ ((off >> 3) & (RB == 32 ? 0x10u : 0x30u));
}

// Eight fp32 values times a power of two as 16 bytes of leading halves and 16 bytes of 2^11 times what those leave, rounded to nearest even.
__device__ __forceinline__ void half_split(const float (&v)[8], float scale, uint4 &hi, uint4 &lo)
{
   uint32_t h[4], l[4];
   const uint64_t scale2 = pack_f32x2(scale, scale), minus_one2 = pack_f32x2(-1.f, -1.f), trailing2 = pack_f32x2(kHalfTrailing, kHalfTrailing);
#pragma unroll
   for (int i = 0; i < 4; i++) {
      const uint64_t v2 = fma_f32x2(pack_f32x2(v[2 * i], v[2 * i + 1]), scale2, 0);
      float a, b;
      unpack_f32x2(v2, a, b);
      const __half2 p = __floats2half2_rn(a, b);
      const float2 back = __half22float2(p);
      unpack_f32x2(fma_f32x2(fma_f32x2(pack_f32x2(back.x, back.y), minus_one2, v2), trailing2, 0), a, b); // the difference is exact
      const __half2 q = __floats2half2_rn(a, b);
      h[i] = *reinterpret_cast<const uint32_t *>(&p);
      l[i] = *reinterpret_cast<const uint32_t *>(&q);
   }
   hi = make_uint4(h[0], h[1], h[2], h[3]);
   lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// Largest magnitude of eight values, and the smallest of those that are not zero less one, as twice the magnitude's bits (no sign).
__device__ __forceinline__ void half_extremes(const float (&v)[8], uint32_t &largest, uint32_t &smallest)
{
#pragma unroll
   for (int i = 0; i < 8; i++) {
      const uint32_t m = __float_as_uint(v[i]) << 1;
      largest = max(largest, m);
      smallest = __viaddmin_u32(m, 0xffffffffu, smallest);
   }
}

// The scale that brings the largest magnitude into [2^14, 2^15), or 2^126 where that is less, and its inverse; false when the parts would not hold
// the values (see the head of this file). Everything fits under 2^126: subnormal values are multiples of 2^-23 then, which two halves hold exactly.
__device__ __forceinline__ bool half_scale(uint32_t largest, uint32_t smallest, float &scale, float &inverse)
{
   const uint32_t e = largest >> 24, e_small = (smallest + 1) >> 24;
   scale = inverse = 1.f;
   if (largest == 0) return true;
   if (e == 255) return false;
   const uint32_t lift = e > 15 ? e : 15;
   scale = __uint_as_float((268u - lift) << 23);
   inverse = __uint_as_float((lift - 14u) << 23);
   return e <= 15 || (e_small > 0 && e - e_small <= kHalfSpread);
}

// Output pixel (h, w) of image n as chains of fp32 FMAs, without bias: J channels from c on, consecutive ones or (PAIRS) two of every eight.
template <int C, int J, bool PAIRS>
__device__ __forceinline__ void half_conv_exact(const HalfConvParams &p, int n, int h, int w, int c, float (&acc)[J])
{
#pragma unroll
   for (int j = 0; j < J; j++) acc[j] = 0.f;
#pragma unroll 1
   for (int tap = 0; tap < 9; tap++) {
      const int ih = h + tap / 3 - 1, iw = w + tap % 3 - 1;
      const bool in = ih >= 0 && ih < p.H && iw >= 0 && iw < p.W_;
      const float4 *x = reinterpret_cast<const float4 *>(p.X + (((size_t)n * p.H + (in ? ih : 0)) * p.W_ + (in ? iw : 0)) * C);
#pragma unroll 1
      for (int c4 = 0; c4 < C / 4; c4++) {
         float4 xv = x[c4];
         if (!in) xv = make_float4(0.f, 0.f, 0.f, 0.f);
         const float4 *wt = reinterpret_cast<const float4 *>(p.W + (size_t)(c * 9 + tap) * C) + c4;
#pragma unroll
         for (int j = 0; j < J; j++) {
            const int dc = PAIRS ? (j >> 1) * 8 + (j & 1) : j;
            if (c + dc >= p.Cout) break;
            const float4 wv = __ldg(wt + dc * 9 * C / 4);
            acc[j] = fmaf(xv.x, wv.x, acc[j]);
            acc[j] = fmaf(xv.y, wv.y, acc[j]);
            acc[j] = fmaf(xv.z, wv.z, acc[j]);
            acc[j] = fmaf(xv.w, wv.w, acc[j]);
         }
      }
   }
}

template <int BN, int C, bool POOL>
__global__ void __launch_bounds__(kHalfThreads, 1)
umma_conv3x3_half_kernel(const __grid_constant__ CUtensorMap tmX, HalfConvParams p, uint32_t *status)
{
   constexpr int RB = 2 * C;                       // bytes of an operand row: one pixel's or one (tap, output channel)'s halves
   constexpr int KSTEPS = C / 16;                  // MMAs' K steps per tap
   constexpr int PART = half_part_bytes(C), RAW = half_raw_bytes(C);
   constexpr int UPP = C / 8;                      // units of eight channels per pixel
   constexpr int W_ITEM = 2 * BN * RB;             // one tap's weights: BN leading rows, BN trailing rows
   constexpr int NBUF = 512 / (2 * BN) >= 4 ? 4 : 2;
   constexpr int SLOTS = half_slots(BN, C);
   constexpr uint32_t TMEM_COLS = NBUF * 2 * BN;
   constexpr int CW = BN / 2;                      // channels per epilogue warp (two warps a lane quarter)
   constexpr int CH = CW >= 32 ? 32 : CW;
   extern __shared__ unsigned char smem_raw[];
   unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
   unsigned char *w_smem = smem;                   // 9 items
   unsigned char *ops = w_smem + 9 * W_ITEM;       // SLOTS x (leading, trailing)
   unsigned char *raws = ops + (size_t)SLOTS * 2 * PART;
   __shared__ uint64_t raw_full[kHalfMaxSlots], raw_empty[kHalfMaxSlots], op_full[kHalfMaxSlots], op_empty[kHalfMaxSlots];
   __shared__ uint64_t tmem_full[NBUF], tmem_empty[NBUF], w_ready;
   __shared__ uint32_t tmem_base_holder;
   __shared__ volatile uint32_t abort_flag;
   __shared__ int w_spread;                        // a channel's weights have to be taken as fp32
   __shared__ __align__(16) float s_bias[BN], s_winv[BN];
   __shared__ volatile float s_xinv[kHalfScales];  // inverse scale of a tile's patch, 0: take the tile as fp32
   __shared__ uint2 s_red[kHalfConvGroups][2][kHalfConvGroupWarps];

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   SOFIE_PROF_DECL
   griddep_launch_dependents(); // the next kernel may set itself up while this one runs
   for (int c = threadIdx.x; c < BN; c += kHalfThreads) s_bias[c] = (c < p.Cout && p.bias) ? p.bias[c] : 0.f;
   if (threadIdx.x == 0) {
      for (int s = 0; s < kHalfMaxSlots; s++) {
         mbar_init(&raw_full[s], 1);
         mbar_init(&raw_empty[s], kHalfConvGroupWarps);
         mbar_init(&op_full[s], kHalfConvGroupWarps);
         mbar_init(&op_empty[s], 1);
      }
      for (int b = 0; b < NBUF; b++) {
         mbar_init(&tmem_full[b], 1);
         mbar_init(&tmem_empty[b], kHalfEpiWarps);
      }
      mbar_init(&w_ready, kHalfConvWarps);
      abort_flag = 0;
      w_spread = 0;
      fence_mbar_init();
      prefetch_tensormap(&tmX);
   }
   if (warp == 1) {
      tmem_alloc(&tmem_base_holder, TMEM_COLS);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = tmem_base_holder;

   if (warp == 0) {
      // ---------------- TMA producer: one box per tile ----------------
      griddep_wait(); // the activations are the previous kernel's output
      if (lane == 0) {
         TileWalker tw;
         tw.init(blockIdx.x, gridDim.x, p.tilesH, p.tilesW);
         int s = 0, g = 0;
         uint32_t ph = 0;
         for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, g++, ring_next(s, ph, SLOTS), tw.next()) {
            if (!SOFIE_PROF_WAIT(mbar_wait(&raw_empty[s], ph ^ 1, &abort_flag, status, kStatusWaitEmpty, g))) break;
            mbar_expect_tx(&raw_full[s], RAW);
            // rows and columns start at -1: zero fill; the channel coordinate is 0
            tma_load_4d(raws + (size_t)s * RAW, &tmX, 0, tw.tw * kHalfTileW - 1, tw.th * kHalfTileH - 1, tw.n, &raw_full[s]);
         }
      }
   } else if (warp == 1 || warp == kHalfIssuerB) {
      // ---------------- MMA issuers: even and odd tiles ----------------
      if (lane == 0) {
         constexpr uint32_t idesc = make_idesc<kF16>(128, BN), idesc_wide = make_idesc<kF16>(128, 2 * BN);
         bool ok = SOFIE_PROF_WAIT(mbar_wait(&w_ready, 0, &abort_flag, status, kStatusWaitConv, 0x4000));
         const uint64_t db0 = make_smem_desc(smem_u32(w_smem), RB);
         const uint32_t b_hi_word = (uint32_t)(db0 >> 32), b_lo_word = (uint32_t)db0;
         const int step = gridDim.x;
         for (int lt = warp == 1 ? 0 : 1; ok && blockIdx.x + (long long)lt * step < p.num_tiles; lt += 2) {
            const int s = lt % SLOTS, buf = lt % NBUF;
            ok = SOFIE_PROF_WAIT(mbar_wait(&op_full[s], (uint32_t)(lt / SLOTS) & 1u, &abort_flag, status, kStatusWaitConv, lt)) &&
                 SOFIE_PROF_WAIT(mbar_wait(&tmem_empty[buf], ((uint32_t)(lt / NBUF) & 1u) ^ 1u, &abort_flag, status, kStatusWaitAccum, 0x2000 + lt));
            if (!ok) break;
            tc_fence_after();
            const uint32_t d = tmem_base + (uint32_t)(buf * 2 * BN);
            // eight pixels of a tile row are one 8-row group, the next group is one patch row further (make_smem_desc_rows)
            const uint64_t da0 = make_smem_desc_rows(smem_u32(ops + (size_t)s * 2 * PART), RB, kHalfPatchW * RB);
            const uint32_t a_hi_word = (uint32_t)(da0 >> 32), a_lo_word = (uint32_t)da0;
            auto adesc = [&](uint32_t off) { return ((uint64_t)a_hi_word << 32) | (uint64_t)(a_lo_word + (off >> 4)); };
            auto bdesc = [&](uint32_t off) { return ((uint64_t)b_hi_word << 32) | (uint64_t)(b_lo_word + (off >> 4)); };
#pragma unroll
            for (int tap = 0; tap < 9; tap++) {
#pragma unroll
               for (int k = 0; k < KSTEPS; k++) {
                  const uint32_t a = (uint32_t)(((tap / 3) * kHalfPatchW + tap % 3) * RB + k * 32), b = (uint32_t)(tap * W_ITEM + k * 32);
                  tc_mma<kF16>(d, adesc(a), bdesc(b), idesc_wide, (tap | k) ? 1u : 0u); // leading x [leading | trailing]
                  tc_mma<kF16>(d + BN, adesc(a + PART), bdesc(b), idesc, 1u);           // trailing x leading
               }
            }
            tc_commit(&op_empty[s]);
            tc_commit(&tmem_full[buf]);
         }
      }
   } else if (warp >= 2 + kHalfEpiWarps) {
      // ---------------- converters ----------------
      const int cw = warp - 2 - kHalfEpiWarps, group = cw / kHalfConvGroupWarps, gw = cw % kHalfConvGroupWarps;
      {
         // the weights, once per CTA, by all converter warps: TPR neighbouring threads a row
         constexpr int TPR = kHalfConvWarps * 32 / BN, UNITS = 9 * UPP;
         static_assert(TPR >= 1 && 32 % TPR == 0, "the threads of a row are in one warp");
         const int t = cw * 32 + lane, row = t / TPR, sub = t % TPR;
         const float4 *src = reinterpret_cast<const float4 *>(p.W + (size_t)(row < p.Cout ? row : 0) * 9 * C);
         auto load = [&](int u, float (&v)[8]) {
            float4 a = __ldg(src + 2 * u), b = __ldg(src + 2 * u + 1);
            if (row >= p.Cout) a = b = make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
         };
         uint32_t largest = 0, smallest = 0xffffffffu;
#pragma unroll 4
         for (int u = sub; u < UNITS; u += TPR) {
            float v[8];
            load(u, v);
            half_extremes(v, largest, smallest);
         }
#pragma unroll
         for (int o = 1; o < TPR; o <<= 1) {
            largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, o));
            smallest = min(smallest, __shfl_xor_sync(0xffffffffu, smallest, o));
         }
         float scale, inverse;
         if (!half_scale(largest, smallest, scale, inverse)) w_spread = 1;
         if (sub == 0) s_winv[row] = inverse;
#pragma unroll 4
         for (int u = sub; u < UNITS; u += TPR) {
            float v[8];
            load(u, v);
            uint4 hi, lo;
            half_split(v, scale, hi, lo);
            unsigned char *item = w_smem + (u / UPP) * W_ITEM;
            const uint32_t off = half_swizzled<RB>((uint32_t)(row * RB + (u % UPP) * 16));
            *reinterpret_cast<uint4 *>(item + off) = hi;
            *reinterpret_cast<uint4 *>(item + BN * RB + off) = lo;
         }
         fence_proxy_async();
         __syncwarp();
         if (lane == 0) mbar_arrive(&w_ready);
      }
      constexpr int GT = kHalfConvGroupWarps * 32, UNITS = kHalfPatchPixels * UPP, PER = (UNITS + GT - 1) / GT;
      const int t = gw * 32 + lane;
      // a warp whose wait gave up goes on to the group's barrier, where the four leave together: nobody waits there for one that has left
      bool ok = true;
      for (int lt = group; blockIdx.x + (long long)lt * gridDim.x < p.num_tiles; lt += kHalfConvGroups) {
         const int s = lt % SLOTS;
         ok = ok && SOFIE_PROF_WAIT(mbar_wait(&raw_full[s], (uint32_t)(lt / SLOTS) & 1u, &abort_flag, status, kStatusWaitFull, 0x6000 + lt));
         float v[PER][8];
         // 32 bytes a unit: the lanes of a quarter warp read different halves of their units at a time, so that no banks collide
         const float4 *raw = reinterpret_cast<const float4 *>(raws + (size_t)s * RAW);
         const int swap = (lane >> 2) & 1;
#pragma unroll
         for (int i = 0; i < PER; i++) {
            const int u = t + i * GT;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (u < UNITS) {
               a = raw[2 * u + swap];
               b = raw[2 * u + 1 - swap];
            }
            v[i][0] = swap ? b.x : a.x; v[i][1] = swap ? b.y : a.y; v[i][2] = swap ? b.z : a.z; v[i][3] = swap ? b.w : a.w;
            v[i][4] = swap ? a.x : b.x; v[i][5] = swap ? a.y : b.y; v[i][6] = swap ? a.z : b.z; v[i][7] = swap ? a.w : b.w;
         }
         uint32_t largest = 0, smallest = 0xffffffffu;
#pragma unroll
         for (int i = 0; i < PER; i++) half_extremes(v[i], largest, smallest);
         largest = __reduce_max_sync(0xffffffffu, largest);
         smallest = __reduce_min_sync(0xffffffffu, smallest);
         uint2 *red = s_red[group][(lt >> 1) & 1];
         if (lane == 0) {
            mbar_arrive(&raw_empty[s]); // the patch is in registers
            red[gw] = make_uint2(largest, smallest);
         }
         uint32_t all_ok;
         asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                      : "=r"(all_ok)
                      : "r"(ok ? 1u : 0u), "r"(1 + group), "n"(GT)
                      : "memory");
         if (!all_ok) break;
#pragma unroll
         for (int i = 0; i < kHalfConvGroupWarps; i++) {
            const uint2 o = red[i];
            largest = max(largest, o.x);
            smallest = min(smallest, o.y);
         }
         float scale, inverse;
         const bool fits = half_scale(largest, smallest, scale, inverse);
         ok = SOFIE_PROF_WAIT(mbar_wait(&op_empty[s], ((uint32_t)(lt / SLOTS) & 1u) ^ 1u, &abort_flag, status, kStatusWaitEmpty, 0x7000 + lt));
         // read by the epilogue after the tile's MMAs, which wait for this group's arrivals below
         if (t == 0) s_xinv[lt % kHalfScales] = fits ? inverse : 0.f;
         unsigned char *op = ops + (size_t)s * 2 * PART;
#pragma unroll
         for (int i = 0; i < PER; i++) {
            const int u = t + i * GT;
            if (ok && u < UNITS) {
               uint4 hi, lo;
               half_split(v[i], scale, hi, lo);
               const uint32_t off = half_swizzled<RB>((uint32_t)u * 16);
               *reinterpret_cast<uint4 *>(op + off) = hi;
               *reinterpret_cast<uint4 *>(op + PART + off) = lo;
            }
         }
         fence_proxy_async();
         __syncwarp();
         if (ok && lane == 0) mbar_arrive(&op_full[s]);
      }
   } else {
      // ---------------- epilogue: warps 2..9, two per lane quarter ----------------
      const int c_begin = ((warp - 2) >> 2) * CW;
      const int lane_base = (warp & 3) * 32;
      TileWalker tw;
      tw.init(blockIdx.x, gridDim.x, p.tilesH, p.tilesW);
      // the weights' scales and verdict are the converters'
      bool ok = SOFIE_PROF_WAIT(mbar_wait(&w_ready, 0, &abort_flag, status, kStatusWaitConv, 0x5000));
      const bool w_exact = w_spread != 0;
      // largest and smallest inverse scale of a channel's weights (positive: ordered as their bits are)
      uint32_t w_low = 0x7f800000u, w_high = 0;
      for (int c = lane; c < BN; c += 32) {
         w_low = min(w_low, __float_as_uint(s_winv[c]));
         w_high = max(w_high, __float_as_uint(s_winv[c]));
      }
      const float winv_low = __uint_as_float(__reduce_min_sync(0xffffffffu, w_low)), winv_high = __uint_as_float(__reduce_max_sync(0xffffffffu, w_high));
      // pooled: this lane's channels are 2 (lane % 4), +1 of every eight, its window is lane / 8 of pooled row lane_base / 16 + (lane / 4) % 2
      const int c2 = 2 * (lane & 3);
      const bool second = (lane & 4) != 0;
      float2 winv2[CH / 8], bias2[CH / 8];
      auto load_constants = [&](int c0) {
         if (!POOL) return;
#pragma unroll
         for (int k = 0; k < CH / 8; k++) {
            winv2[k] = *reinterpret_cast<const float2 *>(s_winv + c0 + c2 + 8 * k);
            bias2[k] = *reinterpret_cast<const float2 *>(s_bias + c0 + c2 + 8 * k);
         }
      };
      load_constants(c_begin);
      int lt = 0;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, lt++, tw.next()) {
         const int buf = lt % NBUF;
         ok = SOFIE_PROF_WAIT(mbar_wait(&tmem_full[buf], (uint32_t)(lt / NBUF) & 1u, &abort_flag, status, kStatusWaitAccum, 0x3000 + lt));
         if (!ok) break;
         tc_fence_after();
         const float xinv = s_xinv[lt % kHalfScales];
         // a product of the inverse scales may be subnormal (an exact power of two all the same), but neither zero nor infinite
         const bool exact = w_exact || !(xinv * winv_low > 0.f && xinv * winv_high < __uint_as_float(0x7f800000u));
         const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)(buf * 2 * BN);
#pragma unroll 1
         for (int c0 = c_begin; c0 < c_begin + CW; c0 += CH) {
            if (CW != CH) load_constants(c0);
            float r[CH];
            {
               uint32_t a[CH], b[CH];
               if constexpr (POOL) {
                  tmem_ld_16x256<CH>(t_row + (uint32_t)c0, a);
                  tmem_ld_16x256<CH>(t_row + (uint32_t)(BN + c0), b);
               } else {
                  tmem_ld_cols<CH>(t_row + (uint32_t)c0, a);
                  tmem_ld_cols<CH>(t_row + (uint32_t)(BN + c0), b);
               }
               tmem_ld_wait();
#pragma unroll
               for (int j = 0; j < CH; j++) r[j] = fmaf(__uint_as_float(b[j]), 1.f / kHalfTrailing, __uint_as_float(a[j]));
            }
            if (c0 + CH == c_begin + CW) { // all of this warp's columns have been read: the buffer is the issuers' again
               tc_fence_before();
               __syncwarp();
               if (lane == 0) mbar_arrive(&tmem_empty[buf]);
            }
            if (c0 >= p.Cout) continue;
            if (exact) griddep_wait(); // this thread reads the activations itself
            // sum x the two inverse scales (rounded once) + bias, Relu
            auto finish = [&](float sum, float winv, float bias) {
               const float v = fmaf(sum, xinv * winv, bias);
               return p.relu ? relu_ref(v) : v;
            };
            if constexpr (POOL) {
               // 2x2 MaxPool: the pixel below is in the same thread, the one beside it in lane ^ 4, which keeps the windows of the other half
               // of the quarter; the scales are positive, so the largest sum is the largest result
               const int oh = tw.th * (kHalfTileH / 2) + lane_base / 16 + (second ? 1 : 0), ow = tw.tw * (kHalfTileW / 2) + (lane >> 3);
               float v[CH / 4];
               if (!exact) {
#pragma unroll
                  for (int j = 0; j < CH / 4; j++) {
                     const int k = (j >> 1) * 4 + (j & 1);
                     const float m0 = r[k + 2] > r[k] ? r[k + 2] : r[k], m1 = r[CH / 2 + k + 2] > r[CH / 2 + k] ? r[CH / 2 + k + 2] : r[CH / 2 + k];
                     const float mine = second ? m1 : m0, got = __shfl_xor_sync(0xffffffffu, second ? m0 : m1, 4);
                     v[j] = finish(got > mine ? got : mine, (j & 1) ? winv2[j >> 1].y : winv2[j >> 1].x, (j & 1) ? bias2[j >> 1].y : bias2[j >> 1].x);
                  }
               } else {
#pragma unroll 1
                  for (int pos = 0; pos < 4; pos++) {
                     float acc[CH / 4];
                     half_conv_exact<C, CH / 4, true>(p, tw.n, 2 * oh + (pos >> 1), 2 * ow + (pos & 1), c0 + c2, acc);
#pragma unroll
                     for (int j = 0; j < CH / 4; j++) {
                        const float sum = acc[j] + ((j & 1) ? bias2[j >> 1].y : bias2[j >> 1].x), x = p.relu ? relu_ref(sum) : sum;
                        v[j] = pos == 0 || x > v[j] || v[j] != v[j] ? x : v[j];
                     }
                  }
               }
               float *y = p.Y + (((size_t)tw.n * (p.H / 2) + oh) * (p.W_ / 2) + ow) * p.Cout + c0 + c2;
               const bool pairs = ((p.Cout & 1) | (int)(reinterpret_cast<uintptr_t>(p.Y) & 7)) == 0;
#pragma unroll
               for (int k = 0; k < CH / 8; k++) {
                  const int c = c0 + c2 + 8 * k;
                  if (pairs) {
                     if (c < p.Cout) *reinterpret_cast<float2 *>(y + 8 * k) = make_float2(v[2 * k], v[2 * k + 1]);
                  } else {
                     if (c < p.Cout) y[8 * k] = v[2 * k];
                     if (c + 1 < p.Cout) y[8 * k + 1] = v[2 * k + 1];
                  }
               }
            } else {
               const int pix = lane_base + lane, h = tw.th * kHalfTileH + pix / kHalfTileW, w = tw.tw * kHalfTileW + pix % kHalfTileW;
               if (!exact) {
#pragma unroll
                  for (int j = 0; j < CH; j += 4) {
                     const float4 wi = *reinterpret_cast<const float4 *>(s_winv + c0 + j), bi = *reinterpret_cast<const float4 *>(s_bias + c0 + j);
                     r[j] = finish(r[j], wi.x, bi.x);
                     r[j + 1] = finish(r[j + 1], wi.y, bi.y);
                     r[j + 2] = finish(r[j + 2], wi.z, bi.z);
                     r[j + 3] = finish(r[j + 3], wi.w, bi.w);
                  }
               } else {
#pragma unroll
                  for (int j0 = 0; j0 < CH; j0 += 16) {
                     float acc[16];
                     half_conv_exact<C, 16, false>(p, tw.n, h, w, c0 + j0, acc);
#pragma unroll
                     for (int j = 0; j < 16; j++) {
                        const float sum = acc[j] + s_bias[c0 + j0 + j];
                        r[j0 + j] = p.relu ? relu_ref(sum) : sum;
                     }
                  }
               }
               float *y = p.Y + (((size_t)tw.n * p.H + h) * p.W_ + w) * p.Cout + c0;
               if (c0 + CH <= p.Cout && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
#pragma unroll
                  for (int j = 0; j < CH; j += 4) *reinterpret_cast<float4 *>(y + j) = make_float4(r[j], r[j + 1], r[j + 2], r[j + 3]);
               } else {
#pragma unroll
                  for (int j = 0; j < CH; j++)
                     if (c0 + j < p.Cout) y[j] = r[j];
               }
            }
         }
      }
   }
   SOFIE_PROF_REPORT(warp == 0 ? "producer" : (warp == 1 || warp == kHalfIssuerB ? "mma" : (warp < 2 + kHalfEpiWarps ? "epilogue" : "converter")));
   tc_fence_before();
   __syncthreads();
   if (warp == 1) {
      __syncwarp();
      tc_fence_after();
      tmem_dealloc(tmem_base, TMEM_COLS);
   }
}

template <int BN, int C, bool POOL>
int launch_half(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias, float *Y)
{
   constexpr int smem = half_weight_bytes(BN, C) + half_slots(BN, C) * (half_raw_bytes(C) + 2 * half_part_bytes(C)) + 1024;
   static_assert(smem <= 221 * 1024, "two patches beside the resident weights");
   HalfConvParams p = {};
   p.X = X; p.W = W; p.bias = bias; p.Y = Y;
   p.N = g.N; p.H = g.H; p.W_ = g.W; p.Cout = g.Cout;
   p.tilesH = g.H / kHalfTileH;
   p.tilesW = g.W / kHalfTileW;
   p.num_tiles = g.N * p.tilesH * p.tilesW;
   p.relu = g.relu;
   CUtensorMap tmX;
   uint64_t dims[4] = {(uint64_t)C, (uint64_t)g.W, (uint64_t)g.H, (uint64_t)g.N};
   uint64_t strides[3] = {(uint64_t)C * 4, (uint64_t)g.W * C * 4, (uint64_t)g.H * g.W * C * 4};
   uint32_t box[4] = {(uint32_t)C, (uint32_t)kHalfPatchW, (uint32_t)kHalfPatchH, 1u};
   int rc = make_tensor_map(&tmX, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, X, dims, strides, box, 0);
   if (rc) return rc;
   uint32_t *status = device_status_word(s);
   if (!status) return fail(SOFIE_CUDA_ERR_CUDA, "cannot allocate the device status word");
   const int grid = p.num_tiles < kNumSMs ? p.num_tiles : kNumSMs;
   auto kern = umma_conv3x3_half_kernel<BN, C, POOL>;
   SOFIE_CUDA_TRY(allow_smem(reinterpret_cast<const void *>(kern), smem));
   SOFIE_CUDA_TRY(launch_dependent(kern, dim3(grid), dim3(kHalfThreads), smem, s, tmX, p, status));
   SOFIE_LAUNCH_CHECK("umma_conv3x3_half_kernel");
   set_last_engine(SOFIE_ENGINE_TCGEN05);
   return SOFIE_CUDA_OK;
}

} // namespace
} // namespace umma

// 3x3 / stride 1 / pad 1 NHWC shapes with packed weights and aligned tensors only (the caller has checked those); -1: not this kernel's.
int launch_conv2d_f32_half(cudaStream_t s, const ConvGeom &g, const float *X, const float *W, const float *bias, float *Y)
{
   if (g.H % umma::kHalfTileH != 0 || g.W % umma::kHalfTileW != 0 || (g.pool != 0 && g.pool != 2) || g.N < 1) return -1;
   // rows of 16 or 32 halves; with 64 channels, or 32 to more than 64, the resident weights leave no room for two patches
#define SOFIE_HALF(BN, C) return g.pool ? umma::launch_half<BN, C, true>(s, g, X, W, bias, Y) : umma::launch_half<BN, C, false>(s, g, X, W, bias, Y)
   if (g.C == 16) {
      if (g.Cout <= 32) SOFIE_HALF(32, 16);
      if (g.Cout <= 64) SOFIE_HALF(64, 16);
      SOFIE_HALF(128, 16);
   }
   if (g.C == 32) {
      if (g.Cout <= 32) SOFIE_HALF(32, 32);
      if (g.Cout <= 64) SOFIE_HALF(64, 32);
   }
#undef SOFIE_HALF
   return -1;
}

} // namespace sofie
