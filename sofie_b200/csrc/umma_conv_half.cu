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
// smaller one to 2^-36 after scaling. What keeps that from showing in a result, whatever the values are:
// - Channels in different units, undone by the weights: when an input channel's largest weight is zero or more than 2^6 below another's, that
//   channel is multiplied by a power of two that makes its weights as large as the others' and its values as much smaller (zero where no weight reads it).
// - The converters look for values that the parts do not hold, at EVERY value of the patch and every weight of an output channel, and not at the
//   largest of a pixel or a channel: its neighbours may meet weights that are zero. What such values have lost is below 2^-11 in units of the scaled
//   sums, so that a sum of 2^11 or more has it beyond its 22nd bit and stands. A tile with a smaller one is noted, and computed again after all
//   others (half_careful_tiles): in two passes or more, the values that fit one scale and then what they leave with a scale of its own, added up; and, where
//   it is weights that have lost something, as chains of fp32 FMAs for the sums that do not stand and whose windows are not all zero.
// - Infinities and NaNs of a patch are taken as zeros; a result whose window holds a NaN is one, one whose window holds an infinity
//   is computed as a chain, as are all results of weights that hold either.
// - Two scales whose product leaves fp32's range are applied one after the other.
// Error against float64 (2-norm), N(0,1) operands: 2.1e-7 at 16 and 3.7e-7 at 32 channels, where TF32 parts gave 7.0e-7 and 1.28e-6 (their trailing
// part is truncated, these are rounded, and the sums take half as many steps); operands of one sign 6.1e-7 and 1.4e-6 (1.05e-6 and 2.4e-6).
// 8192 images 16 -> 32 at 32 x 32 with MaxPool 490 -> 322 us, 32 -> 64 at 16 x 16 365 -> 189 us; unpooled 2048 x 16 -> 32 165 -> 120 us; one image
// 4.1 -> 4.0 and 5.5 -> 4.8 us when the kernel has just run, about 1 us more behind others (its instructions come from L2 then). Of the first:
// channels 2^8 ... 2^40 apart 340; values down to 2^-28 of the largest and below in every patch 436; weights of a channel decayed to 1e-12 460; two
// passes for every tile 1.6 ms, for images of exp(-r^2 / 8) 1.9, one infinity in each image 3.4 (as chains of FMAs in the epilogue, one scale and no check
// of single sums, the last four took 20 ms, 10 for the infinities). With two converter groups and all epilogue warps on every tile, in 96 registers and 115 KB,
// these were 332, 360, 403, 427 us, 1.5, 2.0 and 2.6 ms: the check of single sums holds a tile longer now, and the chains have 80 registers and a
// smaller L1 cache (parts packed closer, 159 KB: 3.07 ms, but 324 us; the check out of the epilogue's own sums: 413 us, but 335).
//
// A tile is 16 x 8 pixels of one image; one TMA box brings its 18 x 10 patch (zero fill outside the image) as fp32 rows; two or three groups of
// four converter warps take the patches in turn, find the largest magnitude, split the values and write both parts as K-major swizzled
// rows, from which each of the 9 taps is a start address (see the haloed-patch kernel). One MMA multiplies the leading parts of the
// pixels with [leading | trailing] weights (2 * BN columns), one the trailing parts with the leading weights, into the second BN columns.
// A TMEM buffer goes back to the issuers as soon as it has been read, before pooling and stores. Pooled tiles are read in the shape that puts
// a pixel and the one below it in one thread: a third of the shuffles, which wait for the shared-memory pipe the MMAs keep busy (the epilogue
// set the kernel's time with them: 375 instead of 326 us).
// Waiting with one lane and a vote, or with test_wait, instead of whole warps on try_wait: 5 to 25 % slower. Sixteen epilogue warps on four tiles
// at 32 columns, or four converter groups: 339 and 342 us; the roles then wait for the shared memory, of which a tile moves 134 KB, 1050 of its
// 1370 clocks.
#include "umma.cuh"
#include "contract.cuh"
#include <cuda_fp16.h>

namespace sofie {
namespace umma {
namespace {

constexpr int kHalfTileH = 16, kHalfTileW = 8;
constexpr int kHalfPatchH = kHalfTileH + 2, kHalfPatchW = kHalfTileW + 2;
constexpr int kHalfPatchPixels = kHalfPatchH * kHalfPatchW;
constexpr int kHalfEpiWarps = 8, kHalfConvGroupWarps = 4;
constexpr int kHalfCarefulGroups = 2; // groups that convert the careful tiles
constexpr int kHalfMaxSlots = 6;
constexpr int kHalfWeightWarps = 8;   // converter warps that prepare the weights
constexpr int kHalfScales = 16;       // ring of tile scales: more than the tiles between a converter and the epilogue (slots + TMEM buffers)
constexpr uint32_t kHalfSpread = 28;  // a value may be 2^-28 of the patch's largest (see above)
constexpr float kHalfTrailing = 2048.f; // trailing parts are held times 2^11
constexpr float kHalfStands = 2048.f;   // a scaled sum as large as this hides what the parts of its factors have lost: 2 x 288 x 2^15 x 2^-36 < 2^-22 of it
constexpr uint32_t kHalfChannelSpread = 6;     // input channels whose largest weights span more than this many powers of two get factors
constexpr uint32_t kHalfChannelFactor = 60;    // and no factor is smaller than 2^-60
constexpr int kHalfBitWords = 24;     // a bit for each unit of eight channels of a patch (at most 720), and one word more
constexpr int kHalfNoteWords = 256;   // notes of careful tiles: a bit for each of a CTA's tiles, or for 2, 4, ... of them when there are more
// what the converters found in a patch (x) or in an output channel's weights (w)
constexpr uint32_t kHalfWide = 1;     // values that the parts do not hold to 22 bits (x: they are left to another pass)
constexpr uint32_t kHalfSpecial = 2;  // infinities or NaNs
constexpr uint32_t kHalfChains = 4;   // x: take all of it as chains
// state of a converter warp: which of two sets of words its group exchanges next, whether all of its waits have ended well, whether its group has left
constexpr uint32_t kHalfTurn = 1, kHalfOk = 2, kHalfLeft = 4;

__host__ __device__ constexpr int half_buffers(int BN) { return 512 / (2 * BN) >= 4 ? 4 : 2; } // accumulators in tensor memory
__host__ __device__ constexpr int half_part_bytes(int C) { return (kHalfPatchPixels * 2 * C + 1023) / 1024 * 1024; } // a patch's leading or trailing parts
__host__ __device__ constexpr int half_raw_bytes(int C) { return kHalfPatchPixels * 4 * C; }
__host__ __device__ constexpr int half_weight_bytes(int BN, int C) { return 9 * 2 * BN * 2 * C; }
// Converter groups, which take the patches in turn: a patch's way through one (load, largest magnitude, barrier, split, store) is latency.
// Patches in flight as fp32, and as many as parts: a multiple of the groups and of the two issuers, so that a slot always meets the same ones.
__host__ __device__ constexpr int half_room(int BN, int C) { return (220 * 1024 - half_weight_bytes(BN, C)) / (half_raw_bytes(C) + 2 * half_part_bytes(C)); }
// (A third group where six patches fit gains at 32 columns only: with 64 it made the pooled layer 60.6 -> 64.4 us, 1024 images of 16 channels.)
__host__ __device__ constexpr int half_groups(int BN, int C) { return BN == 32 && half_room(BN, C) >= 6 ? 3 : 2; }
__host__ __device__ constexpr int half_slots(int BN, int C) { return half_room(BN, C) >= 6 ? 6 : (half_room(BN, C) >= 4 ? 4 : 2); }
// slots of one group of careful tiles: the rings of passes and patches below are sized for two
__host__ __device__ constexpr int half_careful_slots(int BN, int C) { return half_slots(BN, C) >= 4 ? 2 : 1; }
// Epilogue warps of a pooled tile: with 32 columns four, which read all of them, and the other four take the next tile. (Eight warps with 16 columns
// each, all of them on every tile, set the kernel's time: 1200 clocks of latency a tile.) Unpooled tiles write four times as much, which is what bounds
// them, and eight warps write it sooner: 1024 x 16 x 32 x 32 to 16 channels 91 -> 47 us (with the words below).
__host__ __device__ constexpr int half_epilogue_groups(int BN, bool POOL) { return BN == 32 && POOL ? 2 : 1; }
__host__ __device__ constexpr int half_conv_warps(int BN, int C) { return half_groups(BN, C) * kHalfConvGroupWarps; }
__host__ __device__ constexpr int half_issuer_b(int BN, int C) { return 2 + kHalfEpiWarps + half_conv_warps(BN, C); }
__host__ __device__ constexpr int half_threads(int BN, int C) { return (half_issuer_b(BN, C) + 1) * 32; }

struct HalfConvParams {
   const float *X, *W, *bias; // NHWC, [Cout][3][3][C], [Cout] or nullptr
   float *Y;                  // NHWC, pooled or not
   int N, H, W_, Cout;
   int tilesH, tilesW, num_tiles;
   int relu;
};

template <int BN, int C>
struct HalfShared {
   uint64_t raw_full[kHalfMaxSlots], raw_empty[kHalfMaxSlots], op_full[kHalfMaxSlots], op_empty[kHalfMaxSlots];
   uint64_t tmem_full[half_buffers(BN)], tmem_empty[half_buffers(BN)], w_ready, drain[2];
   uint64_t careful_op_full[kHalfMaxSlots], careful_op_empty[kHalfMaxSlots]; // of the careful tiles' slots and accumulators
   uint64_t careful_tmem_full[half_buffers(BN)], careful_tmem_empty[half_buffers(BN)];
   uint32_t tmem_base;
   volatile uint32_t abort_flag;
   uint32_t w_found;                         // what some output channel's weights are
   uint32_t w_factors;                       // input channels have factors
   uint32_t w_largest[C];                    // largest weight of an input channel (twice its bits)
   __align__(16) float x_factor[C];
   __align__(16) float bias[BN], winv[BN];   // inverse scales of the output channels' weights
   __align__(16) float stands[BN];           // a sum of this size stands although values or weights have lost something (0: no weights, it always does)
   uint32_t row_found[BN];
   volatile float x_inv[kHalfScales];        // inverse scale of a tile's patch, negative when some of its values have lost something; 0: a careful tile
   uint2 red[half_groups(BN, C)][2][kHalfConvGroupWarps];
   uint32_t any_notes, notes[kHalfNoteWords];
   // Careful tiles, by converter group: of its passes in turn, and the bits of the patches' units of its tiles in turn. A pass or a patch is written when
   // the MMAs of at most the second last pass before it are done, which waited until the epilogue had read the second last accumulator before
   // that: four passes, and six tiles, are in use at most.
   volatile float careful_inv[kHalfCarefulGroups][4];
   volatile uint32_t careful_found[kHalfCarefulGroups][4];
   uint32_t nonzero[kHalfCarefulGroups][8][kHalfBitWords], infinite[kHalfCarefulGroups][8][kHalfBitWords], nan[kHalfCarefulGroups][8][kHalfBitWords];
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

// The scale that brings the largest magnitude into [2^14, 2^15), or 2^126 where that is less, and its inverse; what keeps the parts from holding
// the values (see the head of this file). Everything fits under 2^126: subnormal values are multiples of 2^-23 then, which two halves hold exactly.
__device__ __forceinline__ uint32_t half_scale(uint32_t largest, uint32_t smallest, float &scale, float &inverse)
{
   const uint32_t e = largest >> 24, e_small = (smallest + 1) >> 24;
   scale = inverse = 1.f;
   if (largest == 0) return 0;
   if (e == 255) return kHalfSpecial;
   const uint32_t lift = e > 15 ? e : 15;
   scale = __uint_as_float((268u - lift) << 23);
   inverse = __uint_as_float((lift - 14u) << 23);
   return e <= 15 || (e_small > 0 && e - e_small <= kHalfSpread) ? 0 : kHalfWide;
}

// One pixel's sums over all taps and input channels as chains of fp32 FMAs from global memory, without bias, by a whole warp: lane l gets that
// of output channel c + l % 16 (half of the input channels each for l / 16, then added).
template <int C>
__device__ __noinline__ float half_chains(const HalfConvParams &p, int n, int h, int w, int c, int lane)
{
   c = min(c + (lane & 15), p.Cout - 1);
   const int i0 = (lane >> 4) * (C / 2);
   float acc = 0.f;
#pragma unroll 3
   for (int tap = 0; tap < 9; tap++) {
      const int ih = h + tap / 3 - 1, iw = w + tap % 3 - 1;
      const bool in = ih >= 0 && ih < p.H && iw >= 0 && iw < p.W_;
      const float4 *x = reinterpret_cast<const float4 *>(p.X + (((size_t)n * p.H + (in ? ih : 0)) * p.W_ + (in ? iw : 0)) * C + i0);
      const float4 *wt = reinterpret_cast<const float4 *>(p.W + (size_t)(c * 9 + tap) * C + i0);
#pragma unroll
      for (int k = 0; k < C / 8; k++) {
         float4 xv = x[k];
         const float4 wv = __ldg(wt + k);
         if (!in) xv = make_float4(0.f, 0.f, 0.f, 0.f);
         acc = fmaf(xv.x, wv.x, acc);
         acc = fmaf(xv.y, wv.y, acc);
         acc = fmaf(xv.z, wv.z, acc);
         acc = fmaf(xv.w, wv.w, acc);
      }
   }
   return acc + __shfl_xor_sync(0xffffffffu, acc, 16);
}

// Whether the 3 x 3 window of the tile's pixel (row, col) holds a unit (of eight channels) that has its bit set
template <int C>
__device__ __forceinline__ bool half_window(const uint32_t *bits, int row, int col)
{
   uint32_t found = 0;
#pragma unroll
   for (int r = 0; r < 3; r++) {
      const int unit = ((row + r) * kHalfPatchW + col) * (C / 8);
      found |= __funnelshift_r(bits[unit >> 5], bits[(unit >> 5) + 1], unit & 31);
   }
   return (found & ((1u << (3 * C / 8)) - 1)) != 0;
}

// Two output channels of a pooled pixel / CH of a pixel
__device__ __forceinline__ void half_store_pair(float *y, int c, int Cout, bool pairs, float v0, float v1)
{
   if (pairs) {
      if (c < Cout) *reinterpret_cast<float2 *>(y) = make_float2(v0, v1);
   } else {
      if (c < Cout) y[0] = v0;
      if (c + 1 < Cout) y[1] = v1;
   }
}
// Whole 32-byte sectors where the row is aligned, else words of four channels as far as they go: 1024 x 16 x 32 x 32 to 64 channels 130 us in words,
// 106 in sectors; to 28 channels 176 us where a row that is not whole went out value by value, 59 in words.
template <int CH>
__device__ __forceinline__ void half_store_row(float *y, int c, int Cout, const float (&r)[CH])
{
   const uint32_t at = (uint32_t)reinterpret_cast<uintptr_t>(y);
   if (c + CH <= Cout && (at & 31) == 0) {
#pragma unroll
      for (int j = 0; j < CH; j += 8)
         asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(y + j), "f"(r[j]), "f"(r[j + 1]), "f"(r[j + 2]), "f"(r[j + 3]),
                      "f"(r[j + 4]), "f"(r[j + 5]), "f"(r[j + 6]), "f"(r[j + 7])
                      : "memory");
   } else {
      const bool words = (at & 15) == 0;
#pragma unroll
      for (int j = 0; j < CH; j += 4)
         if (words && c + j + 4 <= Cout) *reinterpret_cast<float4 *>(y + j) = make_float4(r[j], r[j + 1], r[j + 2], r[j + 3]);
         else
#pragma unroll
            for (int i = j; i < j + 4; i++)
               if (c + i < Cout) y[i] = r[i];
   }
}

// How a warp's lanes read an accumulator sixteen columns at a time: value i is of pixel `pos` of this lane (pooled: four pixels below
// one another, 16x256b; else one) and of channel c + channel(j), c of this lane.
template <bool POOL>
struct HalfLanes {
   static constexpr int POS = POOL ? 4 : 1, PER = 16 / POS;
   int c, col, row; // first channel, the lane's pixel in the tile (the first of the four)
   __device__ __forceinline__ HalfLanes(int warp, int lane)
      : c(POOL ? 2 * (lane & 3) : 0), col(POOL ? lane >> 2 : lane & 7), row((warp & 3) * 4 + (POOL ? 0 : lane >> 3)) {}
   static __device__ __forceinline__ constexpr int index(int pos, int j) { return POOL ? (pos >> 1) * 8 + (j >> 1) * 4 + (pos & 1) * 2 + (j & 1) : j; }
   static __device__ __forceinline__ constexpr int channel(int j) { return POOL ? (j >> 1) * 8 + (j & 1) : j; }
   template <int BN>
   static __device__ __forceinline__ void load(uint32_t taddr, float (&v)[16])
   {
      uint32_t a[16], b[16];
      if constexpr (POOL) {
         tmem_ld_16x256<16>(taddr, a);
         tmem_ld_16x256<16>(taddr + BN, b);
      } else {
         tmem_ld_cols<16>(taddr, a);
         tmem_ld_cols<16>(taddr + BN, b);
      }
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; i++) v[i] = fmaf(__uint_as_float(b[i]), 1.f / kHalfTrailing, __uint_as_float(a[i]));
   }
};

// Largest and smallest of a converter group's four warps; false (kHalfLeft is set) when one of them has given up.
template <int BN, int C>
__device__ __forceinline__ bool half_exchange(HalfShared<BN, C> &sh, int group, int gw, int lane, uint32_t &state, uint32_t &largest, uint32_t &smallest)
{
   largest = __reduce_max_sync(0xffffffffu, largest);
   smallest = __reduce_min_sync(0xffffffffu, smallest);
   uint2 *red = sh.red[group][state & kHalfTurn];
   state ^= kHalfTurn;
   if (lane == 0) red[gw] = make_uint2(largest, smallest);
   uint32_t all_ok;
   asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(all_ok)
                : "r"(state & kHalfOk), "r"(1 + group), "n"(kHalfConvGroupWarps * 32)
                : "memory");
#pragma unroll
   for (int i = 0; i < kHalfConvGroupWarps; i++) {
      const uint2 o = red[i];
      largest = max(largest, o.x);
      smallest = min(smallest, o.y);
   }
   if (!all_ok) state |= kHalfLeft;
   return all_ok != 0;
}

// The MMAs of one tile: patch parts at `op`, weights at `w`, accumulator at `d`
template <int BN, int C>
__device__ __forceinline__ void half_issue(uint32_t d, uint32_t op, uint32_t w)
{
   constexpr int RB = 2 * C, KSTEPS = C / 16, PART = half_part_bytes(C), W_ITEM = 2 * BN * RB;
   constexpr uint32_t idesc = make_idesc<kF16>(128, BN), idesc_wide = make_idesc<kF16>(128, 2 * BN);
   // eight pixels of a tile row are one 8-row group, the next group is one patch row further (make_smem_desc_rows)
   const uint64_t da0 = make_smem_desc_rows(op, RB, kHalfPatchW * RB), db0 = make_smem_desc(w, RB);
   const uint32_t a_hi_word = (uint32_t)(da0 >> 32), a_lo_word = (uint32_t)da0, b_hi_word = (uint32_t)(db0 >> 32), b_lo_word = (uint32_t)db0;
   auto adesc = [&](uint32_t off) { return ((uint64_t)a_hi_word << 32) | (uint64_t)(a_lo_word + (off >> 4)); };
   auto bdesc = [&](uint32_t off) { return ((uint64_t)b_hi_word << 32) | (uint64_t)(b_lo_word + (off >> 4)); };
#pragma unroll
   for (int tap = 0; tap < 9; tap++) {
#pragma unroll
      for (int k = 0; k < KSTEPS; k++) {
         const uint32_t a = (uint32_t)(((tap / 3) * kHalfPatchW + tap % 3) * RB + k * 32), b = (uint32_t)(tap * W_ITEM + k * 32);
         warp_mma<kF16>(d, adesc(a), bdesc(b), idesc_wide, (tap | k) ? 1u : 0u); // leading x [leading | trailing]
         warp_mma<kF16>(d + BN, adesc(a + PART), bdesc(b), idesc, 1u);           // trailing x leading
      }
   }
}

// A CTA's careful tiles in order, by the notes of the plain ones: bit b stands for tiles b << shift ... of the CTA's.
struct HalfNotes {
   const uint32_t *notes;
   int tiles, shift;
   bool all;
   static __device__ __forceinline__ int shift_for(int tiles)
   {
      int shift = 0;
      while ((tiles - 1) >> shift >= kHalfNoteWords * 32) shift++;
      return shift;
   }
   __device__ __forceinline__ int from(int lt) const // the next one from lt on, or `tiles`
   {
      while (lt < tiles && !all && !(notes[lt >> shift >> 5] >> (lt >> shift & 31) & 1)) {
         lt = ((lt >> shift) + 1) << shift;
         if ((lt >> shift & 31) == 0)
            while (lt < tiles && notes[lt >> shift >> 5] == 0) lt += 32 << shift;
      }
      return min(lt, tiles);
   }
};

// Where pass q of a converter group goes: every other slot or accumulator (`each` of them a group), and its barriers' phase
struct HalfPlace {
   int at;
   uint32_t phase;
   __device__ __forceinline__ HalfPlace(int group, int q, int each) : at(group + 2 * (q % each)), phase((uint32_t)(q / each) & 1u) {}
};

// Careful tiles, converter warp: patches are read from global memory and written to one of the group's slots for each scale.
template <int BN, int C>
__device__ __forceinline__ void half_careful_convert(const HalfConvParams &p, HalfShared<BN, C> &sh, const HalfNotes &notes, unsigned char *ops, int group, int gw, int lane,
                                                     uint32_t *status)
{
   constexpr int UPP = C / 8, GT = kHalfConvGroupWarps * 32, UNITS = kHalfPatchPixels * UPP, PER = (UNITS + GT - 1) / GT, PART = half_part_bytes(C);
   const int t = gw * 32 + lane;
   const bool factors = sh.w_factors != 0;
   uint32_t state = kHalfOk;
   int count = 0, q = 0;
   for (int lt = notes.from(0); lt < notes.tiles; lt = notes.from(lt + 1), count++) {
      if ((count & 1) != group) continue;
      const int tile = blockIdx.x + lt * gridDim.x, turn = count >> 1 & 7;
      const int tw = tile % p.tilesW, th = tile / p.tilesW % p.tilesH, n = tile / p.tilesW / p.tilesH;
      float v[PER][8];
#pragma unroll
      for (int i = 0; i < PER; i++) {
         const int u = t + i * GT, pixel = u / UPP, ih = th * kHalfTileH - 1 + pixel / kHalfPatchW, iw = tw * kHalfTileW - 1 + pixel % kHalfPatchW;
         float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
         if (u < UNITS && ih >= 0 && ih < p.H && iw >= 0 && iw < p.W_) {
            const float4 *x = reinterpret_cast<const float4 *>(p.X + (((size_t)n * p.H + ih) * p.W_ + iw) * C + u % UPP * 8);
            a = x[0];
            b = x[1];
         }
         v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w; v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
      }
      // what the units hold; infinities and NaNs as zeros, the rest times the channels' factors
      uint32_t special = 0, lossless = 1;
#pragma unroll
      for (int i = 0; i < PER; i++) {
         bool any = false, infinite = false, nan = false;
#pragma unroll
         for (int j = 0; j < 8; j++) {
            const uint32_t m = __float_as_uint(v[i][j]) << 1;
            infinite |= m == 0xff000000u;
            nan |= m > 0xff000000u;
            if (m >= 0xff000000u) v[i][j] = 0.f;
            any |= v[i][j] != 0.f;
         }
         if (factors) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
               const float f = sh.x_factor[t % UPP * 8 + j], x = v[i][j] * f;
               if (v[i][j] != 0.f && f != 0.f && fabsf(x) < __uint_as_float(0x00800000u)) lossless = 0; // the factor may have cost bits
               v[i][j] = x;
            }
         }
         const uint32_t any_bits = __ballot_sync(0xffffffffu, any), inf_bits = __ballot_sync(0xffffffffu, infinite), nan_bits = __ballot_sync(0xffffffffu, nan);
         const int word = gw + i * kHalfConvGroupWarps;
         if (lane == 0 && word < kHalfBitWords) {
            sh.nonzero[group][turn][word] = any_bits;
            sh.infinite[group][turn][word] = inf_bits;
            sh.nan[group][turn][word] = nan_bits;
         }
         special |= inf_bits | nan_bits;
      }
      if (!half_exchange(sh, group, gw, lane, state, special, lossless)) return;
      bool more = true;
      for (; more; q++) {
         uint32_t largest = 0, smallest = 0xffffffffu;
#pragma unroll
         for (int i = 0; i < PER; i++) half_extremes(v[i], largest, smallest);
         if (!half_exchange(sh, group, gw, lane, state, largest, smallest)) return;
         float scale, inverse;
         more = half_scale(largest, smallest, scale, inverse) == kHalfWide;
         const uint32_t e = largest >> 24, below = e > 15 ? max((int)e - (int)kHalfSpread, 1) : 0; // exponents under this wait for the next pass
         const HalfPlace slot(group, q, half_careful_slots(BN, C));
         const bool ok = (state & kHalfOk) && mbar_wait(&sh.careful_op_empty[slot.at], slot.phase ^ 1u, &sh.abort_flag, status, kStatusWaitEmpty, 0xa000 + lt);
         if (!ok) state &= ~kHalfOk; // and on to the group's next exchange
         if (t == 0) {
            sh.careful_inv[group][q & 3] = inverse;
            sh.careful_found[group][q & 3] = (more ? kHalfWide : 0) | (special ? kHalfSpecial : 0) | (lossless ? 0 : kHalfChains);
         }
         unsigned char *op = ops + (size_t)slot.at * 2 * PART;
#pragma unroll
         for (int i = 0; i < PER; i++) {
            const int u = t + i * GT;
            float now[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
               const bool in = __float_as_uint(v[i][j]) << 1 >> 24 >= below;
               now[j] = in ? v[i][j] : 0.f;
               if (in) v[i][j] = 0.f;
            }
            if (ok && u < UNITS) {
               uint4 hi, lo;
               half_split(now, scale, hi, lo);
               const uint32_t off = half_swizzled<2 * C>((uint32_t)u * 16);
               *reinterpret_cast<uint4 *>(op + off) = hi;
               *reinterpret_cast<uint4 *>(op + PART + off) = lo;
            }
         }
         fence_proxy_async();
         __syncwarp();
         if (ok && lane == 0) mbar_arrive(&sh.careful_op_full[slot.at]);
      }
   }
}

// Careful tiles, epilogue warp: its share of the columns of the accumulators. The sums are kept in local memory and the loops over them are not
// unrolled: most often there is one such tile among thousands, and fetching its instructions is what it costs (BN = 128 unrolled: 18 us).
template <int BN, int C, bool POOL>
__device__ __forceinline__ void half_careful_epilogue(const HalfConvParams &p, HalfShared<BN, C> &sh, const HalfNotes &notes, uint32_t taddr, int warp, int lane, uint32_t *status)
{
   using Lanes = HalfLanes<POOL>;
   constexpr int POS = Lanes::POS, PER = Lanes::PER;
   const Lanes l(warp, lane);
   const int c_begin = ((warp - 2) >> 2) * (BN / 2), columns = min(BN / 2, p.Cout - c_begin);
   const float inf = __uint_as_float(0x7f800000u);
   const uint32_t w_found = sh.w_found;
   int count = 0, q[2] = {0, 0};
#pragma unroll 1
   for (int lt = notes.from(0); lt < notes.tiles; lt = notes.from(lt + 1), count++) {
      const int group = count & 1, turn = count >> 1 & 7, tile = blockIdx.x + lt * gridDim.x;
      const int tw = tile % p.tilesW, th = tile / p.tilesW % p.tilesH, n = tile / p.tilesW / p.tilesH;
      uint32_t found = 0;
      float xinv0 = 0.f, v[BN / 2];
      bool more = true;
#pragma unroll 1
      for (int pass = 0; more; pass++, q[group]++) {
         const HalfPlace buf(group, q[group], half_buffers(BN) / 2);
         if (!mbar_wait(&sh.careful_tmem_full[buf.at], buf.phase, &sh.abort_flag, status, kStatusWaitAccum, 0x9000 + lt)) return;
         tc_fence_after();
         const float xinv = sh.careful_inv[group][q[group] & 3];
         const uint32_t x_found = sh.careful_found[group][q[group] & 3];
         if (pass == 0) xinv0 = xinv, found = x_found;
         more = x_found & kHalfWide;
#pragma unroll 1
         for (int k = 0; k < columns; k += 16) {
            float r[16];
            Lanes::template load<BN>(taddr + (uint32_t)(buf.at * 2 * BN + c_begin + k), r);
#pragma unroll
            for (int j = 0; j < PER; j++) {
               // times the two scales: their product, or one after the other, that which keeps the value in range first
               const float winv = sh.winv[c_begin + k + l.c + Lanes::channel(j)], f = xinv * winv;
               const bool one = f > 0.f && f < inf;
               const float first = one ? 1.f : f > 0.f ? fminf(xinv, winv) : fmaxf(xinv, winv), then = one ? f : f > 0.f ? fmaxf(xinv, winv) : fminf(xinv, winv);
#pragma unroll
               for (int pos = 0; pos < POS; pos++) {
                  float &x = v[k + pos * PER + j];
                  x = fmaf(r[Lanes::index(pos, j)] * first, then, pass == 0 ? 0.f : x);
               }
            }
         }
         tc_fence_before();
         __syncwarp();
         if (lane == 0) mbar_arrive(&sh.careful_tmem_empty[buf.at]); // the buffer is the issuer's again
      }
      const int h0 = th * kHalfTileH + l.row, w = tw * kHalfTileW + l.col;
      if ((found & ~kHalfWide) | w_found) {
#pragma unroll 1
         for (int pos = 0; pos < POS; pos++) {
            const bool nonzero = half_window<C>(sh.nonzero[group][turn], l.row + pos, l.col);
            const bool infinite = (found & kHalfSpecial) && half_window<C>(sh.infinite[group][turn], l.row + pos, l.col);
            const bool nan = (found & kHalfSpecial) && half_window<C>(sh.nan[group][turn], l.row + pos, l.col);
#pragma unroll 1
            for (int k = 0; k < columns; k += 16) {
               const int c = c_begin + k + l.c;
               float *x = v + k + pos * PER;
               uint32_t again = 0; // a bit for each of the pixel's values
#pragma unroll 4
               for (int j = 0; j < PER; j++) {
                  const uint32_t row_found = sh.row_found[c + Lanes::channel(j)];
                  const float stands = kHalfStands * (xinv0 * sh.winv[c + Lanes::channel(j)]);
                  const bool lost = (row_found & kHalfWide) && nonzero && !(stands > 0.f && fabsf(x[j]) >= stands);
                  if (nan) x[j] = __uint_as_float(0x7fffffffu);
                  else if ((found & kHalfChains) || (row_found & kHalfSpecial) || infinite || lost) again |= 1u << j;
               }
               // one pixel after the other: the first lane that has one, and those that have channels of the same pixel
               for (uint32_t lanes = __ballot_sync(0xffffffffu, again != 0); lanes != 0;) {
                  const int from = POOL ? (__ffs(lanes) - 1) & ~3 : __ffs(lanes) - 1;
                  lanes &= ~((POOL ? 0xfu : 1u) << from);
                  const float sum = half_chains<C>(p, n, __shfl_sync(0xffffffffu, h0, from) + pos, __shfl_sync(0xffffffffu, w, from), c_begin + k, lane);
                  const bool here = POOL ? (lane & ~3) == from : lane == from;
#pragma unroll 4
                  for (int j = 0; j < PER; j++) {
                     const float got = __shfl_sync(0xffffffffu, sum, l.c + Lanes::channel(j));
                     if (here && (again >> j & 1)) x[j] = got;
                  }
               }
            }
         }
      }
#pragma unroll 1
      for (int k = 0; k < columns; k += 16) {
         const int c = c_begin + k + l.c;
         if constexpr (POOL) {
            // a NaN loses against a number, as in the comparisons of the plain form; the window's other column is in lane ^ 4
            const bool second = (lane & 4) != 0;
            const int oh = (h0 >> 1) + (second ? 1 : 0), ow = tw * (kHalfTileW / 2) + (lane >> 3);
            float *y = p.Y + (((size_t)n * (p.H / 2) + oh) * (p.W_ / 2) + ow) * p.Cout + c;
            const bool pairs = ((p.Cout & 1) | (int)(reinterpret_cast<uintptr_t>(p.Y) & 7)) == 0;
            float m[PER];
#pragma unroll
            for (int j = 0; j < PER; j++) {
               const float m0 = fmaxf(v[k + j], v[k + PER + j]), m1 = fmaxf(v[k + 2 * PER + j], v[k + 3 * PER + j]);
               m[j] = fmaxf(second ? m1 : m0, __shfl_xor_sync(0xffffffffu, second ? m0 : m1, 4)) + sh.bias[c + Lanes::channel(j)];
               if (p.relu) m[j] = relu_ref(m[j]);
            }
#pragma unroll
            for (int j = 0; j < PER; j += 2) half_store_pair(y + Lanes::channel(j), c + Lanes::channel(j), p.Cout, pairs, m[j], m[j + 1]);
         } else {
            float r[16];
#pragma unroll
            for (int i = 0; i < 16; i++) {
               r[i] = v[k + i] + sh.bias[c + i];
               if (p.relu) r[i] = relu_ref(r[i]);
            }
            half_store_row<16>(p.Y + (((size_t)n * p.H + h0) * p.W_ + w) * p.Cout + c, c, p.Cout, r);
         }
      }
   }
}

// The tiles that the plain form has left, after all others and by all warps: a function of its own, so that its registers are not the others' (as
// calls within their loops it made the plain tiles a tenth slower).
template <int BN, int C, bool POOL>
__device__ __noinline__ void half_careful_tiles(const HalfConvParams &p, HalfShared<BN, C> &sh, unsigned char *w_smem, unsigned char *ops, int tiles, uint32_t *status)
{
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const HalfNotes notes = {sh.notes, tiles, HalfNotes::shift_for(tiles), (sh.w_found & kHalfSpecial) != 0};
   griddep_wait(); // the activations are read by these threads themselves
   if (warp == 1) {
      int count = 0, q[2] = {0, 0};
      for (int lt = notes.from(0); lt < notes.tiles; lt = notes.from(lt + 1), count++) {
         const int group = count & 1;
         bool more = true;
         for (; more; q[group]++) {
            const HalfPlace slot(group, q[group], half_careful_slots(BN, C)), buf(group, q[group], half_buffers(BN) / 2);
            if (!mbar_wait_warp(&sh.careful_op_full[slot.at], slot.phase, &sh.abort_flag, status, kStatusWaitConv, 0xb000 + lt) ||
                !mbar_wait_warp(&sh.careful_tmem_empty[buf.at], buf.phase ^ 1u, &sh.abort_flag, status, kStatusWaitAccum, 0xb000 + lt)) {
               warp_commit(&sh.drain[0]); // what is under way ends before the tensor memory is given back
               mbar_drain(&sh.drain[0], 0);
               return;
            }
            more = __any_sync(0xFFFFFFFFu, sh.careful_found[group][q[group] & 3] & kHalfWide);
            tc_fence_after();
            half_issue<BN, C>(sh.tmem_base + (uint32_t)(buf.at * 2 * BN), smem_u32(ops + (size_t)slot.at * 2 * half_part_bytes(C)), smem_u32(w_smem));
            warp_commit(&sh.careful_op_empty[slot.at]);
            warp_commit(&sh.careful_tmem_full[buf.at]);
         }
      }
   } else if (warp >= 2 && warp < 2 + kHalfEpiWarps) {
      half_careful_epilogue<BN, C, POOL>(p, sh, notes, sh.tmem_base + ((uint32_t)((warp & 3) * 32) << 16), warp, lane, status);
   } else if (warp >= 2 + kHalfEpiWarps && warp < 2 + kHalfEpiWarps + kHalfCarefulGroups * kHalfConvGroupWarps) {
      const int cw = warp - 2 - kHalfEpiWarps, group = cw / kHalfConvGroupWarps;
      half_careful_convert<BN, C>(p, sh, notes, ops, group, cw % kHalfConvGroupWarps, lane, status);
   }
}

template <int BN, int C, bool POOL>
__global__ void __launch_bounds__(half_threads(BN, C), 1)
umma_conv3x3_half_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ HalfConvParams p, uint32_t *status)
{
   constexpr int RB = 2 * C;                       // bytes of an operand row: one pixel's or one (tap, output channel)'s halves
   constexpr int PART = half_part_bytes(C), RAW = half_raw_bytes(C);
   constexpr int UPP = C / 8;                      // units of eight channels per pixel
   constexpr int W_ITEM = 2 * BN * RB;             // one tap's weights: BN leading rows, BN trailing rows
   constexpr int NBUF = half_buffers(BN);
   constexpr int SLOTS = half_slots(BN, C), GROUPS = half_groups(BN, C), ISSUER_B = half_issuer_b(BN, C), EPI_GROUPS = half_epilogue_groups(BN, POOL);
   static_assert(SLOTS % GROUPS == 0, "a slot always meets the same converter group");
   constexpr uint32_t TMEM_COLS = NBUF * 2 * BN;
   constexpr int CW = BN / 2 * EPI_GROUPS;         // channels per epilogue warp
   constexpr int CH = CW >= 32 ? 32 : CW;
   extern __shared__ unsigned char smem_raw[];
   unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
   unsigned char *w_smem = smem;                   // 9 items
   unsigned char *ops = w_smem + 9 * W_ITEM;       // SLOTS x (leading, trailing)
   unsigned char *raws = ops + (size_t)SLOTS * 2 * PART;
   __shared__ HalfShared<BN, C> sh;

   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   SOFIE_PROF_DECL
   griddep_launch_dependents(); // the next kernel may set itself up while this one runs
   for (int c = threadIdx.x; c < BN; c += half_threads(BN, C)) sh.bias[c] = (c < p.Cout && p.bias) ? p.bias[c] : 0.f;
   if (threadIdx.x < C) sh.w_largest[threadIdx.x] = 0;
   if (threadIdx.x < kHalfNoteWords) sh.notes[threadIdx.x] = 0;
   if (threadIdx.x == 0) {
      for (int s = 0; s < kHalfMaxSlots; s++) {
         mbar_init(&sh.raw_full[s], 1);
         mbar_init(&sh.raw_empty[s], kHalfConvGroupWarps);
         mbar_init(&sh.op_full[s], kHalfConvGroupWarps);
         mbar_init(&sh.op_empty[s], 1);
         mbar_init(&sh.careful_op_full[s], kHalfConvGroupWarps);
         mbar_init(&sh.careful_op_empty[s], 1);
      }
      for (int b = 0; b < NBUF; b++) {
         mbar_init(&sh.tmem_full[b], 1);
         mbar_init(&sh.tmem_empty[b], kHalfEpiWarps / EPI_GROUPS);
         mbar_init(&sh.careful_tmem_full[b], 1);
         mbar_init(&sh.careful_tmem_empty[b], kHalfEpiWarps);
      }
      mbar_init(&sh.w_ready, kHalfWeightWarps);
      for (int i = 0; i < 2; i++) mbar_init(&sh.drain[i], 1);
      sh.abort_flag = 0;
      sh.w_found = sh.any_notes = 0;
      fence_mbar_init();
      prefetch_tensormap(&tmX);
   }
   if (warp == 1) {
      tmem_alloc(&sh.tmem_base, TMEM_COLS);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = sh.tmem_base;
   const int tiles = (p.num_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x; // this CTA's

   if (warp == 0) {
      // ---------------- TMA producer: one box per tile ----------------
      griddep_wait(); // the activations are the previous kernel's output
      TileWalker tw;
      tw.init(blockIdx.x, gridDim.x, p.tilesH, p.tilesW);
      int s = 0, g = 0;
      uint32_t ph = 0;
      // when the weights send all tiles to the careful form, nobody looks at the patches
      auto unread = [&] { return __all_sync(0xFFFFFFFFu, mbar_wait(&sh.w_ready, 0, &sh.abort_flag, status, kStatusWaitConv, 0x8000) && (sh.w_found & kHalfSpecial)); };
      for (int tile = blockIdx.x; tile < p.num_tiles; tile += gridDim.x, g++, ring_next(s, ph, SLOTS), tw.next()) {
         if (g == SLOTS && unread()) break; // from the second round of slots on
         if (!SOFIE_PROF_WAIT(mbar_wait_warp(&sh.raw_empty[s], ph ^ 1, &sh.abort_flag, status, kStatusWaitEmpty, g))) break;
         warp_expect_tx(&sh.raw_full[s], RAW);
         // rows and columns start at -1: zero fill; the channel coordinate is 0
         warp_tma_load_4d(raws + (size_t)s * RAW, &tmX, 0, tw.tw * kHalfTileW - 1, tw.th * kHalfTileH - 1, tw.n, &sh.raw_full[s]);
      }
      drain_copies(sh.raw_full, s, ph, g, SLOTS); // and of patches that nobody looks at
   } else if (warp == 1 || warp == ISSUER_B) {
      // ---------------- MMA issuers: all tiles, or even and odd ones ----------------
      // one of them keeps the pipe full with 36 MMAs a tile (32 channels: 185 us instead of 199), two do with 18 (320 instead of 338)
      constexpr int ISSUERS = C == 32 ? 1 : 2;
      const bool plain = __all_sync(0xFFFFFFFFu, SOFIE_PROF_WAIT(mbar_wait(&sh.w_ready, 0, &sh.abort_flag, status, kStatusWaitConv, 0x4000)) && !(sh.w_found & kHalfSpecial));
      const uint32_t w = smem_u32(w_smem);
      const int step = gridDim.x, parity = warp == 1 ? 0 : 1;
      WarpWait wait;
      for (int lt = parity; plain && parity < ISSUERS && blockIdx.x + (long long)lt * step < p.num_tiles; lt += ISSUERS) {
         const int s = lt % SLOTS, buf = lt % NBUF;
         wait(&sh.op_full[s], (uint32_t)(lt / SLOTS) & 1u);
         wait(&sh.tmem_empty[buf], ((uint32_t)(lt / NBUF) & 1u) ^ 1u);
         tc_fence_after();
         half_issue<BN, C>(tmem_base + (uint32_t)(buf * 2 * BN), smem_u32(ops + (size_t)s * 2 * PART), w);
         wait.commit(&sh.op_empty[s]);
         wait.commit(&sh.tmem_full[buf]);
      }
      wait.finish(&sh.drain[parity], &sh.abort_flag, status, kStatusWaitConv, 0x2000);
   } else if (warp >= 2 + kHalfEpiWarps) {
      // ---------------- converters ----------------
      const int cw = warp - 2 - kHalfEpiWarps, group = cw / kHalfConvGroupWarps, gw = cw % kHalfConvGroupWarps;
      if (cw < kHalfWeightWarps) {
         // the weights, once per CTA, by the first converter warps: TPR neighbouring threads a row, each with the units of the same eight channels
         constexpr int TPR = kHalfWeightWarps * 32 / BN, UNITS = 9 * UPP, PER = (UNITS + TPR - 1) / TPR;
         static_assert(TPR >= 1 && 32 % TPR == 0, "the threads of a row are in one warp");
         static_assert(TPR % UPP == 0, "a thread's units are of the same channels");
         const int t = cw * 32 + lane, row = t / TPR, sub = t % TPR, c_first = sub % UPP * 8;
         const float4 *src = reinterpret_cast<const float4 *>(p.W + (size_t)(row < p.Cout ? row : 0) * 9 * C);
         float v[PER][8];
#pragma unroll
         for (int i = 0; i < PER; i++) {
            const int u = sub + i * TPR;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (u < UNITS && row < p.Cout) {
               a = __ldg(src + 2 * u);
               b = __ldg(src + 2 * u + 1);
            }
            v[i][0] = a.x; v[i][1] = a.y; v[i][2] = a.z; v[i][3] = a.w; v[i][4] = b.x; v[i][5] = b.y; v[i][6] = b.z; v[i][7] = b.w;
         }
         // the input channels' factors (a power of two: exact, unless a value becomes subnormal, which the converters look for)
#pragma unroll
         for (int j = 0; j < 8; j++) {
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < PER; i++) m = max(m, __float_as_uint(v[i][j]) << 1);
            // threads whose units are of the same channels are UPP lanes apart
#pragma unroll
            for (int o = UPP; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane < UPP) atomicMax(&sh.w_largest[c_first + j], m);
         }
         asm volatile("bar.sync %0, %1;" ::"n"(1 + GROUPS), "n"(kHalfWeightWarps * 32) : "memory");
         const uint32_t all = sh.w_largest[lane % C], high = __reduce_max_sync(0xffffffffu, all), low = __reduce_min_sync(0xffffffffu, all), e_high = max(high >> 24, 1u);
         if (high != 0 && e_high < 255 && (low == 0 || e_high - max(low >> 24, 1u) > kHalfChannelSpread)) {
            auto below = [&](uint32_t largest) { return min(e_high - max(largest >> 24, 1u), kHalfChannelFactor); }; // powers of two
#pragma unroll
            for (int j = 0; j < 8; j++) {
               const float factor = __uint_as_float((127u + below(sh.w_largest[c_first + j])) << 23);
#pragma unroll
               for (int i = 0; i < PER; i++) v[i][j] *= factor;
            }
            if (cw == 0) {
               if (lane < C) sh.x_factor[lane] = all == 0 ? 0.f : __uint_as_float((127u - below(all)) << 23);
               if (lane == 0) sh.w_factors = 1;
            }
         } else if (cw == 0 && lane == 0) {
            sh.w_factors = 0;
         }
         uint32_t largest = 0, smallest = 0xffffffffu;
#pragma unroll
         for (int i = 0; i < PER; i++) half_extremes(v[i], largest, smallest);
#pragma unroll
         for (int o = 1; o < TPR; o <<= 1) {
            largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, o));
            smallest = min(smallest, __shfl_xor_sync(0xffffffffu, smallest, o));
         }
         float scale, inverse;
         const uint32_t found = half_scale(largest, smallest, scale, inverse);
         if (sub == 0) {
            sh.winv[row] = inverse;
            sh.row_found[row] = found;
            sh.stands[row] = largest == 0 ? 0.f : kHalfStands;
            if (found) atomicOr(&sh.w_found, found);
         }
#pragma unroll
         for (int i = 0; i < PER; i++) {
            const int u = sub + i * TPR;
            if (u < UNITS) {
               uint4 hi, lo;
               half_split(v[i], scale, hi, lo);
               unsigned char *item = w_smem + (u / UPP) * W_ITEM;
               const uint32_t off = half_swizzled<RB>((uint32_t)(row * RB + (u % UPP) * 16));
               *reinterpret_cast<uint4 *>(item + off) = hi;
               *reinterpret_cast<uint4 *>(item + BN * RB + off) = lo;
            }
         }
         fence_proxy_async();
         __syncwarp();
         if (lane == 0) mbar_arrive(&sh.w_ready);
      }
      constexpr int GT = kHalfConvGroupWarps * 32, UNITS = kHalfPatchPixels * UPP, PER = (UNITS + GT - 1) / GT;
      const int t = gw * 32 + lane;
      // a warp whose wait gave up goes on to the group's barrier, where the four leave together: nobody waits there for one that has left
      // what all the weights are is known
      uint32_t state = mbar_wait(&sh.w_ready, 0, &sh.abort_flag, status, kStatusWaitConv, 0x8000) ? kHalfOk : 0, none = 0;
      const bool factors = sh.w_factors != 0, go = !(sh.w_found & kHalfSpecial);
      if (!go) half_exchange(sh, group, gw, lane, state, none, none); // a warp whose wait gave up may not know that, and goes on to an exchange
      for (int lt = group; go && lt < tiles; lt += GROUPS) {
         const int s = lt % SLOTS;
         if (!((state & kHalfOk) && SOFIE_PROF_WAIT(mbar_wait(&sh.raw_full[s], (uint32_t)(lt / SLOTS) & 1u, &sh.abort_flag, status, kStatusWaitFull, 0x6000 + lt)))) state = state & ~kHalfOk;
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
         if (factors) {
            const float4 fa = *reinterpret_cast<const float4 *>(sh.x_factor + t % UPP * 8), fb = *reinterpret_cast<const float4 *>(sh.x_factor + t % UPP * 8 + 4);
            const float f[8] = {fa.x, fa.y, fa.z, fa.w, fb.x, fb.y, fb.z, fb.w};
#pragma unroll
            for (int i = 0; i < PER; i++) half_extremes(v[i], largest, smallest);
            // a value that the smallest factor may make subnormal: the careful form looks closer
            const bool small = smallest < ((1 + kHalfChannelFactor) << 24) - 1;
            largest = 0;
            smallest = 0xffffffffu;
#pragma unroll
            for (int i = 0; i < PER; i++) {
#pragma unroll
               for (int j = 0; j < 8; j++) v[i][j] *= f[j];
               half_extremes(v[i], largest, smallest);
            }
            if (small) smallest = 0;
         } else {
#pragma unroll
            for (int i = 0; i < PER; i++) half_extremes(v[i], largest, smallest);
         }
         __syncwarp();
         if (lane == 0) mbar_arrive(&sh.raw_empty[s]); // the patch is in registers
         if (!half_exchange(sh, group, gw, lane, state, largest, smallest)) break;
         float scale, inverse;
         const uint32_t found = half_scale(largest, smallest, scale, inverse);
         const bool ok = SOFIE_PROF_WAIT(mbar_wait(&sh.op_empty[s], ((uint32_t)(lt / SLOTS) & 1u) ^ 1u, &sh.abort_flag, status, kStatusWaitEmpty, 0x7000 + lt));
         if (!ok) state = state & ~kHalfOk;
         // read by the epilogue after the tile's MMAs, which wait for this group's arrivals below
         if (t == 0) sh.x_inv[lt % kHalfScales] = found == 0 ? inverse : found == kHalfWide && !(factors && smallest < 0xffffffu) ? -inverse : 0.f;
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
         if (ok && lane == 0) mbar_arrive(&sh.op_full[s]);
      }
   } else {
      // ---------------- epilogue: warps 2..9, two per lane quarter, on the same tile or on two in turn ----------------
      const int egroup = EPI_GROUPS == 2 ? (warp - 2) >> 2 : 0, c_begin = EPI_GROUPS == 2 ? 0 : ((warp - 2) >> 2) * CW;
      const int lane_base = (warp & 3) * 32, step = EPI_GROUPS * gridDim.x;
      TileWalker tw;
      tw.init(blockIdx.x + egroup * gridDim.x, step, p.tilesH, p.tilesW);
      // the weights' scales and verdict are the converters'
      bool ok = SOFIE_PROF_WAIT(mbar_wait(&sh.w_ready, 0, &sh.abort_flag, status, kStatusWaitConv, 0x5000)) && !(sh.w_found & kHalfSpecial);
      // largest and smallest inverse scale of a channel's weights (positive: ordered as their bits are)
      uint32_t w_low = 0x7f800000u, w_high = 0;
      for (int c = lane; c < BN; c += 32) {
         w_low = min(w_low, __float_as_uint(sh.winv[c]));
         w_high = max(w_high, __float_as_uint(sh.winv[c]));
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
            winv2[k] = *reinterpret_cast<const float2 *>(sh.winv + c0 + c2 + 8 * k);
            bias2[k] = *reinterpret_cast<const float2 *>(sh.bias + c0 + c2 + 8 * k);
         }
      };
      load_constants(c_begin);
      const int note_shift = HalfNotes::shift_for(tiles);
      const bool w_lossy = sh.w_found != 0;
      int lt = egroup;
      for (int tile = blockIdx.x + egroup * gridDim.x; ok && tile < p.num_tiles; tile += step, lt += EPI_GROUPS, tw.next()) {
         const int buf = lt % NBUF;
         ok = SOFIE_PROF_WAIT(mbar_wait(&sh.tmem_full[buf], (uint32_t)(lt / NBUF) & 1u, &sh.abort_flag, status, kStatusWaitAccum, 0x3000 + lt));
         if (!ok) break;
         tc_fence_after();
         const float x_inv = sh.x_inv[lt % kHalfScales], xinv = fabsf(x_inv);
         const uint32_t t_row = tmem_base + ((uint32_t)lane_base << 16) + (uint32_t)(buf * 2 * BN);
         // a product of the inverse scales may be subnormal (an exact power of two all the same), but neither zero nor infinite
         const bool plain = xinv * winv_low > 0.f && xinv * winv_high < __uint_as_float(0x7f800000u);
         if (!plain || x_inv < 0.f || w_lossy) {
            bool stand = plain;
#pragma unroll 1
            for (int c = c_begin; stand && c < c_begin + CW; c += 16) {
               float v[16];
               HalfLanes<POOL>::template load<BN>(t_row + (uint32_t)c, v);
#pragma unroll
               for (int i = 0; i < 16; i++) stand &= fabsf(v[i]) >= sh.stands[POOL ? c + c2 + (i % 8 >> 2) * 8 + (i & 1) : c + i];
               stand = __all_sync(0xffffffffu, stand);
            }
            if (!stand && lane == 0) { // the careful form computes this tile again
               atomicOr(&sh.notes[lt >> note_shift >> 5], 1u << (lt >> note_shift & 31));
               sh.any_notes = 1;
            }
            if (!plain) {
               tc_fence_before();
               __syncwarp();
               if (lane == 0) mbar_arrive(&sh.tmem_empty[buf]);
               continue;
            }
         }
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
               if (lane == 0) mbar_arrive(&sh.tmem_empty[buf]);
            }
            if (c0 >= p.Cout) continue;
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
#pragma unroll
               for (int j = 0; j < CH / 4; j++) {
                  const int k = (j >> 1) * 4 + (j & 1);
                  const float m0 = r[k + 2] > r[k] ? r[k + 2] : r[k], m1 = r[CH / 2 + k + 2] > r[CH / 2 + k] ? r[CH / 2 + k + 2] : r[CH / 2 + k];
                  const float mine = second ? m1 : m0, got = __shfl_xor_sync(0xffffffffu, second ? m0 : m1, 4);
                  v[j] = finish(got > mine ? got : mine, (j & 1) ? winv2[j >> 1].y : winv2[j >> 1].x, (j & 1) ? bias2[j >> 1].y : bias2[j >> 1].x);
               }
               float *y = p.Y + (((size_t)tw.n * (p.H / 2) + oh) * (p.W_ / 2) + ow) * p.Cout + c0 + c2;
               const bool pairs = ((p.Cout & 1) | (int)(reinterpret_cast<uintptr_t>(p.Y) & 7)) == 0;
#pragma unroll
               for (int k = 0; k < CH / 8; k++) half_store_pair(y + 8 * k, c0 + c2 + 8 * k, p.Cout, pairs, v[2 * k], v[2 * k + 1]);
            } else {
               const int pix = lane_base + lane, h = tw.th * kHalfTileH + pix / kHalfTileW, w = tw.tw * kHalfTileW + pix % kHalfTileW;
#pragma unroll
               for (int j = 0; j < CH; j += 4) {
                  const float4 wi = *reinterpret_cast<const float4 *>(sh.winv + c0 + j), bi = *reinterpret_cast<const float4 *>(sh.bias + c0 + j);
                  r[j] = finish(r[j], wi.x, bi.x);
                  r[j + 1] = finish(r[j + 1], wi.y, bi.y);
                  r[j + 2] = finish(r[j + 2], wi.z, bi.z);
                  r[j + 3] = finish(r[j + 3], wi.w, bi.w);
               }
               half_store_row<CH>(p.Y + (((size_t)tw.n * p.H + h) * p.W_ + w) * p.Cout + c0, c0, p.Cout, r);
            }
         }
      }
   }
   SOFIE_PROF_REPORT(warp == 0 ? "producer" : (warp == 1 || warp == ISSUER_B ? "mma" : (warp < 2 + kHalfEpiWarps ? "epilogue" : "converter")));
   tc_fence_before();
   __syncthreads();
   if ((sh.any_notes || (sh.w_found & kHalfSpecial)) && !sh.abort_flag) {
      tc_fence_after();
      half_careful_tiles<BN, C, POOL>(p, sh, w_smem, ops, tiles, status);
      tc_fence_before();
      __syncthreads();
   }
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
   SOFIE_CUDA_TRY(launch_dependent(kern, dim3(grid), dim3(half_threads(BN, C)), smem, s, tmX, p, status));
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
