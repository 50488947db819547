// What the two fp32 GEMMs out of three bfloat16 parts share (umma_gemm_any.cu, umma_gemm_parts.cu): how an operand is read, the split
// of a value, the epilogue's arithmetic, and which sums the parts do not hold.
#pragma once

#include "umma.cuh"

namespace sofie {
namespace umma {
namespace {

constexpr int kAnyBM = 128;             // rows of the tile = TMEM lanes
constexpr int kAnyKE = 32;              // floats of K per stage: one 64-byte swizzle row of each of the three parts
constexpr int kAnyRow = kAnyKE * 2;

// How an operand of `rows` x K is read.
enum AnyMode { kVecK = 0, kScalarK = 1, kRowsContiguous = 2 };
struct AnyOperand {
   const float *p;
   long long ld; // distance of rows (kVecK, kScalarK) or of consecutive K (kRowsContiguous)
   int rows, mode;
};

// Two values in three bfloat16 parts each, packed: round, take off, twice. Both remainders are exact, and the second has at most
// seven bits, so that its upper half is all of it: p0 + p1 + p2 is the value itself.
__device__ __forceinline__ uint32_t any_part(float lo, float hi)
{
   uint32_t p;
   asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo)); // the first source lands in the upper half
   return p;
}
__device__ __forceinline__ void any_split(float x, float y, uint32_t &p0, uint32_t &p1, uint32_t &p2)
{
   p0 = any_part(x, y);
   x -= __uint_as_float(p0 << 16), y -= __uint_as_float(p0 & 0xFFFF0000u);
   p1 = any_part(x, y);
   x -= __uint_as_float(p1 << 16), y -= __uint_as_float(p1 & 0xFFFF0000u);
   p2 = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

struct AnyEpilogue {
   float alpha, beta;
   const float *C;
   float *Y;
   int bias_kind, relu, vec; // vec: rows of Y (and of a full C) start on 16-byte boundaries
   int unit;                 // stages added up in one TMEM buffer (the tensor core's sums truncate) before they are promoted
};

__device__ __forceinline__ float any_finish(const AnyEpilogue &ep, float v, float c)
{
   v = ep.alpha * v;
   if (ep.bias_kind) v += ep.beta * c;
   return ep.relu ? relu_ref(v) : v;
}

// The parts of an operand that is infinite, not a number or above the largest bfloat16 do not add up to it (Inf - Inf, Inf x 0), and
// those of one below 2^-110 lose bits to bfloat16's range. The first kind shows in the sum, the second where the sum is tiny too
// (and not where a factor above 2^14 or more lifts it back into the range; an operand below 2^-134 counts as zero). Such a sum is
// doubtful: it is taken again as the chain of FMAs that the CUDA-core kernel forms, term by term.
__device__ __forceinline__ bool any_doubtful(float v)
{
   const uint32_t e = __float_as_uint(v) & 0x7FFFFFFFu, tiny = 31u << 23; // 2^-96
   return e - tiny >= 0x7F800000u - tiny && e != 0u;
}

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
} // namespace
} // namespace umma
} // namespace sofie
