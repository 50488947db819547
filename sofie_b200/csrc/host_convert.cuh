// What the host does to a model input on its way into pinned memory: copy it, or quantise it while it copies. A quantised
// network reads its float input once, to quantise it; the host has to touch every one of those floats anyway when they lie in
// pageable memory, and what it puts on the wire is then a quarter of the bytes. The loops are plain C for the compiler to
// vectorise, with the IEEE division of the operator's definition (an AVX-512 core does 11 GB/s of floats, fourteen of a 16-core host 100
// together; eight do 66), and give the bytes the device kernels give (quantize_u8_*, quantize_e4m3_* in eltwise.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace sofie {

enum HostConvertKind { kHostCopy = 0, kHostU8 = 1, kHostE4M3 = 2 };

struct HostConvert {
   int kind = kHostCopy;
   float scale = 1.f;
   int zp = 0;
   // bytes of the source behind one byte of the destination
   size_t ratio() const { return kind == kHostCopy ? 1 : sizeof(float); }
};

inline float host_bits_to_float(uint32_t u)
{
   float f;
   std::memcpy(&f, &u, 4);
   return f;
}
inline uint32_t host_float_to_bits(float f)
{
   uint32_t u;
   std::memcpy(&u, &f, 4);
   return u;
}

// q = clamp(rint(x / scale), -zp, 255 - zp) + zp. The clamp first: then |v| <= 255 and adding 1.5 * 2^23 rounds to the nearest
// integer, ties to even. A NaN takes the lower bound, as on the device.
__attribute__((always_inline)) inline void host_quantize_u8_loop(uint8_t *__restrict__ y, const float *__restrict__ x, size_t n, float scale, int zp)
{
   const float lo = (float)(0 - zp), hi = (float)(255 - zp);
   for (size_t i = 0; i < n; i++) {
      float v = x[i] / scale;
      v = v > lo ? v : lo;
      v = v < hi ? v : hi;
      y[i] = (uint8_t)((int32_t)(host_float_to_bits(v + 12582912.f) - 0x4B400000u) + zp);
   }
}

// E4M3 of x / scale, nearest even, saturating at 448. Normal results: the fp32 word rounded to three mantissa bits and rebased from
// exponent bias 127 to 7. Below 2^-6 the codes are multiples of 2^-9, which is the spacing of fp32 between 2^14 and 2^15: adding
// 1.5 * 2^14 rounds to it.
__attribute__((always_inline)) inline void host_quantize_e4m3_loop(uint8_t *__restrict__ y, const float *__restrict__ x, size_t n, float scale)
{
   for (size_t i = 0; i < n; i++) {
      const float v = x[i] / scale;
      const uint32_t u = host_float_to_bits(v), sign = (u >> 24) & 0x80u;
      float a = host_bits_to_float(u & 0x7FFFFFFFu);
      a = a > 448.f ? 448.f : a;
      const uint32_t ua = host_float_to_bits(a);
      const uint32_t normal = ((ua + 0x7FFFFu + ((ua >> 20) & 1u)) >> 20) - (120u << 3);
      const uint32_t small = host_float_to_bits(a + 24576.f) - 0x46C00000u;
      const uint32_t code = (a < 0.015625f ? small : normal) | sign;
      y[i] = (uint8_t)(v == v ? code : 0x7Fu);
   }
}

// A copy past the caches, for results larger than they are: the lines of the destination are not fetched first. FP8 chain on 8192 rows
// (134 MB of results) 5.1 -> 4.35 ms per call on hosts whose memory gives about 85 GB/s.
#if defined(__x86_64__)
__attribute__((target("avx"), noinline)) inline void host_stream_avx(char *dst, const char *src, size_t bytes)
{
   size_t head = (64 - (reinterpret_cast<uintptr_t>(dst) & 63)) & 63;
   if (head > bytes) head = bytes;
   std::memcpy(dst, src, head);
   size_t i = head;
   for (; i + 64 <= bytes; i += 64) {
      const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(src + i)), b = _mm256_loadu_si256(reinterpret_cast<const __m256i *>(src + i + 32));
      _mm256_stream_si256(reinterpret_cast<__m256i *>(dst + i), a);
      _mm256_stream_si256(reinterpret_cast<__m256i *>(dst + i + 32), b);
   }
   std::memcpy(dst + i, src + i, bytes - i);
   _mm_sfence(); // before another thread is told that the piece is done
}
#endif
inline void host_stream_copy(void *dst, const void *src, size_t bytes)
{
#if defined(__x86_64__)
   static const bool avx = __builtin_cpu_supports("avx");
   if (avx) return host_stream_avx(static_cast<char *>(dst), static_cast<const char *>(src), bytes);
#endif
   std::memcpy(dst, src, bytes);
}

#if defined(__x86_64__)
#define SOFIE_HOST_V4 __attribute__((target("avx512f,avx512bw,avx512vl,avx512dq,prefer-vector-width=512"), optimize("O3"), noinline))
#define SOFIE_HOST_V3 __attribute__((target("avx2"), optimize("O3"), noinline))
SOFIE_HOST_V4 inline void host_quantize_u8_v4(uint8_t *y, const float *x, size_t n, float scale, int zp) { host_quantize_u8_loop(y, x, n, scale, zp); }
SOFIE_HOST_V3 inline void host_quantize_u8_v3(uint8_t *y, const float *x, size_t n, float scale, int zp) { host_quantize_u8_loop(y, x, n, scale, zp); }
SOFIE_HOST_V4 inline void host_quantize_e4m3_v4(uint8_t *y, const float *x, size_t n, float scale) { host_quantize_e4m3_loop(y, x, n, scale); }
SOFIE_HOST_V3 inline void host_quantize_e4m3_v3(uint8_t *y, const float *x, size_t n, float scale) { host_quantize_e4m3_loop(y, x, n, scale); }
#undef SOFIE_HOST_V4
#undef SOFIE_HOST_V3
inline int host_vector_level()
{
   static const int level = __builtin_cpu_supports("avx512bw") && __builtin_cpu_supports("avx512vl") && __builtin_cpu_supports("avx512dq") ? 4
                            : __builtin_cpu_supports("avx2")                                                                          ? 3
                                                                                                                                      : 0;
   return level;
}
#endif

// `bytes` destination bytes
inline void host_convert(const HostConvert &c, void *dst, const void *src, size_t bytes)
{
   if (c.kind == kHostCopy) {
      std::memcpy(dst, src, bytes);
      return;
   }
   uint8_t *y = static_cast<uint8_t *>(dst);
   const float *x = static_cast<const float *>(src);
#if defined(__x86_64__)
   const int level = host_vector_level();
   if (level == 4) return c.kind == kHostU8 ? host_quantize_u8_v4(y, x, bytes, c.scale, c.zp) : host_quantize_e4m3_v4(y, x, bytes, c.scale);
   if (level == 3) return c.kind == kHostU8 ? host_quantize_u8_v3(y, x, bytes, c.scale, c.zp) : host_quantize_e4m3_v3(y, x, bytes, c.scale);
#endif
   c.kind == kHostU8 ? host_quantize_u8_loop(y, x, bytes, c.scale, c.zp) : host_quantize_e4m3_loop(y, x, bytes, c.scale);
}

} // namespace sofie
