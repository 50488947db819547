// Shared host/device helpers of libSOFIE_cuda: status handling, launch checks, small math.
#pragma once

#include <cuda_runtime.h>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "sofie_cuda.h"

namespace sofie {

// Thread-local text of the last failure, returned by sofie_cuda_last_error().
char *last_error_buffer();
int fail(int status, const char *fmt, ...);
void set_last_engine(int engine);
int forced_engine();

// Status word of the kernels that have bounded waits. A kernel that gives up stores a non-zero code
// there and returns normally, so the context stays usable. A stream that belongs to a context reports
// into that context's own word, which lies in mapped pinned host memory: sofie_cuda_ctx_fetch and
// sofie_cuda_ctx_check read it with a plain host load after the stream synchronisation they do anyway,
// and one Session never sees (or clears) another Session's failure. Launches on any other stream share
// one word per device in device memory, read by sofie_cuda_device_check().
uint32_t *device_status_word(cudaStream_t stream); // address the kernel writes to, nullptr on failure
void register_stream_status(cudaStream_t stream, uint32_t *word);
void unregister_stream_status(cudaStream_t stream);

#define SOFIE_CUDA_TRY(expr)                                                                         \
   do {                                                                                              \
      cudaError_t err__ = (expr);                                                                    \
      if (err__ != cudaSuccess)                                                                      \
         return ::sofie::fail(SOFIE_CUDA_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,                   \
                              cudaGetErrorString(err__), __FILE__, __LINE__);                        \
   } while (0)

#define SOFIE_LAUNCH_CHECK(name)                                                                     \
   do {                                                                                              \
      cudaError_t err__ = cudaGetLastError();                                                        \
      if (err__ != cudaSuccess)                                                                      \
         return ::sofie::fail(SOFIE_CUDA_ERR_CUDA, "launch of %s failed: %s", name,                  \
                              cudaGetErrorString(err__));                                            \
   } while (0)

#define SOFIE_REQUIRE(cond, ...)                                                                     \
   do {                                                                                              \
      if (!(cond)) return ::sofie::fail(SOFIE_CUDA_ERR_INVALID, __VA_ARGS__);                        \
   } while (0)

inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

constexpr int kNumSMs = 148; // B200

// ---- programmatic dependent launch ---------------------------------------------------------------
// A kernel launched with launch_dependent() may start while the kernel before it on the stream is
// still running: its blocks become resident as soon as every block of the predecessor has executed
// griddep_launch_dependents() (or exited) and resources are free, run their prologue (barrier setup,
// TMEM allocation, constant weights into shared memory) and then block in griddep_wait() until the
// predecessor has completed and its writes are visible. Rules kept by every kernel launched this way:
// every block executes griddep_wait() before it reads or writes anything another kernel touches and
// before it exits (so that completion of this grid implies completion of all earlier ones); only
// constant data (weights, biases, descriptors) is touched before it. Both instructions are no-ops in
// a kernel that was launched the ordinary way. SOFIE_CUDA_PDL=0 turns the attribute off.
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// `dependent`: the kernel's restrict pointers to what it reads behind the wait. What such a pointer leads to no statement of the kernel can write, so the compiler may take a load through it before the
// wait (and one of __ldg through any pointer); behind an empty statement that might have changed the pointer itself it may not.
template <typename P>
__device__ __forceinline__ void may_have_changed(P &pointer) { asm volatile("" : "+l"(pointer)); }
template <typename... P>
__device__ __forceinline__ void griddep_wait(P &...dependent)
{
   asm volatile("griddepcontrol.wait;" ::: "memory");
   (may_have_changed(dependent), ...);
}
// A load through such a pointer that may move freely behind the wait, before stores too (what the pointer leads to does not change any more): where a loop's loads are to be under way together.
__device__ __forceinline__ uint8_t load_settled(const uint8_t *p)
{
   uint32_t v;
   asm("ld.global.u8 %0, [%1];" : "=r"(v) : "l"(p));
   return (uint8_t)v;
}
__device__ __forceinline__ float load_settled(const float *p)
{
   float v;
   asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
   return v;
}
__device__ __forceinline__ float4 load_settled(const float4 *p)
{
   float4 v;
   asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
   return v;
}
// A read of what an earlier kernel wrote that stays where it is written.
__device__ __forceinline__ float load_dependent(const float *p)
{
   float v;
   asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
   return v;
}
bool pdl_enabled();

template <typename... KArgs, typename... Args>
cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args)
{
   cudaLaunchConfig_t cfg = {};
   cfg.gridDim = grid;
   cfg.blockDim = block;
   cfg.dynamicSmemBytes = smem;
   cfg.stream = stream;
   cudaLaunchAttribute attr[1];
   attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
   cfg.attrs = attr;
   cfg.numAttrs = 1;
   return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename T>
__host__ __device__ constexpr T ceil_div(T a, T b)
{
   return (a + b - 1) / b;
}

// ---- division of 32-bit indices by a number known at launch ---------------------------------------
// q = floor(n / d) for n < 2^31 as one multiplication and a shift: with p = 31 + ceil(log2 d) and m = ceil(2^p / d), which fits in
// 32 bits, floor(n * m / 2^p) is exact (round-up method).
struct FastDiv {
   uint32_t d = 1, m = 0, s = 0;
   FastDiv() = default;
   explicit FastDiv(uint32_t divisor) : d(divisor)
   {
      if (d <= 1) return; // n / 1: no multiplication
      uint32_t log = 0;
      while ((uint64_t(1) << log) < d) log++;
      m = (uint32_t)(((uint64_t(1) << (31 + log)) + d - 1) / d);
      s = log - 1;
   }
   __device__ __forceinline__ uint32_t div(uint32_t n) const { return d <= 1 ? n : __umulhi(n, m) >> s; }
   __device__ __forceinline__ uint32_t divmod(uint32_t n, uint32_t &rem) const
   {
      const uint32_t q = div(n);
      rem = n - q * d;
      return q;
   }
};

// Dynamic shared memory above 48 KB has to be allowed per kernel and device; the launchers call this on every launch. The allowance
// belongs to the function, for all threads of the process, and setting a smaller one lowers it: it is only ever raised here, under
// one lock, so that no thread's launch (nor the replay of a kernel captured earlier) is refused because another needed less.
inline cudaError_t allow_smem(const void *kernel, int bytes)
{
   static std::mutex mu;
   static std::map<std::pair<const void *, int>, int> allowed;
   int dev = 0;
   cudaError_t err = cudaGetDevice(&dev);
   if (err != cudaSuccess) return err;
   try {
      std::lock_guard<std::mutex> lock(mu);
      int &now = allowed[{kernel, dev}];
      if (now >= bytes) return cudaSuccess;
      err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
      if (err == cudaSuccess) now = bytes;
   } catch (...) {
      return cudaErrorMemoryAllocation; // the callers are C functions
   }
   return err;
}

// CTAs of kernels of one CTA an SM (their shared memory takes more than half of one) that run at a time in clusters of 1, 2, 4 and 8, for the estimates that cut a product along K. Cards
// differ with the SMs that their processing clusters have (132 and 140 of 148 were seen at four, 104 and 120 at eight), and a cluster too many costs a whole round: the least seen. One
// figure for every card, not the one a product runs on, since the cut decides the last bits of its sums: a model gives the same result on all of them.
constexpr int kClusterRoom[4] = {kNumSMs, kNumSMs, 132, 104};

// ---- requantisation recipe shared by every int8 kernel -------------------------------------------
// q = clamp(rne((float)acc * mult), qmin - zp, qmax - zp) + zp, with no FMA contraction, so a CPU
// evaluating nearbyintf((float)acc * mult) under the default rounding mode gets the same bits.
__device__ __forceinline__ int requant_u8(int acc, float mult, int y_zp, int relu)
{
   // The clamp runs on the float product, the rounding after it: clamp(rne(v), lo, hi) == rne(clamp(v, lo, hi)) for
   // integer bounds because rounding is monotone. A clamped value lies in [-255, 255], where adding 1.5 * 2^23
   // rounds it to the nearest integer, ties to even, in the adder (full rate) and leaves that integer in the low
   // mantissa bits; the float-to-int conversion instruction this replaces runs at a fraction of that rate.
   // Relu on a quantised value, max(q, y_zp), is the lower bound 0 before the zero point is added.
   float v = __fmul_rn(__int2float_rn(acc), mult);
   if (y_zp == 0) {
      // zero point 0: the clamp to [0, 255] (whose lower bound is also the Relu) and the rounding are ONE conversion with
      // round-to-nearest-even and saturation to the uint8 range
      uint32_t q;
      asm("cvt.rni.sat.u8.f32 %0, %1;" : "=r"(q) : "f"(v));
      return (int)q;
   }
   const float lo = relu ? 0.f : (float)(-y_zp), hi = (float)(255 - y_zp);
   v = fminf(fmaxf(v, lo), hi);
   return __float_as_int(__fadd_rn(v, 12582912.f)) - 0x4B400000 + y_zp;
}

// ---- two fp32 values per instruction, each rounded as by the scalar one ------------------------
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi)
{
   uint64_t v;
   asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
   return v;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c)
{
   uint64_t v;
   asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
   return v;
}

// 32 bytes of a 32-byte aligned row in one load
__device__ __forceinline__ void load_f32x8(const float *p, float (&v)[8])
{
   asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                : "l"(p));
}
// 32 bytes of a 32-byte aligned row in one store: a whole sector per thread
__device__ __forceinline__ void store_f32x8(float *p, const float *v)
{
   asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
                "f"(v[5]), "f"(v[6]), "f"(v[7])
                : "memory");
}

__device__ __forceinline__ float relu_ref(float v)
{
   // The reference's `x > 0 ? x : 0`: NaN and -0 both become +0.
   return v > 0.f ? v : 0.f;
}

__device__ __forceinline__ uint16_t f32_to_bf16_rne(float x)
{
   uint32_t u = __float_as_uint(x);
   if ((u & 0x7FFFFFFFu) > 0x7F800000u) return (uint16_t)((u >> 16) | 0x40);
   u += 0x7FFFu + ((u >> 16) & 1u);
   return (uint16_t)(u >> 16);
}

__device__ __forceinline__ float bf16_to_f32(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }

} // namespace sofie
