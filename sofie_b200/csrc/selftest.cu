// Self test of the bounded waits every tensor-core kernel of this library is built from.
//
// One CTA allocates tensor memory, initialises an mbarrier that nothing ever arrives on and lets two
// warps wait for it with the same helper the contraction kernels use (umma::mbar_wait), but with a cycle
// limit chosen by the caller instead of the library's one second. The first waiter whose limit runs out
// raises the CTA's abort flag and stores a code in the status word of the stream's context; the second
// waiter leaves through the abort flag; every thread then reaches the common exit, where the tensor
// memory is released. The kernel therefore ends by itself after `limit_cycles` SM clocks, nothing
// faults, and the context stays usable: exactly the path a contraction kernel takes when a copy it
// waits for never completes.
#include "umma.cuh"

namespace sofie {
namespace {

using namespace umma;

constexpr uint32_t kStatusSelfTest = 0x1ff;

__global__ void __launch_bounds__(96, 1) wait_timeout_kernel(uint32_t *status, long long limit_cycles, uint32_t *reached_exit)
{
   __shared__ uint64_t never_bar;
   __shared__ uint32_t tmem_base_holder;
   __shared__ volatile uint32_t abort_flag;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   if (threadIdx.x == 0) {
      mbar_init(&never_bar, 1);
      abort_flag = 0;
      fence_mbar_init();
   }
   if (warp == 1) {
      tmem_alloc(&tmem_base_holder, 32);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = tmem_base_holder;
   if (warp == 0 && lane == 0) {
      // the role whose wait runs out
      (void)mbar_wait(&never_bar, 0, &abort_flag, status, kStatusSelfTest, 0x7e57, limit_cycles);
   } else if (warp == 2 && lane == 0) {
      // a role with the library's own (one second) limit: it leaves because the CTA was aborted
      (void)mbar_wait(&never_bar, 0, &abort_flag, nullptr, kStatusSelfTest, 0x7e58);
   }
   tc_fence_before();
   __syncthreads();
   if (warp == 1) {
      __syncwarp();
      tc_fence_after();
      tmem_dealloc(tmem_base, 32);
   }
   if (threadIdx.x == 0 && reached_exit) *reached_exit = 1u;
}

// The same for the waits of whole warps: a copying, an MMA-issuing and a reading role over a ring of two stages, in the form the contraction
// kernels have. One wait in the fourth of their eight stages, the issuer's (role 1) or the copying warp's (role 2), is for a barrier that
// nothing arrives on and has the caller's limit. out: 1 at the exit | stages copied | accumulators handed to the reader | 1 when the issuer gave
// up | 1 when every copy had landed at the exit.
constexpr int kTestStages = 8, kTestRing = 2, kTestStageBytes = 4096, kTestRows = 32; // 128 and 32 rows of 32 bytes
__global__ void __launch_bounds__(96, 1) warp_waits_kernel(uint32_t *status, int role, long long limit_cycles, uint32_t polls, const unsigned char *src, uint32_t *out)
{
   __shared__ __align__(1024) unsigned char stages[kTestRing * kTestStageBytes], weights[kTestRows * 32];
   __shared__ uint64_t full_bar[kTestRing], empty_bar[kTestRing], tmem_full, never_bar, drain_bar;
   __shared__ uint32_t tmem_base_holder, copied, handed_over, gave_up;
   __shared__ volatile uint32_t abort_flag;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   for (int i = threadIdx.x; i < kTestRows * 32; i += 96) weights[i] = 1;
   fence_proxy_async();
   if (threadIdx.x == 0) {
      for (int s = 0; s < kTestRing; s++) {
         mbar_init(&full_bar[s], 1);
         mbar_init(&empty_bar[s], 1);
      }
      mbar_init(&tmem_full, 1);
      mbar_init(&never_bar, 1);
      mbar_init(&drain_bar, 1);
      abort_flag = copied = handed_over = gave_up = 0;
      fence_mbar_init();
   }
   if (warp == 1) {
      tmem_alloc(&tmem_base_holder, 32);
      tmem_relinquish();
   }
   tc_fence_before();
   __syncthreads();
   tc_fence_after();
   const uint32_t tmem_base = tmem_base_holder;
   if (warp == 0) {
      int g = 0, s = 0;
      uint32_t ph = 0;
      for (; g < kTestStages; g++, ring_next(s, ph, kTestRing)) {
         if (role == 2 && g == 3 && !mbar_wait_warp(&never_bar, 0, &abort_flag, status, kStatusSelfTest, 0x7e59, limit_cycles)) break;
         if (!mbar_wait_warp(&empty_bar[s], ph ^ 1, &abort_flag, status, kStatusSelfTest, 0x7e5a)) break;
         warp_expect_tx(&full_bar[s], kTestStageBytes);
         warp_bulk_load(stages + s * kTestStageBytes, src, kTestStageBytes, &full_bar[s]);
      }
      drain_copies(full_bar, s, ph, g, kTestRing);
      if (lane == 0) copied = g;
   } else if (warp == 1) {
      constexpr uint32_t idesc = make_idesc<kI8>(128, kTestRows);
      const uint64_t db = make_smem_desc_noswizzle(smem_u32(weights), kTestRows * 16, 128);
      int s = 0;
      uint32_t ph = 0;
      WarpWait wait;
      wait.limit = kPollLimit / 16; // it does not see the flag: a quarter of a second
      for (int g = 0; g < kTestStages; g++, ring_next(s, ph, kTestRing)) {
         if (role == 1 && g == 3) {
            wait.limit = polls;
            wait(&never_bar, 0);
         }
         wait(&full_bar[s], ph);
         tc_fence_after();
         warp_mma<kI8>(tmem_base, make_smem_desc_noswizzle(smem_u32(stages + s * kTestStageBytes), 128 * 16, 128), db, idesc, g ? 1u : 0u);
         wait.commit(&empty_bar[s]);
      }
      wait.commit(&tmem_full);
      wait.finish(&drain_bar, &abort_flag, status, kStatusSelfTest, 0x7e5c);
      if (lane == 0) gave_up = wait.gave_up != 0;
   } else if (mbar_wait(&tmem_full, 0, &abort_flag, nullptr, kStatusSelfTest, 0x7e5b)) {
      tc_fence_after();
      uint32_t r[8];
      tmem_ld_32x8(tmem_base + (64u << 16), r); // warp 2 reads its quarter of the lanes
      tmem_ld_wait();
      if (lane == 0) handed_over = r[0] == 32u * kTestStages * src[0] ? 1 : 2;
   }
   tc_fence_before();
   __syncthreads();
   if (warp == 1) {
      __syncwarp();
      tc_fence_after();
      tmem_dealloc(tmem_base, 32);
   }
   if (threadIdx.x == 0) {
      bool landed = true; // the last copies of both slots
      for (int g = copied < kTestRing ? 0 : copied - kTestRing; g < (int)copied; g++) landed &= mbar_try_wait(&full_bar[g % kTestRing], (uint32_t)(g / kTestRing) & 1u);
      out[0] = 1;
      out[1] = copied;
      out[2] = handed_over;
      out[3] = gave_up;
      out[4] = landed;
   }
}

} // namespace
} // namespace sofie

extern "C" int sofie_cuda_selftest_wait_timeout(void *stream, int64_t limit_cycles, uint32_t *reached_exit_device)
{
   using namespace sofie;
   SOFIE_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000LL, "limit_cycles must be in (0, 2e8]: this is a test of a short wait");
   cudaStream_t s = as_stream(stream);
   uint32_t *status = device_status_word(s);
   if (!status) return fail(SOFIE_CUDA_ERR_CUDA, "cannot obtain the status word");
   wait_timeout_kernel<<<1, 96, 0, s>>>(status, (long long)limit_cycles, reached_exit_device);
   SOFIE_LAUNCH_CHECK("wait_timeout_kernel");
   return SOFIE_CUDA_OK;
}

extern "C" int sofie_cuda_selftest_warp_waits(void *stream, int32_t role, int64_t limit_cycles, const void *src_device, uint32_t *out_device)
{
   using namespace sofie;
   SOFIE_REQUIRE(role >= 0 && role <= 2, "role must be 0 (no wait runs out), 1 (the issuer's) or 2 (the copying warp's)");
   SOFIE_REQUIRE(limit_cycles > 0 && limit_cycles <= 200000000LL, "limit_cycles must be in (0, 2e8]: this is a test of a short wait");
   SOFIE_REQUIRE(src_device && out_device && (reinterpret_cast<uintptr_t>(src_device) & 15) == 0, "NULL or misaligned argument");
   cudaStream_t s = as_stream(stream);
   uint32_t *status = device_status_word(s);
   if (!status) return fail(SOFIE_CUDA_ERR_CUDA, "cannot obtain the status word");
   uint32_t polls = 1; // the issuer's waits count polls: a power of two of them, of some 8000 clocks each
   while (polls * 8000LL < limit_cycles) polls *= 2;
   warp_waits_kernel<<<1, 96, 0, s>>>(status, role, (long long)limit_cycles, polls, static_cast<const unsigned char *>(src_device), out_device);
   SOFIE_LAUNCH_CHECK("warp_waits_kernel");
   return SOFIE_CUDA_OK;
}
