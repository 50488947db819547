// Helper threads for the host's share of a transfer: moving bytes between the caller's pageable memory and pinned memory. One core moves 14 GB/s on the Xeon hosts measured, a quarter of what the PCIe link takes (55 GB/s each way);
// four reach 54 GB/s and eight 110 GB/s as long as the pinned side stays in the last-level cache.
#pragma once

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "host_convert.cuh"

namespace sofie {

// A job is cut into numbered pieces that the caller and the helpers claim one after the other, so a helper that is still
// asleep or was descheduled delays nothing but the piece it holds. A claim carries the job's generation: a helper that comes
// late finds another generation (or no piece left) and touches nothing of the next job. Helpers spin for half a millisecond
// after a job (the next one of the same transfer comes within that time, and waking a sleeping thread costs tens of
// microseconds), then sleep on a condition variable. They end with the pool.
class HostPool {
public:
   using PieceFn = void (*)(void *arg, size_t piece);
   explicit HostPool(int helpers)
   {
      try {
         for (int i = 0; i < helpers; i++) threads_.emplace_back([this] { helper(); });
      } catch (...) { // no more threads to be had: those there are, and the caller, do the work
      }
   }
   ~HostPool()
   {
      {
         std::lock_guard<std::mutex> lock(mu_);
         stop_.store(true);
      }
      wake_.notify_all();
      for (auto &t : threads_) t.join();
   }
   HostPool(const HostPool &) = delete;
   HostPool &operator=(const HostPool &) = delete;

   // Starts fn(arg, i) for every i below `pieces` (at most 2^31), in any order, on the helpers; `arg` stays valid until
   // finish(), which takes part in what is left and returns when all is done. One caller at a time, one job at a time.
   void begin(PieceFn fn, void *arg, size_t pieces)
   {
      finish();
      if (threads_.empty() || pieces <= 1) { // nothing to share: the caller does it in finish()
         own_fn_ = fn, own_arg_ = arg, own_pieces_ = pieces;
         return;
      }
      // a helper that still holds the last job's ticket must not claim with the new job's piece count: the ticket is closed
      // (odd generation, no piece can be claimed) while the job's fields change
      ticket_.store(((uint64_t)++generation_ << 32) | 0xFFFFFFFFu, std::memory_order_seq_cst);
      std::atomic_thread_fence(std::memory_order_seq_cst);
      fn_ = fn, arg_ = arg;
      pieces_.store((uint32_t)pieces, std::memory_order_relaxed);
      done_.store(0, std::memory_order_relaxed);
      open_ = true;
      ticket_.store((uint64_t)++generation_ << 32, std::memory_order_seq_cst);
      if (sleepers_.load(std::memory_order_seq_cst) > 0) {
         std::lock_guard<std::mutex> lock(mu_);
         wake_.notify_all();
      }
   }
   void finish()
   {
      for (size_t i = 0; i < own_pieces_; i++) own_fn_(own_arg_, i);
      own_pieces_ = 0;
      if (!open_) return;
      claim(generation_);
      while (done_.load(std::memory_order_acquire) != pieces_.load(std::memory_order_relaxed)) relax();
      open_ = false;
   }
   void run(PieceFn fn, void *arg, size_t pieces)
   {
      begin(fn, arg, pieces);
      finish();
   }
   size_t threads() const { return threads_.size() + 1; }

   // A copy below kAloneBytes is the caller's alone: two threads' hand-over costs as much as it saves.
   // past_caches: the destination is part of something larger than the host's caches.
   void copy(void *dst, const void *src, size_t bytes, bool past_caches = false)
   {
      if (threads_.empty() || bytes < kAloneBytes) {
         std::memcpy(dst, src, bytes);
         return;
      }
      CopyJob job{static_cast<char *>(dst), static_cast<const char *>(src), bytes, kPieceBytes, past_caches};
      // enough pieces that every thread gets several, each still long enough for the prefetchers
      while (job.piece > size_t(32) << 10 && bytes / job.piece < 3 * (threads_.size() + 1)) job.piece >>= 1;
      run(copy_piece, &job, (bytes + job.piece - 1) / job.piece);
   }

   static constexpr size_t kAloneBytes = size_t(96) << 10;
   static constexpr size_t kPieceBytes = size_t(256) << 10;

private:
   struct CopyJob {
      char *dst;
      const char *src;
      size_t bytes, piece;
      bool past_caches;
   };
   static void copy_piece(void *arg, size_t i)
   {
      const CopyJob &j = *static_cast<CopyJob *>(arg);
      const size_t off = i * j.piece, n = j.bytes - off < j.piece ? j.bytes - off : j.piece;
      if (j.past_caches) host_stream_copy(j.dst + off, j.src + off, n);
      else std::memcpy(j.dst + off, j.src + off, n);
   }
   static void relax()
   {
#if defined(__x86_64__)
      __builtin_ia32_pause();
#else
      std::this_thread::yield();
#endif
   }
   // takes pieces of job `gen` until none is left; the job's fields are stable while one of its pieces is not done
   void claim(uint32_t gen)
   {
      uint64_t t = ticket_.load(std::memory_order_acquire);
      for (;;) {
         if ((uint32_t)(t >> 32) != gen || (uint32_t)t >= pieces_.load(std::memory_order_relaxed)) return;
         if (!ticket_.compare_exchange_weak(t, t + 1, std::memory_order_acq_rel, std::memory_order_acquire)) continue;
         fn_(arg_, (uint32_t)t);
         done_.fetch_add(1, std::memory_order_release);
         t = ticket_.load(std::memory_order_acquire);
      }
   }
   void helper()
   {
      uint32_t seen = 0;
      auto news = [&] { return stop_.load(std::memory_order_relaxed) || (uint32_t)(ticket_.load(std::memory_order_seq_cst) >> 32) != seen; };
      for (;;) {
         const auto t0 = std::chrono::steady_clock::now();
         while (!news()) {
            for (int i = 0; i < 32 && !news(); i++) relax();
            if (std::chrono::steady_clock::now() - t0 < std::chrono::microseconds(500)) continue;
            std::unique_lock<std::mutex> lock(mu_);
            sleepers_.fetch_add(1, std::memory_order_seq_cst); // before the last look: begin() reads it after it has published
            wake_.wait(lock, news);
            sleepers_.fetch_sub(1, std::memory_order_relaxed);
         }
         if (stop_.load()) return;
         seen = (uint32_t)(ticket_.load(std::memory_order_acquire) >> 32);
         claim(seen);
      }
   }
   std::vector<std::thread> threads_;
   std::mutex mu_;
   std::condition_variable wake_;
   PieceFn fn_ = nullptr, own_fn_ = nullptr;
   void *arg_ = nullptr, *own_arg_ = nullptr;
   size_t own_pieces_ = 0;
   bool open_ = false;
   std::atomic<uint32_t> pieces_{0};
   uint32_t generation_ = 0;
   std::atomic<uint64_t> ticket_{0}; // generation of the job in the upper half, its next piece in the lower
   std::atomic<uint32_t> done_{0};
   std::atomic<int> sleepers_{0};
   std::atomic<bool> stop_{false};
};

// The pools of the process. A context borrows one while a transfer of its own runs and gives it back, so that any number of Sessions
// called one after the other share one set of helpers; a pool is added only for a transfer that finds the others in use. The first may
// have all the threads that were asked for, the later ones what is left of the cores, but three helpers at least. All are ended with
// the last context.
class HostPools {
public:
   static HostPools &get()
   {
      static HostPools *p = new HostPools; // never destroyed: a context may outlive the statics
      return *p;
   }
   // Threads of a transfer: all cores but two, fourteen at most (SOFIE_CUDA_COPY_THREADS overrides it, up to the cores and sixteen).
   // Measured on a 16-core host, int8 CNN on 16384 images (268 MB of floats quantised while they are staged): 4.06 ms per call with
   // eight threads, 3.83 with ten, 3.0 with twelve, 2.65 with fourteen.
   static int wanted_threads()
   {
      const int cores = (int)std::thread::hardware_concurrency();
      int threads = cores - 2 < 14 ? cores - 2 : 14;
      if (const char *e = std::getenv("SOFIE_CUDA_COPY_THREADS")) threads = std::atoi(e);
      if (cores > 0 && threads > cores) threads = cores;
      return threads < 1 ? 1 : (threads > 16 ? 16 : threads);
   }
   // nullptr: no memory
   HostPool *borrow()
   {
      try {
         std::lock_guard<std::mutex> lock(mu_);
         size_t best = idle_.size();
         for (size_t i = 0; i < idle_.size(); i++)
            if (best == idle_.size() || idle_[i]->threads() > idle_[best]->threads()) best = i;
         if (best < idle_.size()) {
            HostPool *p = idle_[best];
            idle_.erase(idle_.begin() + (long)best);
            return p;
         }
         int helpers = wanted_threads() - 1;
         if (helpers_ > 0) {
            const int left = (int)std::thread::hardware_concurrency() - 2 - helpers_, later = left < 3 ? 3 : left;
            if (helpers > later) helpers = later;
         }
         idle_.reserve(idle_.size() + lent_ + 1); // give_back() does not allocate
         HostPool *p = new HostPool(helpers);
         helpers_ += (int)p->threads() - 1;
         lent_++;
         return p;
      } catch (...) {
         return nullptr;
      }
   }
   void give_back(HostPool *p)
   {
      std::lock_guard<std::mutex> lock(mu_);
      idle_.push_back(p);
      if (users_ == 0) end_idle();
   }
   void user_begins()
   {
      std::lock_guard<std::mutex> lock(mu_);
      users_++;
   }
   void user_ends()
   {
      std::lock_guard<std::mutex> lock(mu_);
      if (--users_ == 0) end_idle();
   }

private:
   void end_idle()
   {
      for (HostPool *p : idle_) {
         helpers_ -= (int)p->threads() - 1;
         lent_--;
         delete p;
      }
      idle_.clear();
   }
   std::mutex mu_;
   std::vector<HostPool *> idle_;
   size_t lent_ = 0; // pools there are, lent or idle
   int helpers_ = 0; // their threads
   int users_ = 0;   // contexts there are
};

} // namespace sofie
