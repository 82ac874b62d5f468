// A few host threads that help to copy pageable memory into a pinned ring.
//
// A transfer from pageable memory goes through a pinned buffer on its way to the device, and one core fills such a buffer
// at about 12 GB/s -- a fifth of what the bus carries.  All threads of the pool copy a share of every piece, so that the
// first piece is on its way after a few microseconds and the pieces come in order.
//
// One pool per process, threads and ring, shared by all nets that have used the host pipeline: the first of them sets it up
// (pinning the ring is the dear part), the last one to go takes it down (CopyPool::Ref).  A job has the pool to itself;
// a caller that finds it busy leaves its copy to the driver.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace cnn {

class CopyPool {
 public:
  static constexpr int kMaxThreads = 6;        // helpers and the caller: six cores fill the ring as fast as the bus empties it
  static constexpr int kSlots = 4;             // ring: pieces of kPiece bytes at most (a copy to the device costs 4 us before
  static constexpr size_t kPiece = 2 * 1024 * 1024;      // its first byte: pieces of 256 KB run at 30 GB/s)

  // The source is cut into chunks, each chunk into pieces; piece p goes to ring slot p % kSlots.
  struct Job {
    const unsigned char* src = nullptr;
    unsigned char* ring = nullptr;
    size_t total = 0, chunk_bytes = 0, piece_bytes = 0;
    long pieces_per_chunk = 1, pieces = 0;
    std::atomic<long> released{0};             // pieces whose ring slot may be written
    std::atomic<int> done[kSlots];          // per ring slot: helpers that have written their share
    std::atomic<bool> cancelled{false};

    size_t offset(long p) const { return (size_t)(p / pieces_per_chunk) * chunk_bytes + (size_t)(p % pieces_per_chunk) * piece_bytes; }
    size_t bytes(long p) const {
      const size_t in_chunk = (size_t)(p % pieces_per_chunk) * piece_bytes, at = offset(p);
      size_t b = chunk_bytes - in_chunk < piece_bytes ? chunk_bytes - in_chunk : piece_bytes;
      return total - at < b ? total - at : b;
    }
    unsigned char* slot(long p) const { return ring + (size_t)(p % kSlots) * kPiece; }
  };

  class Ref {                                  // held by a net: keeps the threads alive
   public:
    Ref() { CopyPool::get().acquire(); }
    ~Ref() { CopyPool::get().release(); }
    Ref(const Ref&) = delete;
    Ref& operator=(const Ref&) = delete;
  };

  static CopyPool& get() {
    static CopyPool* pool = new CopyPool();    // never destroyed: its threads are gone by then or end with the process
    return *pool;
  }

  // Takes the pool for `job` and gives it the ring; the number of helpers that will work on it (0: busy, or there are none).
  int begin(Job* job) {
    if (!owner_.try_lock()) return 0;
    if (helpers_ == 0 || !ring_) {
      owner_.unlock();
      return 0;
    }
    job->ring = ring_;
    {
      std::lock_guard<std::mutex> l(m_);
      job_ = job;
      working_.store(helpers_, std::memory_order_relaxed);
      turn_.fetch_add(1, std::memory_order_release);
    }
    wake_.notify_all();
    return helpers_;
  }
  // Waits until no helper touches the job any more and gives the pool back.
  void end() {
    while (working_.load(std::memory_order_acquire) != 0) pause();
    owner_.unlock();
  }

  // Share `who` of `parts` of piece p (whole cache lines).
  static void copy_share(const Job& j, long p, int who, int parts) {
    const size_t bytes = j.bytes(p), share = ((bytes + parts - 1) / parts + 63) & ~(size_t)63, lo = share * who;
    if (lo < bytes) copy_past_caches(j.slot(p) + lo, j.src + j.offset(p) + lo, bytes - lo < share ? bytes - lo : share);
  }
  // dst is 64-byte aligned.  The copy is written around the caches: the device reads it next, and lines that lie modified
  // in some core's cache come over the bus at a fraction of its rate (10,000 uint8 images: 383 against 625 us with the same pieces).
  static void copy_past_caches(unsigned char* dst, const unsigned char* src, size_t bytes) {
    size_t i = 0;
#if defined(__SSE2__)
    for (; i + 64 <= bytes; i += 64) {
      const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 16));
      const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 48));
      _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i), a);
      _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 16), b);
      _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 32), c);
      _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 48), d);
    }
    _mm_sfence();
#endif
    if (i < bytes) std::memcpy(dst + i, src + i, bytes - i);
  }
  static void pause() {
#if defined(__SSE2__)
    _mm_pause();
#endif
  }

 private:
  void acquire() {
    std::lock_guard<std::mutex> o(owner_);
    if (users_++ > 0) return;
    const int cores = (int)std::thread::hardware_concurrency();
    const int want = cores > 2 * kMaxThreads ? kMaxThreads - 1 : cores / 2 - 1;
    stop_.store(false);
    const long now = turn_.load();
    try {
      for (int i = 0; i < want; ++i) threads_.emplace_back([this, i, now] { work(i, now); });
    } catch (...) {                            // fewer helpers, or none
    }
    helpers_ = (int)threads_.size();
    if (helpers_ > 0) make_ring();
  }
  // Huge pages where the system has them: pinning 8 MB then takes 0.5 ms (and touching it 1.1 ms) instead of 5 ms.
  void make_ring() {
    void* p = std::aligned_alloc(kPiece, kPiece * kSlots);
    if (!p) return;
#if defined(MADV_HUGEPAGE)
    madvise(p, kPiece * kSlots, MADV_HUGEPAGE);
#endif
    std::memset(p, 0, kPiece * kSlots);
    if (cudaHostRegister(p, kPiece * kSlots, cudaHostRegisterPortable) == cudaSuccess) {
      ring_ = static_cast<unsigned char*>(p);
    } else {
      cudaGetLastError();                      // the driver's own staging still works
      std::free(p);
    }
  }
  void release() {
    std::lock_guard<std::mutex> o(owner_);
    if (--users_ > 0) return;
    {
      std::lock_guard<std::mutex> l(m_);
      stop_.store(true);
      turn_.fetch_add(1, std::memory_order_release);
    }
    wake_.notify_all();
    for (std::thread& t : threads_) t.join();
    threads_.clear();
    helpers_ = 0;
    if (ring_) {
      cudaHostUnregister(ring_);
      std::free(ring_);
      ring_ = nullptr;
    }
  }
  void work(int who, long seen) {
    for (;;) {
      // a short spin (some 50 us) catches the next call of a loop of calls, then the thread sleeps
      for (int spin = 0; spin < 2000 && turn_.load(std::memory_order_acquire) == seen; ++spin) pause();
      if (turn_.load(std::memory_order_acquire) == seen) {
        std::unique_lock<std::mutex> l(m_);
        wake_.wait(l, [&] { return turn_.load(std::memory_order_acquire) != seen; });
      }
      seen = turn_.load(std::memory_order_acquire);
      if (stop_.load()) return;
      Job& j = *job_;
      for (long p = 0; p < j.pieces; ++p) {
        while (p >= j.released.load(std::memory_order_acquire) && !j.cancelled.load(std::memory_order_acquire)) pause();
        if (j.cancelled.load(std::memory_order_acquire)) break;
        copy_share(j, p, who + 1, helpers_ + 1);
        j.done[p % kSlots].fetch_add(1, std::memory_order_release);
      }
      working_.fetch_sub(1, std::memory_order_release);
    }
  }

  std::mutex owner_, m_;
  std::condition_variable wake_;
  std::vector<std::thread> threads_;
  unsigned char* ring_ = nullptr;              // pinned
  Job* job_ = nullptr;                         // written before the turn advances, read after
  std::atomic<long> turn_{0};
  std::atomic<int> working_{0};
  std::atomic<bool> stop_{false};
  int helpers_ = 0, users_ = 0;
};

}  // namespace cnn
