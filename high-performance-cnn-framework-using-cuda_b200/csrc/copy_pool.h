// A few host threads that help to copy pageable memory into a pinned ring.
//
// A transfer from pageable memory goes through a pinned buffer on its way to the device, and one core fills such a buffer
// at about 12 GB/s -- a fifth of what the bus carries.  All threads of the pool copy a share of every piece, so that the
// first piece is on its way after a few microseconds and the pieces come in order.
//
// One pool per process, threads and ring, shared by all nets that have used the host pipeline: the first of them sets it up
// (1.1 ms; with the ring touched by one thread, and with cudaMallocHost for the results, the first call of a net took 3 to 5.4 ms instead of
// 1.7), the last one to go takes it down (CopyPool::Ref).  A job has the pool to itself;
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
#include <new>
#include <thread>
#include <vector>

namespace cnn {

// Pinned host memory in whole huge pages (where the system has them), touched by several threads: 8 MB take 1 ms and 2 MB 0.3 ms.
// (cudaMallocHost: 3.3 ms for 8 MB, and 1 to 2.6 ms for the first few bytes of a program, as it pins 2 MB at a time in small pages.)
class PinnedBlock {
 public:
  static constexpr size_t kPage = 2 * 1024 * 1024;

  PinnedBlock() = default;
  PinnedBlock(const PinnedBlock&) = delete;
  PinnedBlock& operator=(const PinnedBlock&) = delete;
  ~PinnedBlock() { release(); }

  unsigned char* get() const { return p_; }
  bool allocate(size_t bytes) {                // (of an empty block)
    const size_t pages = (bytes + kPage - 1) / kPage;
    unsigned char* p = static_cast<unsigned char*>(std::aligned_alloc(kPage, kPage * pages));
    if (!p) return false;
#if defined(MADV_HUGEPAGE)
    madvise(p, kPage * pages, MADV_HUGEPAGE);
#endif
    auto touch = [p](size_t page) {
      for (size_t i = 0; i < kPage; i += 4096) const_cast<volatile unsigned char*>(p)[page * kPage + i] = 0;
    };
    std::vector<std::thread> others;
    try {
      for (size_t i = 1; i < pages; ++i) others.emplace_back(touch, i);
    } catch (...) {                            // fewer threads: the rest is done here
    }
    touch(0);
    for (size_t i = others.size() + 1; i < pages; ++i) touch(i);
    for (std::thread& t : others) t.join();
    if (cudaHostRegister(p, kPage * pages, cudaHostRegisterPortable) != cudaSuccess) {
      cudaGetLastError();
      std::free(p);
      return false;
    }
    p_ = p;
    return true;
  }
  void release() {
    if (!p_) return;
    cudaHostUnregister(p_);
    std::free(p_);
    p_ = nullptr;
  }

 private:
  unsigned char* p_ = nullptr;
};

// Small pieces of such memory, for all nets of the process: cells of a quarter page, first come first served; a page is given back
// when its last cell is.  (A page for each net took 0.3 ms of a net's first call, also where other nets are alive.)
class PinnedHeap {
 public:
  static constexpr int kCells = 4;
  static constexpr size_t kCell = PinnedBlock::kPage / kCells;

  // A lease of some cells in a row; empty where there is no memory.
  class Lease {
   public:
    Lease() = default;
    Lease(const Lease&) = delete;
    Lease& operator=(const Lease&) = delete;
    ~Lease() { PinnedHeap::get().release(*this); }
    unsigned char* get() const { return at_; }
    size_t bytes() const { return kCell * cells_; }
    bool take(size_t bytes) { return PinnedHeap::get().take(*this, bytes); }       // gives back what it had; a page at most

   private:
    friend class PinnedHeap;
    unsigned char* at_ = nullptr;
    int cells_ = 0;
  };

  static PinnedHeap& get() {
    static PinnedHeap* heap = new PinnedHeap();
    return *heap;
  }

 private:
  struct Page {
    PinnedBlock block;
    unsigned used = 0;                         // a bit per cell
    Page* next = nullptr;
  };
  bool take(Lease& l, size_t bytes) {
    release(l);
    const int cells = (int)((bytes + kCell - 1) / kCell);
    if (cells < 1 || cells > kCells) return false;
    std::lock_guard<std::mutex> g(m_);
    const unsigned want = (1u << cells) - 1;
    for (Page* p = pages_; p; p = p->next)
      for (int i = 0; i + cells <= kCells; ++i)
        if (!(p->used & (want << i))) return give(l, *p, i, cells);
    Page* p = new (std::nothrow) Page();
    if (!p || !p->block.allocate(PinnedBlock::kPage)) {
      delete p;
      return false;
    }
    p->next = pages_;
    pages_ = p;
    return give(l, *p, 0, cells);
  }
  static bool give(Lease& l, Page& p, int first, int cells) {
    p.used |= ((1u << cells) - 1) << first;
    l.at_ = p.block.get() + kCell * first;
    l.cells_ = cells;
    return true;
  }
  void release(Lease& l) {
    if (!l.at_) return;
    std::lock_guard<std::mutex> g(m_);
    for (Page** p = &pages_; *p; p = &(*p)->next) {
      const size_t off = (size_t)(l.at_ - (*p)->block.get());      // (of another page: out of range, either way)
      if (off >= PinnedBlock::kPage) continue;
      (*p)->used &= ~(((1u << l.cells_) - 1) << (off / kCell));
      if ((*p)->used == 0) {
        Page* gone = *p;
        *p = gone->next;
        delete gone;
      }
      break;
    }
    l.at_ = nullptr;
    l.cells_ = 0;
  }

  std::mutex m_;
  Page* pages_ = nullptr;
};

class CopyPool {
 public:
  static constexpr int kMaxThreads = 6;        // helpers and the caller: six cores fill the ring as fast as the bus empties it
  static constexpr int kSlots = 4;             // ring: pieces of kPiece bytes at most (a copy to the device costs 4 us before
  static constexpr size_t kPiece = 2 * 1024 * 1024;      // its first byte: pieces of 256 KB run at 30 GB/s)

  // The source is cut into pieces; piece p is the bytes from at[p] to at[p + 1] and goes to ring slot p % kSlots.
  struct Job {
    const unsigned char* src = nullptr;
    unsigned char* ring = nullptr;
    const size_t* at = nullptr;
    long pieces = 0;
    std::atomic<long> released{0};             // pieces whose ring slot may be written
    std::atomic<int> done[kSlots];          // per ring slot: helpers that have written their share
    std::atomic<bool> cancelled{false};

    size_t bytes(long p) const { return at[p + 1] - at[p]; }
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
    if (helpers_ == 0 || !ring_.get()) {
      owner_.unlock();
      return 0;
    }
    job->ring = ring_.get();
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
    if (lo < bytes) copy_past_caches(j.slot(p) + lo, j.src + j.at[p] + lo, bytes - lo < share ? bytes - lo : share);
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
    if (helpers_ > 0) ring_.allocate(kPiece * kSlots);       // (without it the driver's own staging still works)
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
    ring_.release();
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
  PinnedBlock ring_;
  Job* job_ = nullptr;                         // written before the turn advances, read after
  std::atomic<long> turn_{0};
  std::atomic<int> working_{0};
  std::atomic<bool> stop_{false};
  int helpers_ = 0, users_ = 0;
};

}  // namespace cnn
