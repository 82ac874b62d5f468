// The forward pass through host buffers: copy in, kernel and results out, in chunks that overlap.
//
// A request is cut into chunks of images; four slots (a device buffer, a stream and a result buffer each) take them in
// turn, so that the copies of the next chunks run under a chunk's kernel.  The last chunk is the short one: its kernel and results come behind
// everything else.  Pinned images are copied from where they lie.
// Pageable images go through a pinned ring that several cores fill (copy_pool.h): 10,000 uint8 images 620-750 -> 250 us on a B200
// (the driver's own staging fills its buffer with one core, 12 GB/s; the bus carries 55 GB/s).  Results for pageable
// buffers go through pinned memory too, one copy per chunk.  (Written there by the kernel itself, over the bus, they cost
// 80 us per 2,500 images.)
#include <cstring>
#include <memory>
#include <new>

#include "copy_pool.h"
#include "net.cuh"

namespace cnn {

int forward_kernel_for(const cnn_net* net, long n_total, bool u8);
int forward_device(cnn_net* net, int path, const float* d_images, long n, float* d_out, int* d_argmax,
                   cudaStream_t stream);
int forward_device_u8(cnn_net* net, int path, const unsigned char* d_pixels, long n, float* d_out, int* d_argmax,
                      cudaStream_t stream);

constexpr int kHpSlots = 4;
constexpr long kHpMaxChunk = 8192, kHpMinChunk = 512;       // images per chunk
static_assert(kHpSlots * (sizeof(float) * (kOut + 1) * kHpMaxChunk + 256) + sizeof(int) * kHpSlots <= PinnedBlock::kPage, "results fit a lease");
constexpr size_t kHpMinQuarter = 4608 * 1024;               // pinned images: below, two halves
constexpr size_t kHpMinStaged = 128 * 1024;                 // below, the driver's own staging is as fast

struct HostPipeline {
  struct Slot {
    cudaStream_t stream = nullptr;
    unsigned char* d_img = nullptr;            // chunk images on the device
    float* d_res = nullptr;                    // results on the device: 10 sigmoids per image, then the argmax
    float* h_res = nullptr;                    // the same in pinned memory, for pageable result buffers
    long first = 0, count = 0;                 // the chunk whose results wait in h_res (count 0: none)
  } slot[kHpSlots];
  unsigned char* d_block = nullptr;            // all slots' images and results
  size_t d_bytes = 0;
  PinnedHeap::Lease h_block;                   // all slots' results (for pageable ones), and behind them:
  int* h_status = nullptr;                     // the net's status word after each slot's last kernel
  cudaEvent_t piece[CopyPool::kSlots] = {};    // a ring slot's copy to the device is done
  cudaEvent_t order_event = nullptr;           // ties the slots' streams behind the legacy stream
  std::unique_ptr<CopyPool::Ref> pool;

  ~HostPipeline() {
    for (Slot& s : slot)
      if (s.stream) cudaStreamDestroy(s.stream);
    cudaFree(d_block);
    for (cudaEvent_t e : piece)
      if (e) cudaEventDestroy(e);
    if (order_event) cudaEventDestroy(order_event);
  }

  // One allocation each for all slots, which only grows: a cudaMalloc costs 0.4 ms whatever its size, and of two requests the larger one may have
  // the shorter or the fewer slots (10,000 images two of 7,952, 11,000 three of 4,476).
  int reserve(int slots, long chunk, size_t image_bytes, bool pinned_results, bool staged) {
    if (!order_event) {
      for (Slot& s : slot)
        if (!s.stream) CNN_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
      CNN_CUDA(cudaEventCreateWithFlags(&order_event, cudaEventDisableTiming));
    }
    const size_t img = ((size_t)chunk * image_bytes + 255) & ~(size_t)255, res = (sizeof(float) * (kOut + 1) * (size_t)chunk + 255) & ~(size_t)255;
    if (d_bytes < (img + res) * slots) {
      cudaFree(d_block);
      d_block = nullptr;
      d_bytes = 0;
      CNN_CUDA(cudaMalloc(&d_block, (img + res) * slots));
      d_bytes = (img + res) * slots;
    }
    const size_t pinned = (pinned_results ? res * slots : 0) + sizeof(int) * kHpSlots;
    if (h_block.bytes() < pinned && !h_block.take(pinned)) {
      set_error("cnn_forward_batched_host: no pinned memory");
      return CNN_ERR_CUDA;
    }
    for (int i = 0; i < slots; ++i) {
      slot[i].d_img = d_block + (img + res) * i;
      slot[i].d_res = reinterpret_cast<float*>(slot[i].d_img + img);
      slot[i].h_res = pinned_results ? reinterpret_cast<float*>(h_block.get() + res * i) : nullptr;
    }
    h_status = reinterpret_cast<int*>(h_block.get() + (pinned_results ? res * slots : 0));
    if (staged && !pool) {
      for (cudaEvent_t& e : piece)
        if (!e) CNN_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      pool.reset(new (std::nothrow) CopyPool::Ref());
    }
    return CNN_OK;
  }
};

void destroy_host_pipeline(HostPipeline* p) { delete p; }

static bool is_pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// One request on its way through the pipeline.
struct HostRequest {
  cnn_net* net;
  HostPipeline& hp;
  const unsigned char* images;
  bool u8;
  long n;
  float* out;
  int* argmax;
  size_t image_bytes;
  bool pinned_results, staged;
  // Chunks: equal ones, and a last one.
  long chunk, rest;                              // images of an equal chunk, and of all of them
  int slots, path;
  std::unique_ptr<size_t[]> at = nullptr;        // where the pieces of a staged request begin, and where the last one ends
  std::unique_ptr<long[]> chunk_end = nullptr;   // per piece: the number of images up to the chunk that it completes, else 0

  long count_at(long first) const {
    if (first >= rest) return n - rest;
    return rest - first < chunk ? rest - first : chunk;
  }

  // Pageable results of the chunk that was in this slot.
  int hand_over(HostPipeline::Slot& s) {
    if (s.count == 0) return CNN_OK;
    CNN_CUDA(cudaStreamSynchronize(s.stream));
    if (out) std::memcpy(out + s.first * kOut, s.h_res, sizeof(float) * kOut * (size_t)s.count);
    if (argmax) std::memcpy(argmax + s.first, s.h_res + s.count * kOut, sizeof(int) * (size_t)s.count);
    s.count = 0;
    return CNN_OK;
  }
  // Kernel and results of a chunk whose images are on their way into slot si.
  int compute(int si, long first, long count) {
    HostPipeline::Slot& s = hp.slot[si];
    float* o = out ? s.d_res : nullptr;
    int* a = argmax ? reinterpret_cast<int*>(s.d_res + count * kOut) : nullptr;
    const int rc = u8 ? forward_device_u8(net, path, s.d_img, count, o, a, s.stream)
                      : forward_device(net, path, reinterpret_cast<const float*>(s.d_img), count, o, a, s.stream);
    if (rc != CNN_OK) return rc;
    if (pinned_results) {
      const long lo = out ? 0 : count * kOut, hi = argmax ? count * (kOut + 1) : count * kOut;      // what was asked for
      if (lo < hi) CNN_CUDA(cudaMemcpyAsync(s.h_res + lo, s.d_res + lo, sizeof(float) * (size_t)(hi - lo), cudaMemcpyDeviceToHost, s.stream));
      s.first = first;
      s.count = count;
    } else {
      if (out) CNN_CUDA(cudaMemcpyAsync(out + first * kOut, o, sizeof(float) * kOut * (size_t)count, cudaMemcpyDeviceToHost, s.stream));
      if (argmax) CNN_CUDA(cudaMemcpyAsync(argmax + first, a, sizeof(int) * (size_t)count, cudaMemcpyDeviceToHost, s.stream));
    }
    const long equal = (rest + chunk - 1) / chunk;
    if ((first < rest ? first / chunk : equal) + slots >= equal + 1)      // this slot's last chunk
      CNN_CUDA(cudaMemcpyAsync(&hp.h_status[si], net->d_status, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    return CNN_OK;
  }
  int run_direct() {
    int si = 0;
    for (long first = 0; first < n; first += count_at(first), si = (si + 1) % slots) {
      const long count = count_at(first);
      int rc = hand_over(hp.slot[si]);
      if (rc != CNN_OK) return rc;
      CNN_CUDA(cudaMemcpyAsync(hp.slot[si].d_img, images + (size_t)first * image_bytes, (size_t)count * image_bytes,
                               cudaMemcpyHostToDevice, hp.slot[si].stream));
      if ((rc = compute(si, first, count)) != CNN_OK) return rc;
    }
    return CNN_OK;
  }
  // Pieces of the staged copy: as many as a chunk needs, of equal length.  (A short first piece and short pieces in the last chunk, so that less of
  // the filling and of the bus comes before and behind everything else: 1-8 % slower below 10 MB, every copy costs some microseconds, and 0-2 % faster above.)
  bool cut(long& pieces) {
    const long most = (long)((size_t)n * image_bytes / CopyPool::kPiece) + n / chunk + 3;
    at.reset(new (std::nothrow) size_t[most + 1]);
    chunk_end.reset(new (std::nothrow) long[most]);
    if (!at || !chunk_end) return false;
    pieces = 0;
    at[0] = 0;
    for (long first = 0, end; first < n; first = end) {
      end = first + count_at(first);
      const size_t end_byte = (size_t)end * image_bytes, bytes = end_byte - (size_t)first * image_bytes;
      const size_t parts = (bytes + CopyPool::kPiece - 1) / CopyPool::kPiece, length = ((bytes + parts - 1) / parts + 63) & ~(size_t)63;
      while (at[pieces] < end_byte) {
        at[pieces + 1] = end_byte - at[pieces] > length ? at[pieces] + length : end_byte;
        chunk_end[pieces] = at[pieces + 1] == end_byte ? end : 0;
        ++pieces;
      }
    }
    return true;
  }
  int run_pieces(CopyPool::Job& job, int helpers) {
    long first = 0;                              // the piece's chunk: its first image and its slot
    int si = 0;
    bool begins = true;
    for (long p = 0; p < job.pieces; ++p) {
      HostPipeline::Slot& s = hp.slot[si];
      CopyPool::copy_share(job, p, 0, helpers + 1);
      while (job.done[p % CopyPool::kSlots].load(std::memory_order_acquire) != helpers) CopyPool::pause();
      job.done[p % CopyPool::kSlots].store(0, std::memory_order_relaxed);
      int rc;
      if (begins && (rc = hand_over(s)) != CNN_OK) return rc;
      CNN_CUDA(cudaMemcpyAsync(s.d_img + (job.at[p] - (size_t)first * image_bytes), job.slot(p), job.bytes(p), cudaMemcpyHostToDevice, s.stream));
      CNN_CUDA(cudaEventRecord(hp.piece[p % CopyPool::kSlots], s.stream));
      begins = chunk_end[p] != 0;
      if (begins) {
        if ((rc = compute(si, first, chunk_end[p] - first)) != CNN_OK) return rc;
        first = chunk_end[p];
        si = (si + 1) % slots;
      }
      // Give back the slot of the piece half a ring behind: its copy is done or nearly so.
      const long next = job.released.load(std::memory_order_relaxed);
      if (next < job.pieces && next - CopyPool::kSlots <= p - CopyPool::kSlots / 2) {
        CNN_CUDA(cudaEventSynchronize(hp.piece[next % CopyPool::kSlots]));
        job.released.store(next + 1, std::memory_order_release);
      }
    }
    return CNN_OK;
  }
  int run_staged() {
    CopyPool::Job job;
    if (!cut(job.pieces)) return run_direct();
    job.src = images;
    job.at = at.get();
    for (int i = 0; i < CopyPool::kSlots; ++i) job.done[i].store(0, std::memory_order_relaxed);
    job.released.store(job.pieces < CopyPool::kSlots ? job.pieces : CopyPool::kSlots, std::memory_order_release);
    const int helpers = hp.pool ? CopyPool::get().begin(&job) : 0;
    if (helpers == 0) return run_direct();
    const int rc = run_pieces(job, helpers);
    if (rc != CNN_OK) job.cancelled.store(true, std::memory_order_release);
    // the last pieces have left the ring before the next job may write into it
    for (int i = 0; i < CopyPool::kSlots && i < job.pieces; ++i) cudaEventSynchronize(hp.piece[i]);
    CopyPool::get().end();
    return rc;
  }
  int run(long largest) {
    int rc = hp.reserve(slots, largest, image_bytes, pinned_results, staged);
    if (rc != CNN_OK) return rc;
    // The streams are first put behind everything queued so far on the legacy default stream (a parameter update, a
    // training call), so that a forward issued right after such work sees its result; work on a caller's own non-blocking
    // stream is NOT waited for (the caller synchronises that stream first).
    CNN_CUDA(cudaEventRecord(hp.order_event, cudaStreamLegacy));
    for (int s = 0; s < kHpSlots; ++s) {
      hp.slot[s].count = 0;
      hp.h_status[s] = 0;
      if (s < slots) CNN_CUDA(cudaStreamWaitEvent(hp.slot[s].stream, hp.order_event, 0));
    }
    if ((rc = staged ? run_staged() : run_direct()) != CNN_OK) return rc;
    for (int s = 0; s < slots; ++s) {
      CNN_CUDA(cudaStreamSynchronize(hp.slot[s].stream));
      if ((rc = hand_over(hp.slot[s])) != CNN_OK) return rc;
    }
    return CNN_OK;
  }
};

static int forward_host_impl(cnn_net* net, const void* h_images, bool u8, long n, float* h_out, int* h_argmax) {
  CNN_REQUIRE(net != nullptr, "cnn_forward_batched_host: NULL net");
  CNN_REQUIRE(n >= 0, "cnn_forward_batched_host: negative image count");
  if (n == 0) return CNN_OK;
  CNN_REQUIRE(h_images != nullptr, "cnn_forward_batched_host: NULL images");
  if (!net->host) net->host = new (std::nothrow) HostPipeline();
  CNN_REQUIRE(net->host != nullptr, "cnn_forward_batched_host: out of host memory");
  HostPipeline& hp = *net->host;
  const size_t image_bytes = u8 ? (size_t)kImg : sizeof(float) * kImg;
  const bool pageable = is_pageable(h_images);
  // Behind the last copy there is the last chunk's kernel, the way of its results back and, for pageable result buffers, a copy of them: a
  // quarter of the request, at least 512 images and at most 2,048 (halves: 10,000 uint8 images 256 instead of 249 us, 6,000 181 instead of 172; quarters all over: more hand-overs, 280).
  // Pinned images, without the filling of the ring, leave a small request nothing to gain: halves below 4.5 MB (quarter, half: 5,000 uint8 images
  // 141, 131 us, 1,300 fp32 125, 119; 6,000 uint8 144, 151, 1,500 fp32 131, 136).
  const bool quarter = pageable || (size_t)n * image_bytes >= kHpMinQuarter;
  long last = quarter ? n / 4 : n / 2;
  if (quarter) last = last < kHpMinChunk ? kHpMinChunk : (last > kHpMaxChunk / 4 ? kHpMaxChunk / 4 : last);
  if (n <= 2 * kHpMinChunk) last = n;
  const long rest = n - last, parts = (rest + kHpMaxChunk - 1) / kHpMaxChunk;
  const long chunk = parts > 0 ? (rest + parts - 1) / parts : last;
  const int slots = parts + 1 < kHpSlots ? (int)parts + 1 : kHpSlots;
  HostRequest req{net, hp, static_cast<const unsigned char*>(h_images), u8, n, h_out, h_argmax, image_bytes,
                  (h_out && is_pageable(h_out)) || (h_argmax && is_pageable(h_argmax)),
                  pageable && (size_t)n * image_bytes >= kHpMinStaged, chunk, rest, slots,
                  forward_kernel_for(net, n, u8)};     // one kernel for the whole request, whatever the chunking
  const int rc = req.run(chunk > last ? chunk : last);
  if (rc != CNN_OK) {
    // nothing of this request may still read the caller's buffers or write into them when the call returns
    for (auto& s : hp.slot)
      if (s.stream) cudaStreamSynchronize(s.stream);
    return rc;
  }
  if (hp.h_status[0] | hp.h_status[1] | hp.h_status[2] | hp.h_status[3]) {
    set_error("cnn_forward_batched_host: a bounded device-side wait ran out");
    int zero = 0;
    cudaMemcpy(net->d_status, &zero, sizeof(int), cudaMemcpyHostToDevice);
    return CNN_ERR_TIMEOUT;
  }
  return CNN_OK;
}

}  // namespace cnn

extern "C" int cnn_forward_batched_host(cnn_net* net, const float* h_images, long n, float* h_out, int* h_argmax) {
  return cnn::forward_host_impl(net, h_images, false, n, h_out, h_argmax);
}

extern "C" int cnn_forward_batched_u8_host(cnn_net* net, const unsigned char* h_pixels, long n, float* h_out,
                                           int* h_argmax) {
  return cnn::forward_host_impl(net, h_pixels, true, n, h_out, h_argmax);
}
