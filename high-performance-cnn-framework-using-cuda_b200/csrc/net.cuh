// The fused-network handle shared by the forward, training and host-pipeline translation units.
#pragma once

#include "cnn_common.cuh"

namespace cnn {
struct HostPipeline;
}

struct cnn_net {
  int device = 0;
  unsigned seed = 0;               // what cnn_net_create drew the initial parameters from (kept for checkpoints)
  int ps_kernel = 1;               // per-sample SGD: 1 = six-CTA cluster kernel (default), 0 = single persistent block
  int forward_path = -1;           // batched forward: 0 = exact fp32 SIMT kernel, 1 = tensor cores in two or three fp16 passes
                                   // (fp32-level accuracy), 2 = tensor cores, one fp16 pass + tanh sigmoid,
                                   // -1 (default) = 1 for batches of kTcMinBatch images or more, else 0
  int grad_path = -1;              // gradient of a batch: 0 = CUDA cores, 1 = tensor cores, -1 (default) = by batch size
  float* d_params = nullptr;       // kNParamsPadded floats
  int* d_status = nullptr;         // device status word: 0 ok, non-zero = a bounded wait ran out; behind it what GradLeft describes
  int fast_sigmoid = 1;            // sigmoid of the fused kernels: 0 = reference expression, 1 = short form (default)

  // Training scratch, one allocation on first use: the reduced vector, and behind it per-block partial gradients.
  float* d_partials = nullptr;     // a row of kRowStride floats per SM
  float* d_grad = nullptr;         // kNParamsPadded floats + 8 floats of statistics
  cnn::HostPipeline* host = nullptr;   // host_pipeline.cu (created on first use)
};

namespace cnn {

// ---- mbarrier / bulk-copy primitives (sm_90+ PTX, used in their non-multicast form only) ----
__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// One arrival on an mbarrier of this CTA (release at CTA scope).
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 1-D bulk copy global -> this CTA's shared memory, completion signalled on an mbarrier.
// Both addresses must be 16-byte aligned and bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes,
                                         unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// Programmatic dependent launch: a kernel launched with launch_pdl() may start while its predecessor in the
// stream is still running, once every block of the predecessor has called pdl_launch_dependents() (or
// exited); whatever it reads of the predecessor's results must come after pdl_wait(), which returns when
// the predecessor has completed and its writes are visible.  Both are no-ops in an ordinary launch.
// Such a kernel reads global memory by ordinary loads only: neither __ldg nor `const T* __restrict__` parameters, which allow the
// read-only path.  That path is for data that nobody writes during the kernel's lifetime (which begins before the wait), and its
// loads may be moved in front of the wait.  Pointers that a kernel writes through may stay __restrict__.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Per-thread asynchronous copies global -> shared (LDGSTS), 16 bytes (L2 only) or 4 bytes, and their groups.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after about two seconds of SM clocks, records it in *status and lets the
// caller carry on (with whatever the buffer holds) so that control flow stays uniform and the
// kernel always terminates.  Returns false once a wait has run out.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity,
                                                  int* status, bool& gave_up) {
  if (gave_up) return false;
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > 4000000000LL) {
      gave_up = true;
      if (status) atomicExch(status, 1);
      return false;
    }
  }
  return true;
}

// Partial-gradient rows of the minibatch kernels: arena-ordered gradient [0, 2343), zero padding,
// and at kRowErr the sum over the row's images of ||delta_f||_2.
constexpr int kRowStride = kNParamsPadded + 8;
constexpr int kRowErr = kNParams + 1;  // 2344

// Shares of a batch: the first `more` blocks have one image more than the others.  (Fewer blocks with equal shares would leave SMs idle, where k_grad_left's
// first blocks would start before anything is left.)
struct GradShares {
  int blocks, each, more;
  __host__ __device__ long first(int b) const { return (long)b * each + (b < more ? b : more); }
  __host__ __device__ int size(int b) const { return each + (b < more ? 1 : 0); }
};

// What of a block's share of a batch the tensor-core gradient kernel (grad_tc.cu) leaves to the CUDA cores: the images from `from` on, and before
// them some tiles of kGradTile images.  `next` is a queue beside it: block numbers + 1, in the order in which blocks that leave something finish; 0 = no more yet.
constexpr int kGradTile = 5, kGradSkips = 28;
struct GradLeft {
  int from, written, skips, tile[kGradSkips], next;      // written: the block's row holds the gradient of what is not left
};
// They lie behind the net's status word, one per SM, and before them the number of entries in the queue; all zero between two calls.
inline int* grad_queued(cnn_net* net) { return net->d_status + 1; }
inline GradLeft* grad_left(cnn_net* net) { return reinterpret_cast<GradLeft*>(net->d_status) + 1; }

// Column `col` of rows g, g + GROUPS, g + 2 GROUPS, ... added in that order; five loads at a time are under way (with one
// row per SM and 32 groups that is all of them).
template <int GROUPS>
__device__ __forceinline__ float sum_rows(const float* rows, int n_rows, int col, int g) {
  float acc = 0.f;
  for (int r0 = g; r0 < n_rows; r0 += 5 * GROUPS) {
    float v[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int r = r0 + i * GROUPS;
      v[i] = rows[(size_t)(r < n_rows ? r : g) * kRowStride + col];
    }
#pragma unroll
    for (int i = 0; i < 5; ++i)
      if (r0 + i * GROUPS < n_rows) acc += v[i];
  }
  return acc;
}

// Batched forward with the convolution on the tensor cores (forward_tc.cu): path 1 or 2; uint8 pixels, path 1.
int forward_device_tc(cnn_net* net, int path, const float* d_images, long n, float* d_out, int* d_argmax,
                      cudaStream_t stream);
int forward_device_tc_u8(cnn_net* net, const unsigned char* d_pixels, long n, float* d_out, int* d_argmax,
                         cudaStream_t stream);
int ensure_train_scratch(cnn_net* net);
// Fused forward + backward of n images at fixed parameters, on the CUDA cores or the tensor cores: *rows partial rows in net->d_partials.
// `chained`: the kernel before this one on the stream is this library's reduce + update kernel of the previous
// step of the same call (then, and only then, the gradient kernel may fetch its first images before waiting
// for that kernel: see k_grad_partials).
int launch_gradient(cnn_net* net, const float* d_images, const unsigned* d_labels, long n, cudaStream_t st, bool chained, int* rows);
// Its tensor-core part: a row per share, but for what left[b] says of block b's.
int launch_grad_tc(cnn_net* net, const float* d_images, const unsigned* d_labels, GradShares shares, GradLeft* left, int* pushed, cudaStream_t st);
int launch_persample_cluster8(cnn_net* net, const float* d_images, const unsigned* d_labels, long n, int epochs,
                              float dt, float threshold, float* d_mean, int* d_ran, cudaStream_t st);

}  // namespace cnn
