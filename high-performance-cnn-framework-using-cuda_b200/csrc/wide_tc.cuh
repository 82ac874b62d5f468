// tcgen05 (5th-generation tensor core) building blocks of the tensor-core kernels: shared-memory matrix
// descriptors for the un-swizzled ("interleaved") canonical layouts, the fp16 instruction descriptor, TMEM
// allocation and loads, and the commit -> mbarrier hand-over.  One CTA per MMA (cta_group::1), operands in
// shared memory, fp32 accumulators in tensor memory.
#pragma once

#include <cuda_fp16.h>

#include "net.cuh"

namespace cnn {
namespace tc {

// Canonical un-swizzled layout: "core matrices" of 8 rows x 16 bytes, rows 16 bytes apart.
// Read as a K-major operand (rows = M or N, a row's 16 bytes = 8 fp16 values along K): LBO = distance to the next
// 8 values of K, SBO = distance to the next 8 rows.  Read as an MN-major operand (rows = K, a row's 16 bytes = 8
// values along M or N): LBO = distance to the next 8 values of K, SBO = distance to the next 8 values of M or N.

// 64-bit shared-memory matrix descriptor: start address, leading / stride byte offsets (all in units
// of 16 B), descriptor version 1, no swizzle.
__device__ __forceinline__ unsigned long long smem_desc(unsigned smem_addr, unsigned lbo_bytes, unsigned sbo_bytes) {
  unsigned long long d = 0;
  d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
  d |= (unsigned long long)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (unsigned long long)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;
  return d;
}

// Instruction descriptor for kind::f16 with both operands in fp16 (formats 0) and K-major (bits 15 and 16: MN-major A
// and B), fp32 accumulation (bits 4-5 = 1), N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr unsigned idesc_f16(int M, int N) {
  return (1u << 4) | ((unsigned)(N >> 3) << 17) | ((unsigned)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_alloc(unsigned* smem_dst, unsigned cols) {   // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned cols) {     // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Generic-proxy shared-memory writes -> visible to the async proxy (the tensor core's operand reads).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem], K = 16 fp16 values.  Called by a WHOLE converged warp: the operands are warp-uniform and
// one elected lane issues.  (Measured on B200: a tcgen05.mma issued from inside a divergent branch ("if (tid == 0)")
// costs the issuing thread about 146 cycles whatever its shape; issued this way it costs its operand traffic at
// 128 B/cycle of shared memory.)
__device__ __forceinline__ void mma_f16_elect(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc,
                                              unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// COUNT (5 or 8) of them into one accumulator, the descriptors' start addresses A_STEP and B_STEP (in units of 16 B) further on each time;
// all but the first accumulate.
#define CNN_MMA_NEXT "add.s64 a, a, %5;\n\tadd.s64 b, b, %6;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
#define CNN_MMA_FIRST                                                                                                          \
  "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\tmov.b64 a, %1;\n\tmov.b64 b, %2;\n\t" \
  "elect.sync _|q, 0xffffffff;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
template <int COUNT, int A_STEP, int B_STEP>
__device__ __forceinline__ void mma_f16_run_elect(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
  static_assert(COUNT == 5 || COUNT == 8, "");
  if constexpr (COUNT == 5) {
    asm volatile(CNN_MMA_FIRST CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT "}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc),
                 "r"(accumulate), "n"(A_STEP), "n"(B_STEP)
                 : "memory");
  } else {
    asm volatile(CNN_MMA_FIRST CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT CNN_MMA_NEXT "}" ::"r"(tmem_d), "l"(adesc),
                 "l"(bdesc), "r"(idesc), "r"(accumulate), "n"(A_STEP), "n"(B_STEP)
                 : "memory");
  }
}
#undef CNN_MMA_NEXT
#undef CNN_MMA_FIRST
// Whole converged warp: the lane that elect.sync picks (the same one every time for a full mask)
// arrives on the mbarrier when every MMA it has issued so far has completed.
__device__ __forceinline__ void mma_commit_elect(unsigned long long* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
      : "memory");
}
// Eight consecutive fp32 columns of this warp's 32 tensor-memory lanes; not waited for.
__device__ __forceinline__ void tmem_ld8_nowait(unsigned taddr, unsigned (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// Wait for this warp's outstanding tensor-memory loads; the registers are listed as in/out operands
// so that their uses cannot be scheduled above the wait.
__device__ __forceinline__ void tmem_wait8(unsigned (&a)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
               :: "memory");
}

// Split two fp32 values, times a power of two, into fp16 high parts (round to nearest) and fp16 remainders: hi + lo to
// about 2^-23 relative, or to 2^-25 absolute where lo is an fp16 subnormal.  From 65,520 on hi is infinite.
__device__ __forceinline__ void split_f16x2(float x, float y, float scale, __half2& hi, __half2& lo) {
  const f32x2 s = pack2(scale, scale), v = pack2(x, y);
  float sx, sy;
  unpack2(mul2(v, s), sx, sy);
  hi = __floats2half2_rn(sx, sy);
  const float2 b = __half22float2(hi);
  unpack2(fma2(v, s, pack2(-b.x, -b.y)), sx, sy);
  lo = __floats2half2_rn(sx, sy);
}

}  // namespace tc
}  // namespace cnn
