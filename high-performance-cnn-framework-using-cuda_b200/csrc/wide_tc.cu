// The widened configuration on the 5th-generation tensor cores (tcgen05): convolution, sigmoid and subsample layer of the
// forward pass in one kernel, and everything between the subsample deltas and the conv gradients of the backward pass in
// another, which computes the activations again instead of reading them back (at 56x56 with 64 maps they are 692 KB per
// image: written once and read twice they were 2.1 GB of a 1,024-image step's traffic).  The two kernels are one template:
// operands, convolution and sigmoid are the same.
//
// Convolution, without an im2col copy.  M = 16 groups of 8 output rows (any images' -- an image has ceil(C / 8) groups), a
// unit of work is one group set and one column q of 4x4 windows: four output columns of 64 maps from eight
// input columns 4q .. 4q+7.  A unit's operand is a slab of [16 groups][13 rows][8 columns] fp16: a row is 16 bytes, so a matrix
// descriptor may start at any row, and with a distance of 16 bytes between the two K chunks of an MMA its K = 16 are the
// eight columns of TWO kernel rows: the five rows of the filter take three MMAs (the sixth row's weights are zero).  The
// weights are a banded B operand, the same for every unit:
//   out[y][4q + x][f] = sum_i sum_c slab[y + i][c] * T_i[c][x][f],  T_i[c][x][f] = Wc[f][i][c - x] (0 <= c - x < 5).
// Accumulator columns are ordered 8 * (f / 2) + 2 * x + f % 2: eight columns are one window row of two maps.  An accumulator
// holds half a unit (32 maps, 128 columns); three of them rotate.
//
// Weight gradient (bp_weight_c1, layer.cu:363-381), from the same slabs: with the conv deltas dc of the unit,
//   D[(x, f)][(i, c)] = sum_rows dc[row][x][f] * slab[row + i][c],   G[f][i][j] = sum_x D[(x, f)][(i, x + j)],
// an MMA with K = rows of the unit: the deltas are the A operand (M = 128: (x, f) of 32 maps; M-contiguous, as the epilogue
// lanes, which are rows, have them), the slab is the B operand (N = 48: six kernel rows of eight columns, the sixth unused;
// N-contiguous, one row of the slab per kernel row further).  D does not depend on the unit, so it accumulates in tensor
// memory; every kTwFlush units it is added to fp32 sums in memory (the tensor core's additions truncate).
//
// Accuracy.  Operands are fp16 high parts and remainders, three passes (hi*hi + lo*hi + hi*lo), fp32 accumulation: what is left
// out is lo*lo, about 2^-24 relative ("conv" = 2); one pass of high parts has 11 significant bits ("conv" = 1).  fp16's range
// is met with powers of two taken from the largest magnitudes: of the weights, of the batch's pixels (k_wide_prep) and of
// the batch's subsample deltas (k_wide_bp_fc); they are undone exactly.  (tf32 operands need twice the MMAs, and deltas
// in a layout that costs one 4-byte store per value and part.)
//
// One CTA per SM, 24 warps (80 registers), hand-overs by mbarriers with bounded waits:
//   warps 0-6   load a unit's rows (32 bytes per thread, one unit ahead in registers), split them and store the slab;
//               backward: warps 0-3 also drain the gradient accumulators, of which two sets alternate (374 us against 386 for a
//               step of 1,024 images with one set drained by the epilogue);
//   warp 7      issues the MMAs (an elected lane of the converged warp) and commits to mbarriers;
//   warps 8-23  epilogue, a quarter of the rows and 16 maps: tcgen05.ld of 8 columns at a time; bias, sigmoid.
//               Forward: the window row's four subsample taps, the four rows of a window by a shuffle reduce-scatter, sigmoid, out;
//               all warps half by half, as the tensor core is ahead.  Backward: deltas, their fp16 parts into the A operand,
//               subsample-filter gradient and bias sums in registers; eight warps for each half of a unit, so that one half's work
//               while the other's wait for the tensor core (377 -> 363 us, with one pass 344 -> 325).
// Bounds: forward 97 us for 1,024 images (before, with an im2col gather and a subsample kernel of its own: 174 + 152 us), the
// special-function unit two thirds busy; backward 192 us (454 us, which did not have to compute the activations), special-function
// unit, fp32 pipe and issue slots about half busy each, the rest the hand-overs between tensor core and epilogue.
// Work is cut into equal ranges of units, so a CTA may begin and end in the middle of a group set.
#include <type_traits>

#include "cluster_exchange.cuh"
#include "phase_clocks.cuh"
#include "wide.cuh"
#include "wide_tc.cuh"

namespace cnn {

constexpr int kTwThreads = 768;
constexpr int kTwGroups = 16, kTwGroupRows = 13;
constexpr unsigned kTwGroupStride = kTwGroupRows * 16;              // 208 B
constexpr unsigned kTwPlane = kTwGroups * kTwGroupStride;           // 3,328 B: one part of a slab
constexpr int kTwSlabs = 6;                                         // units in flight between loader and tensor core
constexpr int kTwN = 4 * kTwF;                                      // accumulator columns of a unit
constexpr unsigned kTwBChunk = kTwN * 16;                           // 4,096 B between the two K chunks of a B step
constexpr unsigned kTwBPart = 3 * 2 * kTwBChunk;                    // 24,576 B
constexpr int kTwLoadWarps = 7, kTwMmaWarp = 7, kTwEpiWarp0 = 8, kTwEpiWarps = 16;
constexpr int kTwRows = kTwGroups * kTwGroupRows;                   // 208 loader threads with work
constexpr float kTwMaxExp = 31.f;                                   // (1 + 2^31)^4 is still finite
constexpr int kTwHalf = kTwN / 2;                                   // columns of a half (32 maps): what an accumulator holds
constexpr int kTwAccMax = 4;                                        // accumulators in the forward kernel; the backward kernel has two
// backward
constexpr unsigned kTwDcChunk = 128 * 16;                           // 8 values of (x, f) for 128 rows
constexpr unsigned kTwDcPart = (kTwHalf / 8) * kTwDcChunk;          // 32 KB: one part of a half's deltas
constexpr int kTwGradCol = 2 * kTwHalf;                             // two sets of gradient accumulators (a set: both halves) behind the others
constexpr int kTwFlush = 4;                                         // units between two hand-overs of a set

struct TwSmem {
  alignas(128) unsigned char slab[kTwSlabs][2][kTwPlane];           // [high, low]
  alignas(128) unsigned char b[2][kTwBPart];
  alignas(16) float bias[kTwF];
  alignas(16) float ws[16];
  float bs;
  unsigned long long a_full[kTwSlabs], a_free[kTwSlabs], d_full[kTwAccMax], d_free[kTwAccMax];
  unsigned long long dc_full[2], dc_free[2], g_full[2], g_free[2];  // backward: deltas of a half, sets of gradient accumulators
  float max_of[3][kTwThreads / 32];                                 // largest tap, pixel, subsample delta by warp
  unsigned tmem_base;
  long long clock_base;                                             // phase clocks only
};
struct TwBwdSmem {
  TwSmem s;
  alignas(128) unsigned char dc[2][2][kTwDcPart];                   // [half][high, low]
  float red[kTwEpiWarps][24];                                       // subsample-filter gradient of a warp
};

CNN_PHASE_TABLE(g_phase_clocks_wg, 24)

bool wide_tc_supported(const WideDims& d) { return d.F % kTwF == 0 && d.H % 4 == 0; }

__device__ __forceinline__ float warp_max(float m) {
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, k));
  return m;
}
// Exponent e with 2^e <= v < 2^(e+1), kept where scales built from it stay normal numbers.
__device__ __forceinline__ int exponent_of(float v) {
  const int e = (int)((__float_as_uint(v) >> 23) & 255u) - 127;
  return e > 60 ? 60 : (e < -60 ? -60 : e);
}
// *p += v, not waited for.
__device__ __forceinline__ void red_add(float* p, float v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((127 + e) << 23); }

// What the tensor-core kernels need of a batch beforehand: per-block maxima of the (finite) pixel magnitudes, and the FC weights
// in the order in which those kernels have the subsample activations, [window][map] instead of [map][window].
__global__ void __launch_bounds__(256)
k_wide_prep(WideDims d, const float4* __restrict__ images, long quads, const float* __restrict__ params, float* __restrict__ pixel_max,
            float* __restrict__ wf_t) {
  __shared__ float red[8];
  float m = 0.f;
  pdl_launch_dependents();
  pdl_wait();
#pragma unroll 4
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += (long)gridDim.x * blockDim.x) {
    const float4 v = __ldg(images + i);
    const float a[4] = {fabsf(v.x), fabsf(v.y), fabsf(v.z), fabsf(v.w)};
#pragma unroll
    for (int k = 0; k < 4; ++k) m = (a[k] <= 3.4e38f) ? fmaxf(m, a[k]) : m;
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  const int W = d.P * d.P;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < (long)kOut * d.S; i += (long)gridDim.x * blockDim.x) {
    const int k = (int)(i / d.S), s = (int)(i - (long)k * d.S);
    wf_t[i] = params[d.o_wf + (size_t)k * d.S + (size_t)(s % d.F) * W + s / d.F];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 1; k < 8; ++k) m = fmaxf(m, red[k]);
    pixel_max[blockIdx.x] = m;
  }
}

// FL: sigmoid flavour.  PASSES: 3 or 1.  BWD: false = forward (writes as), true = backward (reads ds, writes the partial gradients).
// as, ds: [image][window][map].  part_g: per CTA (of all map groups) [kTwGradN][256] sums of D; part_b: per CTA [4][64] conv bias
// sums (a row per quarter of the rows) and the 17 subsample-filter sums behind them.
template <int FL, int PASSES, bool BWD>
__global__ void __launch_bounds__(kTwThreads, 1)
k_wide_tc(WideDims d, long n, const float* __restrict__ images, const float* __restrict__ params, const float* __restrict__ pixel_max,
          float* __restrict__ as, const float* __restrict__ ds, const float* __restrict__ ds_max, int ds_blocks,
          float* __restrict__ part_g, float* __restrict__ part_b, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem_base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  TwSmem& sm = *reinterpret_cast<TwSmem*>(smem_base);
  TwBwdSmem& sb = *reinterpret_cast<TwBwdSmem*>(smem_base);        // backward only
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool kShort = (FL == 1);
  constexpr int kAcc = BWD ? 2 : kTwAccMax;
  constexpr float kPre = kShort ? -1.4426950408889634f : 1.0f;     // the short sigmoid form's factor, folded into taps and bias
  const int f0 = blockIdx.y * kTwF;
  const int gi = (d.C + 7) / 8;                                    // groups per image
  // (at most 2,097,120 images: group and unit numbers fit in 32 bits, and a unit's place is advanced, not divided out)
  const long n_units = (n * gi + kTwGroups - 1) / kTwGroups * d.P;
  const unsigned u0 = (unsigned)(n_units * blockIdx.x / gridDim.x);
  const int units = (int)(n_units * (blockIdx.x + 1) / gridDim.x - u0);
  const unsigned set0 = u0 / (unsigned)d.P, q0 = u0 - set0 * (unsigned)d.P;      // group set and window column of the first unit

  if (tid == 0) {
    for (int s = 0; s < kTwSlabs; ++s) {
      mbar_init(&sm.a_full[s], kTwLoadWarps);
      mbar_init(&sm.a_free[s], 1);
    }
    for (int s = 0; s < kAcc; ++s) {
      mbar_init(&sm.d_full[s], 1);
      mbar_init(&sm.d_free[s], BWD ? kTwEpiWarps / 2 : kTwEpiWarps);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&sm.dc_full[h], kTwEpiWarps / 2);
      mbar_init(&sm.dc_free[h], 1);
      mbar_init(&sm.g_full[h], 1);
      mbar_init(&sm.g_free[h], 4);
    }
    mbar_fence_init();
  }
  if (warp == kTwMmaWarp) tc::tmem_alloc(&sm.tmem_base, 512);
  pdl_launch_dependents();
  pdl_wait();

  // ---- scales: taps to 256..512, pixels to 2^14..2^15 at most ------------------------------------------------
  float wmax = 0.f, pmax = 0.f, dmax = 0.f;
  for (int i = tid; i < kTwF * 25; i += kTwThreads) {
    const float a = fabsf(kPre * params[d.o_wc + f0 * 25 + i]);
    wmax = (a <= 3.4e38f) ? fmaxf(wmax, a) : wmax;
  }
  if (tid < kTwPrepBlocks) pmax = pixel_max[tid];
  if (BWD)
    for (int i = tid; i < ds_blocks; i += kTwThreads) dmax = fmaxf(dmax, ds_max[i]);
  wmax = warp_max(wmax);
  pmax = warp_max(pmax);
  dmax = warp_max(dmax);
  if (lane == 0) {
    sm.max_of[0][warp] = wmax;
    sm.max_of[1][warp] = pmax;
    sm.max_of[2][warp] = dmax;
  }
  __syncthreads();
  const int mine_at = lane < kTwThreads / 32 ? lane : 0;
  wmax = warp_max(sm.max_of[0][mine_at]);
  pmax = warp_max(sm.max_of[1][mine_at]);
  dmax = warp_max(sm.max_of[2][mine_at]);
  const int we = 8 - exponent_of(wmax), pe = 14 - exponent_of(pmax);
  const int back = -(we + pe);
  const float w_scale = pow2i(we), px_scale = pow2i(pe), unscale = pow2i(back < -126 ? -126 : (back > 126 ? 126 : back));
  // conv deltas, at most max |Ws| / (C*C) * max |delta_s| / 4, to 2^14 at most
  int dc_exp = 0;
  if (BWD) {
    float ws_max = fabsf(params[d.o_ws + (lane & 15)]);
#pragma unroll
    for (int k = 8; k > 0; k >>= 1) ws_max = fmaxf(ws_max, __shfl_xor_sync(0xffffffffu, ws_max, k));
    dc_exp = 14 - exponent_of(ws_max / (float)(d.C * d.C)) - exponent_of(dmax);
    dc_exp = dc_exp > 100 ? 100 : (dc_exp < -100 ? -100 : dc_exp);
  }

  // ---- weights: step s holds kernel rows 2 s and 2 s + 1, chunk = kernel row, row = accumulator column -----------
  for (int e = tid; e < 3 * 2 * kTwN; e += kTwThreads) {
    const int i = e / kTwN, col = e % kTwN;
    const int f = 2 * (col >> 3) + (col & 1), x = (col & 7) >> 1;
    float w[5];
#pragma unroll
    for (int t = 0; t < 5; ++t) w[t] = i < 5 ? kPre * params[d.o_wc + (f0 + f) * 25 + (i < 5 ? i : 0) * 5 + t] : 0.f;
    __half2 hi[4], lo[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        v[h] = 0.f;
#pragma unroll
        for (int t = 0; t < 5; ++t) v[h] = (2 * c + h - x == t) ? w[t] : v[h];
      }
      tc::split_f16x2(v[0], v[1], w_scale, hi[c], lo[c]);
    }
    const unsigned off = (unsigned)i * kTwBChunk + (unsigned)col * 16u;
    *reinterpret_cast<uint4*>(sm.b[0] + off) = *reinterpret_cast<uint4*>(hi);
    if (PASSES == 3) *reinterpret_cast<uint4*>(sm.b[1] + off) = *reinterpret_cast<uint4*>(lo);
  }
  if (tid < kTwF) sm.bias[tid] = kPre * params[d.o_bc + f0 + tid];
  else if (tid < kTwF + 16) sm.ws[tid - kTwF] = params[d.o_ws + tid - kTwF];
  else if (tid == kTwF + 16) sm.bs = params[d.o_bs];
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const unsigned tmem_base = sm.tmem_base;
  bool gave_up = false;
  CNN_PHASE_BEGIN(blockIdx.x == 0 && blockIdx.y == 0, sm.clock_base)

  if (warp < kTwLoadWarps) {
    // ================= loaders: thread = (group, row) ===============================================
    const int g = tid / kTwGroupRows, row = tid - g * kTwGroupRows;
    const bool mine = tid < kTwRows;
    float4 v0, v1;
    bool have;
    const float* src;
    unsigned G = set0 * kTwGroups + (mine ? g : 0);
    auto place = [&]() {
      const unsigned b = G / (unsigned)gi;
      const int y = 8 * (int)(G - b * (unsigned)gi) + row;
      have = mine && b < n && y < d.H;
      src = images + ((size_t)(have ? b : 0) * d.H + (have ? y : 0)) * d.H;
    };
    auto load = [&](int q) {           // (clamped, not conditional: a load under a condition is waited for on the spot)
      v0 = __ldg(reinterpret_cast<const float4*>(src + 4 * q));
      v1 = __ldg(reinterpret_cast<const float4*>(src + 4 * q) + 1);
    };
    int q = (int)q0;
    place();
    load(q);
    // Backward, warps 0-3: adds (or, the first time, puts) a complete set of gradient accumulators, a warp its quarter of the rows (x, f),
    // to the CTA's sums -- every address has one thread that adds to it, in order; as a reduction, which needs no answer.
    auto flush = [&](int set) {
      if (warp >= 4) return;
      mbar_wait_bounded(&sm.g_full[set & 1], (unsigned)(set >> 1) & 1u, status, gave_up);
      __syncwarp();
      tc::fence_after_sync();
      const unsigned t0 = tmem_base + ((unsigned)(warp * 32) << 16) + (unsigned)(kTwGradCol + (set & 1) * 2 * kTwGradN);
      float* dst = part_g + (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * kTwGradN * kTwGradCols + warp * 32 + lane;
      const float s1 = pow2i(-dc_exp), s2 = pow2i(-pe);
#pragma unroll 1
      for (int c = 0; c < 2 * kTwGradN; c += 8) {
        unsigned r[8];
        tc::tmem_ld8_nowait(t0 + (unsigned)c, r);
        tc::tmem_wait8(r);
        float* to = dst + (c < kTwGradN ? c * kTwGradCols : (c - kTwGradN) * kTwGradCols + 128);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float v = __uint_as_float(r[e]) * s1 * s2;
          if (set > 0) red_add(to + e * kTwGradCols, v);
          else to[e * kTwGradCols] = v;
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.g_free[set & 1]);
    };
    for (int k = 0; k < units; ++k) {
      const int s = k % kTwSlabs;
      CNN_PHASE(0);
      mbar_wait_bounded(&sm.a_free[s], ((unsigned)(k / kTwSlabs) & 1u) ^ 1u, status, gave_up);
      CNN_PHASE(1);
      // (the slab is free: the gradients of the unit that had it are complete, and with the last unit of a set the set)
      if (BWD && k >= kTwSlabs && (k - kTwSlabs) % kTwFlush == kTwFlush - 1) flush((k - kTwSlabs) / kTwFlush);
      __half2 hi[4], lo[4];
      tc::split_f16x2(have ? v0.x : 0.f, have ? v0.y : 0.f, px_scale, hi[0], lo[0]);
      tc::split_f16x2(have ? v0.z : 0.f, have ? v0.w : 0.f, px_scale, hi[1], lo[1]);
      tc::split_f16x2(have ? v1.x : 0.f, have ? v1.y : 0.f, px_scale, hi[2], lo[2]);
      tc::split_f16x2(have ? v1.z : 0.f, have ? v1.w : 0.f, px_scale, hi[3], lo[3]);
      if (mine) {
        *reinterpret_cast<uint4*>(sm.slab[s][0] + tid * 16) = *reinterpret_cast<uint4*>(hi);
        if (PASSES == 3) *reinterpret_cast<uint4*>(sm.slab[s][1] + tid * 16) = *reinterpret_cast<uint4*>(lo);
      }
      if (++q == d.P) {
        q = 0;
        G += kTwGroups;
        place();
      }
      load(q);                         // (after the last unit: a group past the range, or the first rows)
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.a_full[s]);
      CNN_PHASE(2);
    }
    if (BWD)
      for (int set = units > kTwSlabs ? (units - kTwSlabs) / kTwFlush : 0; set <= (units - 1) / kTwFlush; ++set) flush(set);
  } else if (warp == kTwMmaWarp) {
    // ================= MMA issue: the whole warp runs the loop, one elected lane issues =============
    const unsigned idesc = tc::idesc_f16(128, kTwHalf);
    const unsigned idesc_g = tc::idesc_f16(128, kTwGradN) | (1u << 15) | (1u << 16);      // both operands MN-major
    const unsigned long long b_d[2] = {tc::smem_desc(smem_u32(sm.b[0]), kTwBChunk, 128), tc::smem_desc(smem_u32(sm.b[1]), kTwBChunk, 128)};
    const int halves = 2 * units;
    for (int v = 0; v < halves + (BWD ? 2 : 0); ++v) {
      if (v < halves) {
        const int k = v >> 1, h = v & 1, s = k % kTwSlabs, acc = v % kAcc;
        CNN_PHASE(0);
        if (h == 0) mbar_wait_bounded(&sm.a_full[s], (unsigned)(k / kTwSlabs) & 1u, status, gave_up);
        CNN_PHASE(1);
        mbar_wait_bounded(&sm.d_free[acc], ((unsigned)(v / kAcc) & 1u) ^ 1u, status, gave_up);
        CNN_PHASE(2);
        __syncwarp();
        tc::fence_after_sync();
        const unsigned long long a_d[2] = {tc::smem_desc(smem_u32(sm.slab[s][0]), 16, kTwGroupStride),
                                           tc::smem_desc(smem_u32(sm.slab[s][1]), 16, kTwGroupStride)};
#pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) {
#pragma unroll
          for (int st = 0; st < 3; ++st)
            tc::mma_f16_elect(tmem_base + (unsigned)(acc * kTwHalf), a_d[pass == 1 ? 1 : 0] + (unsigned)(2 * st),
                              b_d[pass == 2 ? 1 : 0] + (unsigned)h * (kTwHalf * 16 >> 4) + (unsigned)st * (2 * kTwBChunk >> 4), idesc,
                              (pass | st) ? 1u : 0u);
        }
        tc::mma_commit_elect(&sm.d_full[acc]);
        if (!BWD && h == 1) tc::mma_commit_elect(&sm.a_free[s]);
        CNN_PHASE(3);
      }
      if (BWD && v >= 2) {
        // the gradient of the half two steps back: its deltas were made while the convolutions since then ran
        const int gv = v - 2, k = gv >> 1, h = gv & 1, s = k % kTwSlabs;
        const int set = k / kTwFlush;
        const bool first = k % kTwFlush == 0;
        CNN_PHASE(4);
        mbar_wait_bounded(&sm.dc_full[h], (unsigned)k & 1u, status, gave_up);
        CNN_PHASE(5);
        if (first && h == 0) mbar_wait_bounded(&sm.g_free[set & 1], ((unsigned)(set >> 1) & 1u) ^ 1u, status, gave_up);
        CNN_PHASE(6);
        __syncwarp();
        tc::fence_after_sync();
        const unsigned long long x_d[2] = {tc::smem_desc(smem_u32(sm.slab[s][0]), kTwGroupStride, 16),
                                           tc::smem_desc(smem_u32(sm.slab[s][1]), kTwGroupStride, 16)};
        const unsigned long long dc_d[2] = {tc::smem_desc(smem_u32(sb.dc[h][0]), 128, kTwDcChunk),
                                            tc::smem_desc(smem_u32(sb.dc[h][1]), 128, kTwDcChunk)};
#pragma unroll 1
        for (int pass = 0; pass < PASSES; ++pass) {
          const unsigned long long a = pass == 1 ? dc_d[1] : dc_d[0], b = pass == 2 ? x_d[1] : x_d[0];
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)       // 16 rows = two groups
            tc::mma_f16_elect(tmem_base + (unsigned)(kTwGradCol + (2 * (set & 1) + h) * kTwGradN), a + (unsigned)(ks * 256 >> 4),
                              b + (unsigned)(ks * 2 * kTwGroupStride >> 4), idesc_g, (first && pass == 0 && ks == 0) ? 0u : 1u);
        }
        tc::mma_commit_elect(&sm.dc_free[h]);
        if (h == 1) {
          tc::mma_commit_elect(&sm.a_free[s]);
          if (k % kTwFlush == kTwFlush - 1 || k == units - 1) tc::mma_commit_elect(&sm.g_full[set & 1]);
        }
        CNN_PHASE(7);
      }
    }
  } else {
    // ================= epilogue ====================================================================
    const int ew = warp - kTwEpiWarp0, h = ew >> 3, quarter = warp & 3;
    // The warp's 16 maps: backward 16 of its half h from m0 on, forward eight of each half, m0 .. and 32 + m0 ..
    constexpr int kPartMaps = BWD ? 8 : 32;
    const int m0 = BWD ? 32 * h + 16 * ((ew >> 2) & 1) : 8 * (ew >> 2);
    const int rsub = lane & 3;                     // row of the 4x4 window
    const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;
    const f32x2 one2 = pack2(1.f, 1.f), minus2 = pack2(-1.f, -1.f), unscale2 = pack2(unscale, unscale);
    const float inv_c = 1.0f / (float)(d.C * d.C);
    f32x2 k2[4];                                   // forward: the row's subsample taps; backward: times -2^dc_exp / (C*C)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float w = BWD ? -sm.ws[rsub * 4 + j] * inv_c * pow2i(dc_exp) : sm.ws[rsub * 4 + j];
      k2[j] = pack2(w, w);
    }
    const unsigned lane_base = tmem_base + ((unsigned)(quarter * 32) << 16);
    // backward: sums of this lane's row over units: subsample-filter taps (row rsub, negated) and delta_s in halves by map parity,
    // and the conv bias per map pair of either half
    f32x2 gs2[4], gds2 = pack2(0.f, 0.f), gb2[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) gs2[j] = gb2[j] = gb2[4 + j] = pack2(0.f, 0.f);
    int q = (int)q0;
    unsigned G = set0 * kTwGroups + quarter * 4 + (lane >> 3);
    bool live;
    float* at;                       // this lane's window and maps in as / ds; of a window that does not exist: the zeros behind ds
    auto place = [&]() {
      const unsigned b = G / (unsigned)gi;
      const int p = (8 * (int)(G - b * (unsigned)gi) + (lane & 7)) >> 2;      // C is a multiple of 4: a window's rows are all in or all out
      live = b < n && p < d.P;
      const size_t window = live ? ((size_t)b * d.P + p) * d.P + q : (BWD ? (size_t)n * d.P * d.P : 0);
      at = (BWD ? const_cast<float*>(ds) : as) + window * d.F + f0 + m0;
    };
    place();
    // Backward: the window's deltas of eight maps, the next eight taken as soon as these are used.
    float4 dlo, dhi;
    if (BWD) {
      dlo = __ldg(reinterpret_cast<const float4*>(at));
      dhi = __ldg(reinterpret_cast<const float4*>(at) + 1);
    }
    for (int k = 0; k < units; ++k) {
      unsigned nxt[8];
#pragma unroll
      for (int part = 0; part < 2; ++part) {         // eight maps
        const int acc = BWD ? h : 2 * (k & 1) + part;
        const unsigned t0 = lane_base + (unsigned)(acc * kTwHalf + 4 * (m0 & 31) + (BWD ? 32 * part : 0));
        if (!BWD || part == 0) {
          CNN_PHASE(0);
          mbar_wait_bounded(&sm.d_full[acc], (unsigned)(BWD ? k : k >> 1) & 1u, status, gave_up);
          CNN_PHASE(1);
          __syncwarp();
          tc::fence_after_sync();
          tc::tmem_ld8_nowait(t0, nxt);
          tc::tmem_wait8(nxt);
        }
        if (BWD && part == 1) {      // `at` is only for the loads ahead
          if (live) at += d.F;
          if (++q == d.P) {
            q = 0;
            G += kTwGroups;
            place();
          }
        }
        float z[8];
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {           // a window row of maps m0 + kPartMaps * part + 2 ch + {0, 1}
          const f32x2 bias2 = *reinterpret_cast<const f32x2*>(&sm.bias[m0 + kPartMaps * part + 2 * ch]);
          f32x2 a2[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            a2[j] = fma2(pack2(__uint_as_float(nxt[2 * j]), __uint_as_float(nxt[2 * j + 1])), unscale2, bias2);
          if ((BWD && part == 0) || ch < 3) {
            tc::tmem_ld8_nowait(t0 + (unsigned)((ch + 1) * 8), nxt);
          } else {
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.d_free[acc]);
          }
          if constexpr (BWD && kShort) {
            // -a = 1 / (-1 - 2^t): a reciprocal each, which costs fewer issue slots than sharing them as below
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, yv;
              unpack2(a2[j], x, yv);
              unpack2(fma2(pack2(exp2f_approx(x), exp2f_approx(yv)), minus2, minus2), x, yv);
              a2[j] = pack2(rcp_approx(x), rcp_approx(yv));
            }
          } else if constexpr (kShort) {
            // 1 / d_j with d_j = 1 + 2^t_j: one reciprocal for the row's four (t is capped so that their product stays finite: an
            // activation below 4.7e-10 counts as that)
            f32x2 dd[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, yv;
              unpack2(a2[j], x, yv);
              dd[j] = add2(pack2(exp2f_approx(min_nan(x, kTwMaxExp)), exp2f_approx(min_nan(yv, kTwMaxExp))), one2);
            }
            const f32x2 d01 = mul2(dd[0], dd[1]), d23 = mul2(dd[2], dd[3]);
            float x, yv;
            unpack2(mul2(d01, d23), x, yv);
            const f32x2 r = pack2(rcp_approx(x), rcp_approx(yv));
            const f32x2 n01 = fma2(k2[0], dd[1], mul2(k2[1], dd[0])), n23 = fma2(k2[2], dd[3], mul2(k2[3], dd[2]));
            unpack2(mul2(r, fma2(n01, d23, mul2(n23, d01))), z[2 * ch], z[2 * ch + 1]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, yv;
              unpack2(a2[j], x, yv);
              a2[j] = BWD ? pack2(-sigmoidf<FL>(x), -sigmoidf<FL>(yv)) : pack2(sigmoidf<FL>(x), sigmoidf<FL>(yv));
            }
            if constexpr (!BWD)
              unpack2(fma2(k2[3], a2[3], fma2(k2[2], a2[2], fma2(k2[1], a2[1], mul2(k2[0], a2[0])))), z[2 * ch], z[2 * ch + 1]);
          }
          if constexpr (BWD) {
            const float4 dq = ch < 2 ? dlo : dhi;
            const f32x2 dl = ch % 2 ? pack2(dq.z, dq.w) : pack2(dq.x, dq.y);
            unsigned hi[4], lo[4];
            f32x2 sum;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              // a2 is -a: m = -dl a, m - m a = -dl a (1 - a)
              const f32x2 m = mul2(dl, a2[j]);
              gs2[j] = add2(gs2[j], m);
              const f32x2 dcv = mul2(k2[j], fma2(m, a2[j], m));
              sum = j ? add2(sum, dcv) : dcv;
              float x, yv;
              unpack2(dcv, x, yv);
              const __half2 hv = __floats2half2_rn(x, yv);
              hi[j] = *reinterpret_cast<const unsigned*>(&hv);
              if (PASSES == 3) {
                const float2 bk = __half22float2(hv);
                unpack2(fma2(pack2(bk.x, bk.y), minus2, dcv), x, yv);
                const __half2 lv = __floats2half2_rn(x, yv);
                lo[j] = *reinterpret_cast<const unsigned*>(&lv);
              }
            }
            gb2[4 * part + ch] = add2(gb2[4 * part + ch], sum);
            gds2 = add2(gds2, dl);                 // (the window's four lanes have the same: lane 0's sum is used)
            if (ch == 1) dlo = __ldg(reinterpret_cast<const float4*>(part ? at : at + 8));
            if (ch == 3) dhi = __ldg(reinterpret_cast<const float4*>(part ? at : at + 8) + 1);
            if (part == 0 && ch == 0) {
              CNN_PHASE(2);
              mbar_wait_bounded(&sm.dc_free[h], ((unsigned)k & 1u) ^ 1u, status, gave_up);
              CNN_PHASE(3);
            }
            unsigned char* dst = sb.dc[h][0] + (unsigned)((m0 & 31) / 2 + 4 * part + ch) * kTwDcChunk + (unsigned)(quarter * 32 + lane) * 16u;
            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            if (PASSES == 3) *reinterpret_cast<uint4*>(dst + kTwDcPart) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
          if ((BWD && part == 0) || ch < 3) tc::tmem_wait8(nxt);
        }
        if constexpr (!BWD) {
          // the window's four rows are four neighbouring lanes: reduce-scatter, lane r ends with maps 4 (r & 1) + 2 (r >> 1) + {0, 1}
          float w4[4], w2[2];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float send = b0 ? z[i] : z[i + 4], keep = b0 ? z[i + 4] : z[i];
            w4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float send = b1 ? w4[i] : w4[i + 2], keep = b1 ? w4[i + 2] : w4[i];
            w2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
          }
          if (live)
            *reinterpret_cast<float2*>(at + kPartMaps * part + (b0 ? 4 : 0) + (b1 ? 2 : 0)) =
                make_float2(sigmoidf<FL>(w2[0] + sm.bs), sigmoidf<FL>(w2[1] + sm.bs));
        }
      }
      CNN_PHASE(4);
      if (BWD) {
        tc::fence_async_smem();        // generic-proxy writes -> visible to the tensor core's operand reads
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.dc_full[h]);
      } else {
        at += d.F;
        if (++q == d.P) {
          q = 0;
          G += kTwGroups;
          place();
        }
      }
      CNN_PHASE(5);
    }
    if constexpr (BWD) {
      // conv bias: sum over the quarter's rows; lane i ends with map m0 + i's
      float v[32];
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        unpack2(gb2[i >> 1], v[i], v[i + 1]);
        v[16 + i] = v[17 + i] = 0.f;
      }
      const float mine = warp_reduce_scatter32(v, lane) * pow2i(-dc_exp);
      const size_t cta = (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * kTwPartB;
      if (lane < 16) part_b[cta + quarter * kTwF + m0 + lane] = mine;
      // subsample filter: taps of row rsub, then the sum of delta_s
      float s5[5], x, yv;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        unpack2(gs2[j], x, yv);
        s5[j] = -(x + yv);
      }
      unpack2(gds2, x, yv);
      s5[4] = x + yv;
#pragma unroll
      for (int m = 4; m <= 16; m <<= 1)
#pragma unroll
        for (int j = 0; j < 5; ++j) s5[j] += __shfl_xor_sync(0xffffffffu, s5[j], m);
      if (lane < 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) sb.red[ew][4 * lane + j] = s5[j];
        if (lane == 0) sb.red[ew][16] = s5[4];
      }
    }
  }
  CNN_PHASE_END(g_phase_clocks_wg);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kTwMmaWarp) tc::tmem_dealloc(tmem_base, 512);
  if (BWD && tid < 17) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kTwEpiWarps; ++w) sum += sb.red[w][tid];
    part_b[(size_t)(blockIdx.y * gridDim.x + blockIdx.x) * kTwPartB + 4 * kTwF + tid] = tid == 16 ? sum / (float)d.S : sum;
  }
}

int wide_tc_max_ctas() { return sm_count(); }

static int wide_tc_grid(const WideDims& d, long n) {
  const long units = (n * ((d.C + 7) / 8) + kTwGroups - 1) / kTwGroups * d.P;
  return (int)(units < sm_count() ? units : sm_count());
}

template <int FL, int PASSES, bool BWD>
static int launch_wide_tc(cnn_wide* w, const WideWork& k, const float* d_images, long n, int ds_blocks, cudaStream_t st) {
  const WideDims& d = w->d;
  const size_t smem = (BWD ? sizeof(TwBwdSmem) : sizeof(TwSmem)) + 128;
  CNN_CUDA(cudaFuncSetAttribute(k_wide_tc<FL, PASSES, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaError_t e = launch_pdl(k_wide_tc<FL, PASSES, BWD>, dim3((unsigned)wide_tc_grid(d, n), (unsigned)(d.F / kTwF)), dim3(kTwThreads), smem, st, d, n,
                             d_images, (const float*)w->d_params, (const float*)k.pixel_max, k.as, (const float*)k.ds,
                             (const float*)k.ds_max, ds_blocks, k.part_g, k.part_b, w->d_status);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_tc launch");
  return CNN_OK;
}

#define CNN_WIDE_TC(BWD, ...)                                                                       \
  do {                                                                                              \
    if (w->conv_mode == 2) {                                                                        \
      if (w->flavour == 1) return launch_wide_tc<1, 3, BWD>(__VA_ARGS__);                           \
      if (w->flavour == 2) return launch_wide_tc<2, 3, BWD>(__VA_ARGS__);                           \
      return launch_wide_tc<0, 3, BWD>(__VA_ARGS__);                                                \
    }                                                                                               \
    if (w->flavour == 1) return launch_wide_tc<1, 1, BWD>(__VA_ARGS__);                             \
    if (w->flavour == 2) return launch_wide_tc<2, 1, BWD>(__VA_ARGS__);                             \
    return launch_wide_tc<0, 1, BWD>(__VA_ARGS__);                                                  \
  } while (0)

int wide_tc_forward(cnn_wide* w, const WideWork& k, const float* d_images, long n, cudaStream_t st) {
  const WideDims& d = w->d;
  cudaError_t e = launch_pdl(k_wide_prep, dim3(kTwPrepBlocks), dim3(256), 0, st, d, reinterpret_cast<const float4*>(d_images),
                             n * d.H * d.H / 4, (const float*)w->d_params, k.pixel_max, k.wf_t);
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_prep launch");
  CNN_WIDE_TC(false, w, k, d_images, n, 0, st);
}

int wide_tc_backward(cnn_wide* w, const WideWork& k, const float* d_images, long n, int ds_blocks, int* ctas, cudaStream_t st) {
  *ctas = wide_tc_grid(w->d, n);
  CNN_WIDE_TC(true, w, k, d_images, n, ds_blocks, st);
}
#undef CNN_WIDE_TC

}  // namespace cnn

#ifdef CNN_PHASE_CLOCKS
// Sums of the SM clock at each stamp for the 24 warps of CTA 0 of the last launch (tuning builds only).
extern "C" int cnn_debug_phase_clocks_wg(long long* out /* [24][16] */) {
  return cudaMemcpyFromSymbol(out, cnn::g_phase_clocks_wg, sizeof(cnn::g_phase_clocks_wg)) == cudaSuccess ? 0 : 2;
}
#endif
