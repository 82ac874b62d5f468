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
// One scale serves all images of a call, so an image may not be so bright that it takes the others' pixels out of fp16's
// range.  What the parts of a scaled pixel lose is 2^-25, and the largest is scaled to 2^14 at least; so an image takes part if its
// largest pixel is at most
//   * 2^(10 - E), 2^E <= the largest weight (with the short sigmoid's factor) < 2^(E + 1): then the scale is 2^(E + 4) at least, and what any
//     pixel loses is below 2^-23 in any pre-activation; or
//   * 2^12 times the smallest (non-zero) largest pixel of an image: then no image's pixels lose more than 2^-27 of its own largest.
// Every other image -- and one with a pixel that is not finite; all images, if a weight or delta is 2^60 or more -- is left out
// by loaders and epilogue and computed in plain fp32 at the end of the kernel, by the CTAs in turn (wide_plain_image; 56x56 with 64 maps: 60 us
// forward, 220 us for a gradient, per CTA and image; 1,024 images of which 1,023 go that way 1.8 ms, against 0.34 ms and the fp32 kernels' 0.69).
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
// Bounds: forward 98 us for 1,024 images (before, with an im2col gather and a subsample kernel of its own: 174 + 152 us), the
// special-function unit two thirds busy; backward 184 us (454 us, which did not have to compute the activations), special-function
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
  float max_of[4][kTwThreads / 32];                                 // largest tap, pixel, subsample delta, by warp; smallest pixel maximum
  float limit;                                                      // images with larger pixels are computed in plain fp32 ...
  int any_plain;                                                    // ... and there are some
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

// Largest and smallest over a warp of values that are not negative (whose bits are in the values' order).
__device__ __forceinline__ float warp_max(float m) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m))); }
__device__ __forceinline__ float warp_min(float m) { return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(m))); }
// Exponent e with 2^e <= v < 2^(e+1), kept where scales built from it stay normal numbers.
__device__ __forceinline__ int exponent_of(float v) {
  const int e = (int)((__float_as_uint(v) >> 23) & 255u) - 127;
  return e > 60 ? 60 : (e < -60 ? -60 : e);
}
// *p += v, not waited for.
__device__ __forceinline__ void red_add(float* p, float v) { asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory"); }
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((127 + e) << 23); }

// What the tensor-core kernels need of a batch beforehand: every image's largest pixel magnitude (not a number, if it has such a
// pixel), and the FC weights in the order in which those kernels have the subsample activations, [window][map] instead of
// [map][window].  A team of threads per image, as many as make its pixels eight loads of 16 bytes per thread at most, all under way at once.
__global__ void __launch_bounds__(256)
k_wide_prep(WideDims d, long n, int team, const float4* images, const float* params, float* __restrict__ img_max, float* __restrict__ wf_t) {
  __shared__ unsigned red[8];
  pdl_launch_dependents();
  pdl_wait();
  const int quads = d.H * d.H / 4, teams = 256 / team, mine = threadIdx.x / team, at = threadIdx.x % team;
  // (from the last block down: the first have the weights)
  for (long b0 = (long)(gridDim.x - 1 - blockIdx.x) * teams; b0 < n; b0 += (long)gridDim.x * teams) {
    const long b = b0 + mine;
    const float4* src = images + (size_t)(b < n ? b : 0) * quads;
    unsigned m = 0;                    // magnitudes compared as integers: what is not a number is above infinity
    for (int i0 = at; i0 < quads; i0 += 8 * team) {
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = src[i0 + j * team < quads ? i0 + j * team : i0];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        m = max(max(m, max(__float_as_uint(v[j].x) & 0x7fffffffu, __float_as_uint(v[j].y) & 0x7fffffffu)),
                max(__float_as_uint(v[j].z) & 0x7fffffffu, __float_as_uint(v[j].w) & 0x7fffffffu));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (team > 32) {
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
      __syncthreads();
      if (at == 0)
        for (int k = 1; k < team / 32; ++k) m = max(m, red[(threadIdx.x >> 5) + k]);
      __syncthreads();
    }
    if (at == 0 && b < n) img_max[b] = __uint_as_float(m);
  }
  const int W = d.P * d.P;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < (long)kOut * d.S; i += (long)gridDim.x * blockDim.x) {
    const int k = (int)(i / d.S), s = (int)(i - (long)k * d.S);
    wf_t[i] = params[d.o_wf + (size_t)k * d.S + (size_t)(s % d.F) * W + s / d.F];
  }
}

// The way out for an image whose pixels do not fit the batch's scale: plain fp32 by all threads of a CTA, for its 64 maps from f0 on.  With
// rolled loops and in line: what it needs of registers and stack, or a call, the hot code pays for (1,024 images: forward 117.7 us without it, 120.3
// this way; a gradient 333.3, 332.0 in line and 333.3 with a call).  Thread = map and every twelfth window of a row of windows, taps from shared
// memory.  Forward: the image's subsample activations as[window][map].  Backward: reads ds[window][map] and adds the image's
// share to the CTA's sums, in a fixed order and their layouts (a filter tap (i, j) goes to x = 0, c = j of D).  The deltas of a row of windows go through
// shared memory, where a thread has a map, a tap row (or the bias) and every other row of deltas.
constexpr int kTwPlainTeams = kTwThreads / kTwF;                    // 12 = 2 halves of 5 tap rows and the bias
constexpr int kTwPlainMaxP = 31;                                    // H = 128
struct TwPlain {
  float tap[25][kTwF];
  float filter[kTwThreads / 32][17];                                // backward only from here on
  alignas(16) float4 dc[kTwPlainMaxP * 4][kTwF];                    // [window column, its row][map]
};
static_assert(sizeof(TwPlain::tap) <= offsetof(TwSmem, bias) && sizeof(TwPlain) <= sizeof(TwBwdSmem), "space for wide_plain_image");

template <int FL, bool BWD>
__device__ __forceinline__ void wide_plain_image(int H, int F, int f0, TwPlain& sm, const float* image, const float* params, float* as_or_ds,
                                              float* part_g, float* part_b) {
  const WideDims d = make_wide_dims(H, F);
  const int tid = threadIdx.x, m = tid % kTwF, team = tid / kTwF;
  __syncthreads();                     // (whatever was in sm has been used)
  for (int e = tid; e < 25 * kTwF; e += kTwThreads) sm.tap[e / kTwF][e % kTwF] = params[d.o_wc + (f0 + e % kTwF) * 25 + e / kTwF];
  __syncthreads();
  const int half = team & 1, row = team >> 1;
  float gs[17], g[5];
#pragma unroll
  for (int t = 0; t < 17; ++t) gs[t] = 0.f;
#pragma unroll
  for (int j = 0; j < 5; ++j) g[j] = 0.f;
  auto pixels = [&](int y, int q, float (&v)[8]) {
    const float4* src = reinterpret_cast<const float4*>(image + y * H + 4 * q);
    const float4 lo = src[0], hi = src[1];
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
    v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  };
#pragma unroll 1
  for (int p = 0; p < d.P; ++p) {
#pragma unroll 1
    for (int q = team; q < d.P; q += kTwPlainTeams) {
      float* at = as_or_ds + (size_t)(p * d.P + q) * F + f0 + m;
      float z = params[d.o_bs];
      const float dl = BWD ? *at : 0.f, dlc = dl / (float)(d.C * d.C), bias = params[d.o_bc + f0 + m];
      gs[16] += dl;
      float a[4][4], v[8];
#pragma unroll
      for (int o = 0; o < 16; ++o) a[o / 4][o % 4] = bias;
#pragma unroll 1
      for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          pixels(4 * p + y + i, q, v);
#pragma unroll
          for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) a[y][x] = fmaf(sm.tap[i * 5 + j][m], v[x + j], a[y][x]);
        }
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        float dc[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const float av = sigmoidf<FL>(a[y][x]), w = params[d.o_ws + 4 * y + x];
          z = fmaf(w, av, z);
          gs[4 * y + x] = fmaf(dl, av, gs[4 * y + x]);
          dc[x] = w * dlc * (av * (1.f - av));
        }
        if (BWD) sm.dc[4 * q + y][m] = make_float4(dc[0], dc[1], dc[2], dc[3]);
      }
      if (!BWD) *at = sigmoidf<FL>(z);
    }
    if (!BWD) continue;
    __syncthreads();
#pragma unroll 1
    for (int e = half; e < 4 * d.P; e += 2) {
      const float4 dc = sm.dc[e][m];
      if (row == 5) {
        g[0] += (dc.x + dc.y) + (dc.z + dc.w);
      } else {
        float v[8];
        pixels(4 * p + e % 4 + row, e / 4, v);
#pragma unroll
        for (int j = 0; j < 5; ++j) g[j] = fmaf(dc.w, v[j + 3], fmaf(dc.z, v[j + 2], fmaf(dc.y, v[j + 1], fmaf(dc.x, v[j], g[j]))));
      }
    }
    __syncthreads();
  }
  if (!BWD) return;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {        // one half after the other: the same addresses
    if (h == half) {
      if (row == 5) part_b[m] += g[0];
      else
#pragma unroll
        for (int j = 0; j < 5; ++j) red_add(part_g + (row * 8 + j) * kTwGradCols + 8 * (m >> 1) + (m & 1), g[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < 17; ++t) {
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) gs[t] += __shfl_xor_sync(0xffffffffu, gs[t], k);
    if ((tid & 31) == 0) sm.filter[tid >> 5][t] = gs[t];
  }
  __syncthreads();
  if (tid < 17) {
    float sum = 0.f;
    for (int k = 0; k < kTwThreads / 32; ++k) sum += sm.filter[k][tid];
    part_b[4 * kTwF + tid] += tid == 16 ? sum / (float)d.S : sum;
  }
}

// FL: sigmoid flavour.  PASSES: 3 or 1.  BWD: false = forward (writes as), true = backward (reads ds, writes the partial gradients).
// as, ds: [image][window][map].  part_g: per CTA (of all map groups) [kTwGradN][256] sums of D; part_b: per CTA [4][64] conv bias
// sums (a row per quarter of the rows) and the 17 subsample-filter sums behind them.  scale_of: of each map group {limit, largest
// pixel within it, largest of all}, from the forward kernel for the backward kernel.
template <int FL, int PASSES, bool BWD>
__global__ void __launch_bounds__(kTwThreads, 1)
k_wide_tc(WideDims d, long n, const float* images, const float* params, const float* img_max,
          float* scale_of, float* __restrict__ as, const float* ds, const float* ds_max, int ds_blocks,
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
  float wmax = 0.f, dmax = 0.f, pmax = 0.f, pmin = INFINITY;       // (pmax: what is not finite counts as infinite)
  for (int i = tid; i < kTwF * 25; i += kTwThreads) {
    const float a = fabsf(kPre * params[d.o_wc + f0 * 25 + i]);
    wmax = (a <= 3.4e38f) ? fmaxf(wmax, a) : INFINITY;
  }
  if (BWD) {
    for (int i = tid; i < ds_blocks; i += kTwThreads) dmax = fmaxf(dmax, ds_max[i]);
  } else {
    for (long b0 = tid; b0 < n; b0 += 4 * kTwThreads) {
      float m[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) m[j] = img_max[b0 + j * kTwThreads < n ? b0 + j * kTwThreads : b0];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        pmax = m[j] <= 3.4e38f ? fmaxf(pmax, m[j]) : INFINITY;
        pmin = m[j] > 0.f ? fminf(pmin, m[j]) : pmin;
      }
    }
  }
  wmax = warp_max(wmax);
  dmax = warp_max(dmax);
  pmax = warp_max(pmax);
  pmin = warp_min(pmin);
  if (lane == 0) {
    sm.max_of[0][warp] = wmax;
    sm.max_of[1][warp] = pmax;
    sm.max_of[2][warp] = dmax;
    sm.max_of[3][warp] = pmin;
  }
  __syncthreads();
  const int mine_at = lane < kTwThreads / 32 ? lane : 0;
  wmax = warp_max(sm.max_of[0][mine_at]);
  dmax = warp_max(sm.max_of[2][mine_at]);
  // The images that take part (see above), and the largest pixel among them.
  constexpr float kHuge = 1152921504606846976.f;                   // 2^60
  float limit, all;
  if (BWD) {
    limit = scale_of[4 * blockIdx.y];
    pmax = scale_of[4 * blockIdx.y + 1];
    all = scale_of[4 * blockIdx.y + 2];
  } else {
    all = pmax = warp_max(sm.max_of[1][mine_at]);
    pmin = warp_min(sm.max_of[3][mine_at]);
    limit = wmax < kHuge ? fminf(fmaxf(pow2i(10 - exponent_of(wmax)), 4096.f * pmin), kHuge) : -1.f;
    if (!(all <= limit)) {
      pmax = 0.f;
      for (long b = tid; b < n; b += kTwThreads) pmax = img_max[b] <= limit ? fmaxf(pmax, img_max[b]) : pmax;
      pmax = warp_max(pmax);
      __syncthreads();
      if (lane == 0) sm.max_of[1][warp] = pmax;
      __syncthreads();
      pmax = warp_max(sm.max_of[1][mine_at]);
    }
    if (blockIdx.x == 0 && tid < 3) scale_of[4 * blockIdx.y + tid] = tid == 0 ? limit : (tid == 1 ? pmax : all);
  }
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
    if (!(dmax < kHuge && ws_max < kHuge)) {
      limit = -1.f;
      dc_exp = 0;
    }
  }
  if (tid == 0) {
    sm.limit = limit;
    sm.any_plain = !(all <= limit);
  }

  // ---- weights: step s holds kernel rows 2 s and 2 s + 1, chunk = kernel row, row = accumulator column -----------
  for (int e = tid; e < 3 * 2 * kTwN; e += kTwThreads) {
    const int i = e / kTwN, col = e % kTwN;
    const int f = 2 * (col >> 3) + (col & 1), x = (col & 7) >> 1;
    float w[5];
#pragma unroll
    for (int t = 0; t < 5; ++t) w[t] = i < 5 && wmax < kHuge ? kPre * params[d.o_wc + (f0 + f) * 25 + (i < 5 ? i : 0) * 5 + t] : 0.f;
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
      if (sm.any_plain) have = have && img_max[have ? b : 0] <= sm.limit;
      src = images + ((size_t)(have ? b : 0) * d.H + (have ? y : 0)) * d.H;
    };
    auto load = [&](int q) {           // (clamped, not conditional: a load under a condition is waited for on the spot)
      v0 = *reinterpret_cast<const float4*>(src + 4 * q);
      v1 = reinterpret_cast<const float4*>(src + 4 * q)[1];
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
    float* at;                       // this lane's window and maps in as / ds; of one that does not take part: the zeros behind ds
    auto place = [&]() {
      const unsigned b = G / (unsigned)gi;
      const int p = (8 * (int)(G - b * (unsigned)gi) + (lane & 7)) >> 2;      // C is a multiple of 4: a window's rows are all in or all out
      live = b < n && p < d.P;
      if (sm.any_plain) live = live && img_max[live ? b : 0] <= sm.limit;
      const size_t window = live ? ((size_t)b * d.P + p) * d.P + q : (BWD ? (size_t)n * d.P * d.P : 0);
      at = (BWD ? const_cast<float*>(ds) : as) + window * d.F + f0 + m0;
    };
    place();
    // Backward: the window's deltas of eight maps, the next eight taken as soon as these are used.
    float4 dlo, dhi;
    if (BWD) {
      dlo = *reinterpret_cast<const float4*>(at);
      dhi = reinterpret_cast<const float4*>(at)[1];
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
            if (ch == 1) dlo = *reinterpret_cast<const float4*>(part ? at : at + 8);
            if (ch == 3) dhi = reinterpret_cast<const float4*>(part ? at : at + 8)[1];
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
  const size_t cta = blockIdx.y * gridDim.x + blockIdx.x;
  if (BWD && tid < 17) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kTwEpiWarps; ++w) sum += sb.red[w][tid];
    part_b[cta * kTwPartB + 4 * kTwF + tid] = tid == 16 ? sum / (float)d.S : sum;
  }
  if (sm.any_plain) {
    const float top = sm.limit;
#pragma unroll 1
    for (long b = blockIdx.x; b < n; b += gridDim.x) {
      if (img_max[b] <= top) continue;
      wide_plain_image<FL, BWD>(d.H, d.F, f0, *reinterpret_cast<TwPlain*>(smem_base), images + (size_t)b * d.H * d.H, params,
                                (BWD ? const_cast<float*>(ds) : as) + (size_t)b * d.P * d.P * d.F, part_g + cta * kTwGradN * kTwGradCols,
                                part_b + cta * kTwPartB);
    }
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
                             d_images, (const float*)w->d_params, (const float*)k.img_max, k.scale_of, k.as, (const float*)k.ds,
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
  int team = 32;
  while (team < 256 && 8 * team < d.H * d.H / 4) team *= 2;
  cudaError_t e = launch_pdl(k_wide_prep, dim3(kTwPrepBlocks), dim3(256), 0, st, d, n, team, reinterpret_cast<const float4*>(d_images),
                             (const float*)w->d_params, k.img_max, k.wf_t);
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
