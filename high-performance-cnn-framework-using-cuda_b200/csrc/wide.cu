// Widened variant of the same topology (benchmark configuration 5): input HxH, F maps of 5x5 (valid) ->
// sigmoid -> ONE shared 4x4/stride-4 filter -> sigmoid -> FC F*P*P -> 10 -> sigmoid, with the
// reference's update rule generalised as in the oracle: divisors (H-4)^2 for the conv gradient and
// bias, F*P*P for the subsample bias (layer.cu:369, 389, 312 with 24 -> H-4 and 6*6*6 -> F*P*P).
// The reference's own kernels cannot run this shape (fixed array types; N * thread_index overflows
// int), so its check is the generalised oracle.
//
// This file is the fp32 SIMT path and the FC layer of all paths.  Between the forward and the backward pass the conv
// activations are kept in HBM (at 56x56 / 64 maps one image's activations are 692 KB, more than an
// SM's shared memory); inference does not write them.  All reductions are fixed-order (no atomics).
#include <cooperative_groups.h>

#include <cstring>
#include <new>
#include <vector>

#include "cluster_exchange.cuh"
#include "wide.cuh"

namespace cg = cooperative_groups;

namespace cnn {

// ---- forward ---------------------------------------------------------------------------------
// Convolution, bias, sigmoid and the subsample layer of one 4x4 window for a group of maps, two maps at a time: thread =
// window (of any image: windows are numbered through the batch), the two maps in the halves of packed fp32 registers.
// The 8x8 patch stays in registers over the pairs (64, beside 32 of accumulators; each pixel copied into both halves: 64 moves for
// 400 packed FMAs), the taps are read from shared memory where they are used: with the taps in registers too 58 instead of 55 us.  (Not with
// unaligned rows where conv activations are stored: kept 198, loaded for each pair 167 us for 333 images of 57x57.)  Bound by the fp32 FMA pipe: 400 FMAs per window and map
// = 40 us for 333 images of 56x56 with 64 maps; 55 us measured (a block per image and 8 maps with one output per thread,
// then the subsample layer from memory: 287 + 53 us).
// Writes the subsample activations and, with STORE, the conv activations (what the backward pass reads; pre-activations
// are never needed again because sigmoid' = a (1 - a)).  Positions outside the windows (C not a multiple of 4) reach
// nothing and are not computed.
constexpr int kWideWinThreads = 128;
constexpr int kWideTapStride = 26;      // 25 tap pairs, padded to an even number for 128-bit loads

// Eight pixels of a patch row; VEC: rows are 16-byte aligned (H a multiple of 4).
template <bool VEC>
__device__ __forceinline__ void load_row8(const float* src, float (&v)[8]) {
  if (VEC) {
    const float4 a = *reinterpret_cast<const float4*>(src), b = reinterpret_cast<const float4*>(src)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = src[c];
  }
}

template <int FLAVOR, bool STORE, bool VEC>
__global__ void __launch_bounds__(kWideWinThreads, 4)
k_wide_conv_s1(WideDims d, long n, int maps_per_block, const float* images, const float* params,
               float* __restrict__ ac, float* __restrict__ as) {
  extern __shared__ __align__(16) float sh[];
  // tap pairs [pair][26][2] | subsample taps, doubled [16][2] | bias pairs [pair][2]   (the first two are read 16 bytes at a time)
  // (the short sigmoid form's factor -log2(e) is folded into taps and bias)
  constexpr float kPre = (FLAVOR == 1) ? -1.4426950408889634f : 1.0f;
  const int f0 = blockIdx.y * maps_per_block;
  const int maps = min(maps_per_block, d.F - f0), pairs = (maps + 1) / 2;
  float* tap = sh;
  float* ws = tap + (maps_per_block + 1) / 2 * kWideTapStride * 2;
  float* bias = ws + 32;
  pdl_launch_dependents();
  pdl_wait();
  for (int i = threadIdx.x; i < pairs * kWideTapStride * 2; i += blockDim.x) {
    const int pr = i / (kWideTapStride * 2), t = (i % (kWideTapStride * 2)) >> 1, f = 2 * pr + (i & 1);
    tap[i] = (t < 25 && f < maps) ? kPre * params[d.o_wc + (f0 + f) * 25 + t] : 0.f;
  }
  for (int i = threadIdx.x; i < pairs * 2; i += blockDim.x) bias[i] = (i < maps) ? kPre * params[d.o_bc + f0 + i] : 0.f;
  if (threadIdx.x < 32) ws[threadIdx.x] = params[d.o_ws + (threadIdx.x >> 1)];
  const float bs = params[d.o_bs];
  __syncthreads();
  const int W = d.P * d.P;
  const long t = (long)blockIdx.x * kWideWinThreads + threadIdx.x;
  if (t >= n * W) return;
  const long b = t / W;
  const int w = (int)(t - b * W), p = w / d.P, q = w - p * d.P;
  const float* src = images + ((size_t)b * d.H + 4 * p) * d.H + 4 * q;
  constexpr bool kKeep = VEC || !STORE;
  float patch[8][8];
  if (kKeep) {
#pragma unroll
    for (int r = 0; r < 8; ++r) load_row8<VEC>(src + r * d.H, patch[r]);
  }
#pragma unroll 1
  for (int pr = 0; pr < pairs; ++pr) {
    if (!kKeep) asm volatile("" : "+l"(src));      // (or the compiler moves the loads out of the loop)
    f32x2 acc[4][4];
    const f32x2* wt = reinterpret_cast<const f32x2*>(tap + pr * kWideTapStride * 2);
    const f32x2 bp = reinterpret_cast<const f32x2*>(bias)[pr];
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[y][x] = bp;
    f32x2 z = pack2(0.f, 0.f);
    const ulonglong2* wsp = reinterpret_cast<const ulonglong2*>(ws);
    const int f = f0 + 2 * pr;
    const bool second = 2 * pr + 1 < maps;
    const size_t ac_at = STORE ? ((size_t)(b * d.F + f) * d.C + 4 * p) * d.C + 4 * q : 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float (&v)[8] = patch[r];
      if (!kKeep) load_row8<VEC>(src + r * d.H, v);
      f32x2 v2[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v2[c] = pack2(v[c], v[c]);
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int i = r - y;                 // tap row
        if (i < 0 || i > 4) continue;
#pragma unroll
        for (int j = 0; j < 5; ++j)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[y][x] = fma2(wt[i * 5 + j], v2[x + j], acc[y][x]);
      }
      // output row r - 4 is complete: its sigmoids (special-function unit) go under the next rows' FMAs
      if (r >= 4) {
        const int y = r - 4;
        float a0[4], a1[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float u0, u1;
          unpack2(acc[y][x], u0, u1);
          if (FLAVOR == 1) {
            a0[x] = rcp_approx(1.0f + exp2f_approx(u0));
            a1[x] = rcp_approx(1.0f + exp2f_approx(u1));
          } else {
            a0[x] = sigmoidf<FLAVOR>(u0);
            a1[x] = sigmoidf<FLAVOR>(u1);
          }
        }
#pragma unroll
        for (int x = 0; x < 4; x += 2) {
          const ulonglong2 w2 = wsp[(4 * y + x) / 2];
          z = fma2(w2.x, pack2(a0[x], a1[x]), z);
          z = fma2(w2.y, pack2(a0[x + 1], a1[x + 1]), z);
        }
        if (STORE) {
          float* dst = ac + ac_at + (size_t)y * d.C;
          float* dst1 = dst + (size_t)d.C * d.C;
          if (VEC) {
            *reinterpret_cast<float4*>(dst) = make_float4(a0[0], a0[1], a0[2], a0[3]);
            if (second) *reinterpret_cast<float4*>(dst1) = make_float4(a1[0], a1[1], a1[2], a1[3]);
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              dst[x] = a0[x];
              if (second) dst1[x] = a1[x];
            }
          }
        }
      }
    }
    float z0, z1;
    unpack2(z, z0, z1);
    as[(size_t)(b * d.F + f) * W + w] = sigmoidf<FLAVOR>(z0 + bs);
    if (second) as[(size_t)(b * d.F + f + 1) * W + w] = sigmoidf<FLAVOR>(z1 + bs);
  }
}

// FC, sigmoid, argmax, makeError, error norm by clusters of kWideFcSlices blocks, each of which adds up one slice of the S
// inputs for the cluster's images; the partial sums meet in the first block's shared memory.  A warp has kWideFcImgs
// images and 8 * 10 sums in registers.  `sets` (1, 2 or 4): groups of images in a block, each of 8 / sets warps that share
// the slice; the groups walk it at the same time, so the weights (433 KB at S = 10,816) come from L2 once for all of them and
// from L1 for the others.  One group is the shortest walk (five or six steps): right while the clusters of one group fit the
// chip at once; four groups have the least traffic.  Bound by L2 latency.
constexpr int kWideFcImgs = 8;
constexpr int kWideFcSlices = 8;
constexpr int kWideFcVals = 96;          // kWideFcImgs * kOut sums, padded to whole warps
constexpr int kWideFcSets = 4;

template <int FLAVOR>
__global__ void __launch_bounds__(256, 2) __cluster_dims__(kWideFcSlices, 1, 1)
k_wide_fc_fwd(WideDims d, long n, int sets, const float* as, const float* wf, const float* params,
              const unsigned* labels, float* __restrict__ out, int* __restrict__ argmax,
              float* __restrict__ delta_f, float* __restrict__ err) {
  __shared__ float red[8][kWideFcVals];
  __shared__ float part[kWideFcSlices][kWideFcSets * kWideFcVals];       // the first block's: one row per slice
  __shared__ float o_s[kWideFcSets * kWideFcImgs][kOut];
  cg::cluster_group cluster = cg::this_cluster();
  const int slice = (int)cluster.block_rank();
  const long b0 = (long)(blockIdx.x / kWideFcSlices) * sets * kWideFcImgs;     // the cluster's images
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int set = warp % sets, parts = 8 / sets, part_of = warp / sets;
  const long first = b0 + set * kWideFcImgs;                                   // the warp's images
  const int imgs = (int)((n - first) < kWideFcImgs ? (n - first) : kWideFcImgs);
  const int s_end = (int)((long)d.S * (slice + 1) / kWideFcSlices);
  f32x2 acc[kWideFcImgs][kOut / 2];
#pragma unroll
  for (int g = 0; g < kWideFcImgs; ++g)
#pragma unroll
    for (int k = 0; k < kOut / 2; ++k) acc[g][k] = pack2(0.f, 0.f);
  pdl_launch_dependents();
  pdl_wait();
  if (imgs > 0) {
    for (int s = (int)((long)d.S * slice / kWideFcSlices) + part_of * 32 + lane; s < s_end; s += parts * 32) {
      f32x2 wv[kOut / 2];
#pragma unroll
      for (int k = 0; k < kOut / 2; ++k) wv[k] = pack2(wf[(size_t)(2 * k) * d.S + s], wf[(size_t)(2 * k + 1) * d.S + s]);
#pragma unroll
      for (int g = 0; g < kWideFcImgs; ++g) {
        const float v = as[(size_t)(first + (g < imgs ? g : 0)) * d.S + s];       // (sums of images past the batch are not used)
        const f32x2 v2 = pack2(v, v);
#pragma unroll
        for (int k = 0; k < kOut / 2; ++k) acc[g][k] = fma2(wv[k], v2, acc[g][k]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kWideFcVals / 32; ++c) {       // 32 sums at a time: lane l ends with sum 32 c + l = image * 10 + k
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const int e = 32 * c + i;
      if (e < kWideFcImgs * kOut) unpack2(acc[e / kOut][(e % kOut) / 2], v[i], v[i + 1]);
      else v[i] = v[i + 1] = 0.f;
    }
    red[warp][32 * c + lane] = warp_reduce_scatter32(v, lane);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < sets * kWideFcVals; e += 256) {
    const int g = e / kWideFcVals, v = e - g * kWideFcVals;
    float z = 0.f;
    for (int ww = g; ww < 8; ww += sets) z += red[ww][v];
    cluster.map_shared_rank(&part[0][0], 0)[slice * (kWideFcSets * kWideFcVals) + e] = z;
  }
  cluster.sync();
  if (slice != 0) return;
  const int total = (int)((n - b0) < sets * kWideFcImgs ? (n - b0) : sets * kWideFcImgs);
  for (int e = threadIdx.x; e < total * kOut; e += 256) {
    const int g = e / kOut, k = e % kOut;
    float z = 0.f;
#pragma unroll
    for (int c = 0; c < kWideFcSlices; ++c) z += part[c][g / kWideFcImgs * kWideFcVals + g % kWideFcImgs * kOut + k];
    const float o = sigmoidf<FLAVOR>(z + params[d.o_bf + k]);
    o_s[g][k] = o;
    const long b = b0 + g;
    if (out) out[(size_t)b * kOut + k] = o;
    if (delta_f) delta_f[(size_t)b * kOut + k] = ((labels[b] == (unsigned)k) ? 1.0f : 0.0f) - o;
  }
  __syncthreads();
  if (threadIdx.x < total) {
    const int g = threadIdx.x;
    const long b = b0 + g;
    int best = 0;
    for (int k = 1; k < kOut; ++k)
      if (o_s[g][best] < o_s[g][k]) best = k;
    if (argmax) argmax[b] = best;
    if (err) {
      float ss = 0.f;
      for (int k = 0; k < kOut; ++k) {
        const float dlt = ((labels[b] == (unsigned)k) ? 1.0f : 0.0f) - o_s[g][k];
        ss += dlt * dlt;
      }
      err[b] = sqrtf(ss);
    }
  }
}

// ---- backward --------------------------------------------------------------------------------
// The FC layer's part of the backward pass in one pass over the subsample activations:
//   delta_s[b][s] = (sum_k Wf[k][s] delta_f[b][k]) * as (1 - as)      (bp_output_s1, bp_preact_s1)
//   G_wf[k][s]    = sum_b delta_f[b][k] as[b][s]                      (bp_weight_f)
// (ds_max, if given: the largest finite |delta_s| of each block.)
// Thread = one s; the batch is cut into kWideFcSplit contiguous slices (blockIdx.y), each of which writes partial sums of
// G_wf that k_wide_reduce adds in order, so the result does not depend on scheduling.  The ten weights and ten sums stay
// in registers, the images' output deltas come from shared memory.  Bound by memory: as in, ds out (88 MB for 1,024 images of
// S = 10,816; two kernels that each read as took 65 us, this one 28 with four
// images' loads under way and about 24 with eight, for which it needs more than the 48 registers that the compiler would take).
constexpr int kWideFcSplit = 16;
constexpr int kWideBpImgs = 64;          // images whose output deltas are staged at a time
constexpr int kWideBpAhead = 8;          // images whose activations are under way at a time

__global__ void __launch_bounds__(128, 6)
k_wide_bp_fc(WideDims d, long n, const float* as, const float* delta_f,
             const float* wf, float* __restrict__ ds, float* __restrict__ part_f, float* __restrict__ ds_max) {
  __shared__ __align__(16) float dlt[kWideBpImgs][12];
  __shared__ float red[4];
  float most = 0.f;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = s < d.S;
  const long b0 = (n * blockIdx.y) / kWideFcSplit, b1 = (n * (blockIdx.y + 1)) / kWideFcSplit;
  f32x2 acc[kOut / 2], wv[kOut / 2];
  pdl_launch_dependents();
  pdl_wait();
#pragma unroll
  for (int k = 0; k < kOut / 2; ++k) {
    acc[k] = pack2(0.f, 0.f);
    wv[k] = live ? pack2(wf[(size_t)(2 * k) * d.S + s], wf[(size_t)(2 * k + 1) * d.S + s]) : pack2(0.f, 0.f);
  }
  for (long c0 = b0; c0 < b1; c0 += kWideBpImgs) {
    const int imgs = (int)((b1 - c0) < kWideBpImgs ? (b1 - c0) : kWideBpImgs);
    __syncthreads();
    for (int i = threadIdx.x; i < imgs * kOut; i += blockDim.x) dlt[i / kOut][i % kOut] = delta_f[c0 * kOut + i];
    __syncthreads();
    if (!live) continue;
    const float* src = as + (size_t)c0 * d.S + s;
    float* dst = ds + (size_t)c0 * d.S + s;
    auto image = [&](int g, float a) {
      const f32x2 a2 = pack2(a, a);
      const ulonglong2 d0 = *reinterpret_cast<const ulonglong2*>(&dlt[g][0]), d1 = *reinterpret_cast<const ulonglong2*>(&dlt[g][4]);
      const f32x2 dk[kOut / 2] = {d0.x, d0.y, d1.x, d1.y, *reinterpret_cast<const f32x2*>(&dlt[g][8])};
      f32x2 sum = mul2(wv[0], dk[0]);
#pragma unroll
      for (int k = 1; k < kOut / 2; ++k) sum = fma2(wv[k], dk[k], sum);
#pragma unroll
      for (int k = 0; k < kOut / 2; ++k) acc[k] = fma2(dk[k], a2, acc[k]);
      float lo, hi;
      unpack2(sum, lo, hi);
      const float v = (lo + hi) * a * (1.f - a);
      dst[(size_t)g * d.S] = v;
      most = fabsf(v) <= 3.4e38f ? fmaxf(most, fabsf(v)) : most;
    };
    float ahead[kWideBpAhead];               // (spelt out: a load may not move in front of the stores before it)
    int g = 0;
    for (; g + kWideBpAhead <= imgs; g += kWideBpAhead) {
#pragma unroll
      for (int i = 0; i < kWideBpAhead; ++i) ahead[i] = src[(size_t)(g + i) * d.S];
#pragma unroll
      for (int i = 0; i < kWideBpAhead; ++i) image(g + i, ahead[i]);
    }
    if (g < imgs) {
#pragma unroll
      for (int i = 0; i < kWideBpAhead - 1; ++i) ahead[i] = src[(size_t)(g + i < imgs ? g + i : g) * d.S];
#pragma unroll
      for (int i = 0; i < kWideBpAhead - 1; ++i)
        if (g + i < imgs) image(g + i, ahead[i]);
    }
  }
  if (ds_max) {                            // tensor-core path
    if (blockIdx.y == 0 && s < d.F) ds[(size_t)n * d.S + s] = 0.f;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, m));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = most;
    __syncthreads();
    if (threadIdx.x == 0) ds_max[blockIdx.y * gridDim.x + blockIdx.x] = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  }
  if (!live) return;
#pragma unroll
  for (int k = 0; k < kOut / 2; ++k) {
    float lo, hi;
    unpack2(acc[k], lo, hi);
    part_f[((size_t)blockIdx.y * kOut + 2 * k) * d.S + s] = lo;
    part_f[((size_t)blockIdx.y * kOut + 2 * k + 1) * d.S + s] = hi;
  }
}

// Conv deltas, conv weight and bias gradient and subsample-filter gradient of two maps for a slice of the batch (fp32 SIMT):
//   dc = Ws[i][j] * delta_s * a (1 - a) / (C*C)       (bp_output_s1, bp_preact_c1)
//   G_wc[f][u][v] = sum dc[y][x] * image[y + u][x + v], G_bc[f] = sum dc, G_ws[i][j] = sum delta_s * a
// Thread = one window after another of the slice's images, the two maps in the halves of packed registers, all sums in
// registers until the end: the deltas never exist in memory.  The patch goes by row by row as in the forward kernel.
// Bound by the FMA pipe (400 FMAs per window and map for the weight gradient alone); 333 images of 56x56 with 64 maps: 134 us,
// 154 us with the rows' loads wherever the compiler put them; 128 images: 62 us before that (a kernel that wrote the deltas and one that read them back per map and image: 108 + 200 us).
// Partial rows: part_c[slice][F][26], part_s[slice * pairs + pair][17].
template <bool VEC>
__global__ void __launch_bounds__(kWideWinThreads, 3)
k_wide_grad_win(WideDims d, long n, const float* images, const float* ac,
                const float* ds, const float* params, float* __restrict__ part_c,
                float* __restrict__ part_s) {
  __shared__ __align__(16) f32x2 ws2[16];
  __shared__ float red[kWideWinThreads / 32][3][32];
  const int f = 2 * blockIdx.x, slices = gridDim.y;
  const bool second = f + 1 < d.F;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float inv_c = 1.0f / (float)(d.C * d.C), inv_s = 1.0f / (float)d.S;
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x < 16) ws2[threadIdx.x] = pack2(params[d.o_ws + threadIdx.x], params[d.o_ws + threadIdx.x]);
  __syncthreads();
  const int W = d.P * d.P;
  const size_t CC = (size_t)d.C * d.C;
  const long b0 = (n * blockIdx.y) / slices, b1 = (n * (blockIdx.y + 1)) / slices;
  const long units = (b1 - b0) * W;
  f32x2 acc[26];
  float gs[17];
#pragma unroll
  for (int t = 0; t < 26; ++t) acc[t] = pack2(0.f, 0.f);
#pragma unroll
  for (int t = 0; t < 17; ++t) gs[t] = 0.f;
  const f32x2 one2 = pack2(1.f, 1.f), minus2 = pack2(-1.f, -1.f);
#pragma unroll 1
  for (long t = threadIdx.x; t < units; t += kWideWinThreads) {
    const long bl = t / W;
    const int w = (int)(t - bl * W), p = w / d.P, q = w - p * d.P;
    const long b = b0 + bl;
    const float dl0 = ds[(size_t)(b * d.F + f) * W + w], dl1 = second ? ds[(size_t)(b * d.F + f + 1) * W + w] : 0.f;
    const f32x2 dl2 = pack2(dl0 * inv_c, dl1 * inv_c);
    const float* a_at = ac + (size_t)(b * d.F + f) * CC + (size_t)(4 * p) * d.C + 4 * q;
    const size_t to_second = second ? CC : 0;      // (without a second map the first is read twice: its delta is zero)
    f32x2 dc[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      float a0[4], a1[4];
      const float* s0 = a_at + (size_t)y * d.C;
      if (VEC) {
        const float4 u = *reinterpret_cast<const float4*>(s0), v = *reinterpret_cast<const float4*>(s0 + to_second);
        a0[0] = u.x; a0[1] = u.y; a0[2] = u.z; a0[3] = u.w;
        a1[0] = v.x; a1[1] = v.y; a1[2] = v.z; a1[3] = v.w;
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x) { a0[x] = s0[x]; a1[x] = s0[to_second + x]; }
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const f32x2 a2 = pack2(a0[x], a1[x]);
        gs[4 * y + x] = fmaf(dl1, a1[x], fmaf(dl0, a0[x], gs[4 * y + x]));
        dc[y][x] = mul2(mul2(ws2[4 * y + x], dl2), mul2(a2, fma2(a2, minus2, one2)));
        acc[25] = add2(acc[25], dc[y][x]);
      }
    }
    gs[16] += (dl0 + dl1) * inv_s;
    const float* src = images + ((size_t)b * d.H + 4 * p) * d.H + 4 * q;
    asm volatile("" : "+l"(src));        // the rows' loads begin here, not beside the activations': 100 bytes of spills per unit less
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float v[8];
      load_row8<VEC>(src + r * d.H, v);
      f32x2 v2[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v2[c] = pack2(v[c], v[c]);
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int i = r - y;                 // tap row
        if (i < 0 || i > 4) continue;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int j = 0; j < 5; ++j) acc[i * 5 + j] = fma2(dc[y][x], v2[x + j], acc[i * 5 + j]);
      }
    }
  }
  // block sums, in a fixed order: lane t ends with value t of map f, of map f + 1 and of the filter gradient
  float v0[32], v1[32], vs[32];
#pragma unroll
  for (int t = 0; t < 32; ++t) {
    v0[t] = v1[t] = 0.f;
    if (t < 26) unpack2(acc[t < 26 ? t : 0], v0[t], v1[t]);
    vs[t] = t < 17 ? gs[t < 17 ? t : 0] : 0.f;
  }
  red[warp][0][lane] = warp_reduce_scatter32(v0, lane);
  red[warp][1][lane] = warp_reduce_scatter32(v1, lane);
  red[warp][2][lane] = warp_reduce_scatter32(vs, lane);
  __syncthreads();
  if (threadIdx.x < 96) {
    const int m = warp;
    const float sum = (red[0][m][lane] + red[1][m][lane]) + (red[2][m][lane] + red[3][m][lane]);
    if (m < 2) {
      if (lane < 26 && f + m < d.F) part_c[((size_t)blockIdx.y * d.F + f + m) * 26 + lane] = sum;
    } else if (lane < 17) {
      part_s[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 17 + lane] = sum;
    }
  }
}

// The gradient vector from the partials; G[n_params+1] = sum of the per-image error norms; padding zeroed; everything added in a
// fixed order.  Blocks, in this order:
//   value_blocks: a warp per output value (SIMT path: conv filters; both: conv biases, subsample filter and bias, FC biases,
//     error): lane l adds rows l, l + 32, ..., then the lanes are combined by a fixed shuffle tree.  (One thread per value
//     walking up to 1,024 rows took 79 us of a 1.3 ms step.)
//   filter_blocks, tensor-core path: (map group, kernel row i, four maps).  The CTAs' D[(x, f)][(i, c)] are added first, 16 bytes
//     per thread and CTA, eight threads taking every eighth CTA; then G[f][i][j] = sum_x D[(x, f)][(i, x + j)].
//   the rest: a thread per FC weight adds the batch slices; on the tensor-core path the sums are in [window][map] order.
// (Four blocks per SM = 64 registers: left to itself the compiler takes 32, and a thread's loads wait for one another.
// A tensor-core step of 1,024 images 359 -> 343 us, of 128 images 92.9 -> 77.0; a fp32 step of 128 images 110 -> 108 us.)
template <bool TC>
__global__ void __launch_bounds__(256, 4)
k_wide_reduce(WideDims d, long n, long rows_c, long rows_s, const float* part_c, const float* part_s,
              const float* part_f, const float* delta_f, const float* err, int value_blocks,
              int filter_blocks, float* __restrict__ G) {
  constexpr int kSlices = 8, kTile = 8 * 16;      // of a filter block: CTA slices; 8 c x 16 columns (x, f)
  __shared__ __align__(16) float sums[TC ? kSlices : 1][TC ? kTile : 1];
  pdl_launch_dependents();
  pdl_wait();
  const int block = blockIdx.x;
  if (block >= value_blocks + filter_blocks) {
    const long i = (long)(block - value_blocks - filter_blocks) * blockDim.x + threadIdx.x;   // over kOut * S
    if (i < (long)kOut * d.S) {
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < kWideFcSplit; ++c) sum += part_f[(size_t)c * kOut * d.S + i];
      if (TC) {
        const int k = (int)(i / d.S), s = (int)(i - (long)k * d.S), w = s / d.F;
        G[d.o_wf + (size_t)k * d.S + (size_t)(s - w * d.F) * (d.P * d.P) + w] = sum;
      } else {
        G[d.o_wf + i] = sum;
      }
    }
    return;
  }
  if (TC && block >= value_blocks) {
    const int e = block - value_blocks, quads = kTwF / 4, group = e / (5 * quads), i = e / quads % 5, fq = e % quads;   // maps 4 fq ..
    const int tile = threadIdx.x % (kTile / 4), slice = threadIdx.x / (kTile / 4);         // tile: four columns of row c = tile / 4
    const float* src = part_c + (size_t)(group * rows_c) * kTwGradN * kTwGradCols + (size_t)(i * 8 + tile / 4) * kTwGradCols + 16 * fq +
                       4 * (tile % 4);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (long c = slice; c < rows_c; c += kSlices) {
      const float4 v = *reinterpret_cast<const float4*>(src + (size_t)c * kTwGradN * kTwGradCols);
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    *reinterpret_cast<float4*>(&sums[slice][tile * 4]) = sum;
    __syncthreads();
    if (threadIdx.x < 20) {
      const int m = threadIdx.x / 5, j = threadIdx.x % 5;
      float g = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int at = (x + j) * 16 + 8 * (m >> 1) + 2 * x + (m & 1);
        for (int c = 0; c < kSlices; ++c) g += sums[c][at];
      }
      G[d.o_wc + (group * kTwF + 4 * fq + m) * 25 + i * 5 + j] = g;
    }
    return;
  }
  const int t = block * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int n_c = TC ? d.F : d.F * 26;
  if (t > n_c + 17 + kOut) return;
  const float* src;
  long rows, stride;
  if (t < n_c && TC) { src = part_s + (size_t)(t / kTwF) * rows_c * kTwPartB + t % kTwF; rows = 4 * rows_c; stride = kTwPartB; }
  else if (t < n_c) { src = part_c + t; rows = rows_c; stride = n_c; }
  else if (t < n_c + 17) { src = part_s + (TC ? 4 * kTwF : 0) + (t - n_c); rows = rows_s; stride = TC ? kTwPartB : 17; }
  else if (t < n_c + 17 + kOut) { src = delta_f + (t - n_c - 17); rows = n; stride = kOut; }
  else { src = err; rows = n; stride = 1; }
  float sum = 0.f;
  if (TC && t < n_c) {        // a CTA's conv bias sums: a row for each quarter of its rows
#pragma unroll 4
    for (long b = lane; b < rows; b += 32) sum += src[(size_t)(b >> 2) * stride + (b & 3) * kTwF];
  } else {
#pragma unroll 4
    for (long b = lane; b < rows; b += 32) sum += src[(size_t)b * stride];
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
  if (lane != 0) return;
  if (t < n_c) {
    const int f = TC ? t : t / 26, k = TC ? 25 : t % 26;
    if (k < 25) G[d.o_wc + f * 25 + k] = sum; else G[d.o_bc + f] = sum;
  } else if (t < n_c + 17) {
    const int k = t - n_c;
    if (k < 16) G[d.o_ws + k] = sum; else G[d.o_bs] = sum;
  } else if (t < n_c + 17 + kOut) {
    G[d.o_bf + t - n_c - 17] = sum;
  } else {
    G[d.n_params + 1] = sum;
    G[d.n_params] = 0.f;
    for (int i = d.n_params + 2; i < d.n_padded; ++i) G[i] = 0.f;
  }
}

__global__ void k_wide_update(int n_params, float* __restrict__ params, const float* G, float scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_params) params[i] = fmaf(scale, G[i], params[i]);
}

}  // namespace cnn

using namespace cnn;

// Which kernels a call takes.  The tensor-core path wants whole groups of 64 maps, rows of whole 16-byte pieces (one thread loads
// eight pixels of a row as two float4) and windows without a remainder; everything else runs on the fp32 path.
static bool wide_on_tc(const cnn_wide* w, const float* d_images) {
  return w->conv_mode > 0 && wide_tc_supported(w->d) && (reinterpret_cast<uintptr_t>(d_images) & 15u) == 0;
}

// Slices of the batch for k_wide_grad_win: three blocks per SM and map pair would fit; two waves of them.
static long wide_grad_slices(const WideDims& d, long n) {
  const int pairs = (d.F + 1) / 2;
  const long slices = (6L * sm_count() + pairs - 1) / pairs;
  return slices < n ? slices : n;
}

static int wide_bp_fc_blocks(const WideDims& d) { return (d.S + 127) / 128; }

// Lays the arena out for a call, growing it if it is too small.  One allocation (a cudaMalloc costs about 0.36 ms) of what this
// call's kernels use: inference keeps no deltas, the tensor-core path no conv activations (2.8 GB for 4,096 images of 56x56 / 64).
static int wide_reserve(cnn_wide* w, long n, bool training, bool tc, WideWork& k) {
  const WideDims& d = w->d;
  for (int pass = 0; pass < 2; ++pass) {          // sizes, then pointers
    size_t at = 0;
    auto take = [&](float*& p, size_t floats) {
      p = pass ? w->arena + at : nullptr;
      at += (floats + 63) & ~(size_t)63;
    };
    take(k.as, (size_t)d.S * n);
    if (tc) {
      take(k.img_max, n);
      take(k.scale_of, 4 * (d.F / kTwF));
      take(k.wf_t, (size_t)kOut * d.S);
    }
    if (training) {
      take(k.ds, (size_t)d.S * n + (tc ? d.F : 0));         // (behind it zeros for windows that do not exist: k_wide_bp_fc)
      take(k.delta_f, (size_t)kOut * n);
      take(k.err, n);
      take(k.part_f, (size_t)kWideFcSplit * kOut * d.S);
      if (tc) {
        const size_t ctas = (size_t)wide_tc_max_ctas() * (d.F / kTwF);
        take(k.ds_max, (size_t)wide_bp_fc_blocks(d) * kWideFcSplit);
        take(k.part_g, ctas * kTwGradN * kTwGradCols);
        take(k.part_b, ctas * kTwPartB);
      } else {
        const size_t slices = wide_grad_slices(d, n);
        take(k.ac, (size_t)d.F * d.C * d.C * n);
        take(k.part_c, slices * d.F * 26);
        take(k.part_s, slices * ((d.F + 1) / 2) * 17);
      }
    }
    k.floats = at;
    if (!pass && at > w->arena_floats) {
      cudaFree(w->arena);
      w->arena = nullptr;
      w->arena_floats = 0;
      CNN_CUDA(cudaMalloc(&w->arena, sizeof(float) * at));
      w->arena_floats = at;
    }
  }
  return CNN_OK;
}

template <int FL, bool STORE, bool VEC>
static int launch_conv_s1(cnn_wide* w, const WideWork& k, const float* d_images, long n, cudaStream_t st) {
  const WideDims& d = w->d;
  const long blocks = (n * d.P * d.P + kWideWinThreads - 1) / kWideWinThreads;
  // Maps per block: as many as keep four waves of four blocks per SM, so that a block's set-up (its taps) is shared and the
  // last wave is short; at least two (a packed pair).
  int maps = d.F;
  while (maps > 2 && blocks * ((d.F + maps - 1) / maps) < 16L * sm_count()) maps = (maps / 2 + 1) / 2 * 2;
  const int pairs = (maps + 1) / 2;
  const size_t smem = sizeof(float) * (size_t)(pairs * (kWideTapStride * 2 + 2) + 32);
  CNN_CUDA(cudaFuncSetAttribute(k_wide_conv_s1<FL, STORE, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaError_t e = launch_pdl(k_wide_conv_s1<FL, STORE, VEC>, dim3((unsigned)blocks, (unsigned)((d.F + maps - 1) / maps)),
                             dim3(kWideWinThreads), smem, st, d, n, maps, d_images, (const float*)w->d_params, k.ac, k.as);
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_conv_s1 launch");
  return CNN_OK;
}

template <int FL>
static int wide_forward_impl(cnn_wide* w, const WideWork& k, bool tc, const float* d_images, const unsigned* d_labels, long n,
                             float* d_out, int* d_argmax, bool training, cudaStream_t st) {
  const WideDims& d = w->d;
  int rc;
  if (tc) {
    rc = wide_tc_forward(w, k, d_images, n, st);
  } else {
    const bool vec = d.H % 4 == 0 && (reinterpret_cast<uintptr_t>(d_images) & 15u) == 0;
    if (vec) rc = training ? launch_conv_s1<FL, true, true>(w, k, d_images, n, st) : launch_conv_s1<FL, false, true>(w, k, d_images, n, st);
    else rc = training ? launch_conv_s1<FL, true, false>(w, k, d_images, n, st) : launch_conv_s1<FL, false, false>(w, k, d_images, n, st);
  }
  if (rc != CNN_OK) return rc;
  // Groups of images per FC cluster: as few as let all clusters be on the chip at once (two blocks per SM).
  int sets = 1;
  while (sets < kWideFcSets && (n + kWideFcImgs * sets - 1) / (kWideFcImgs * sets) * kWideFcSlices > 2L * sm_count()) sets *= 2;
  const long clusters = (n + kWideFcImgs * sets - 1) / (kWideFcImgs * sets);
  cudaError_t e = launch_pdl(k_wide_fc_fwd<FL>, dim3((unsigned)(clusters * kWideFcSlices)), dim3(256), 0, st, d, n, sets,
                             (const float*)k.as, (const float*)(tc ? k.wf_t : w->d_params + d.o_wf), (const float*)w->d_params, d_labels,
                             d_out, d_argmax, training ? k.delta_f : nullptr, training ? k.err : nullptr);
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_fc_fwd launch");
  return CNN_OK;
}

static int wide_forward_dispatch(cnn_wide* w, const WideWork& k, bool tc, const float* d_images, const unsigned* d_labels, long n,
                                 float* d_out, int* d_argmax, bool training, cudaStream_t st) {
  switch (w->flavour) {
    case 1: return wide_forward_impl<1>(w, k, tc, d_images, d_labels, n, d_out, d_argmax, training, st);
    case 2: return wide_forward_impl<2>(w, k, tc, d_images, d_labels, n, d_out, d_argmax, training, st);
    default: return wide_forward_impl<0>(w, k, tc, d_images, d_labels, n, d_out, d_argmax, training, st);
  }
}

extern "C" {

int cnn_wide_param_count(int H, int F) {
  if (H < 8 || F < 1) return -1;
  return make_wide_dims(H, F).n_params;
}

int cnn_wide_create(int H, int F, cnn_wide** out) {
  CNN_REQUIRE(out != nullptr, "cnn_wide_create: out is NULL");
  *out = nullptr;
  CNN_REQUIRE(H >= 8 && H <= 128 && F >= 1 && F <= 1024, "cnn_wide_create: unsupported shape");
  cnn_wide* w = new (std::nothrow) cnn_wide();
  CNN_REQUIRE(w != nullptr, "cnn_wide_create: out of host memory");
  w->d = make_wide_dims(H, F);
  cudaError_t e = cudaMalloc(&w->d_params, sizeof(float) * w->d.n_padded);
  if (e == cudaSuccess) e = cudaMemset(w->d_params, 0, sizeof(float) * w->d.n_padded);
  if (e == cudaSuccess) e = cudaMalloc(&w->d_status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(w->d_status, 0, sizeof(int));
  if (e == cudaSuccess) e = cudaDeviceSynchronize();  // memsets are asynchronous to the host
  if (e != cudaSuccess) { delete w; return cuda_fail(e, "cnn_wide_create"); }
  *out = w;
  return CNN_OK;
}

int cnn_wide_destroy(cnn_wide* w) {
  if (!w) return CNN_OK;
  cudaFree(w->d_params);
  cudaFree(w->arena);
  cudaFree(w->d_status);
  delete w;
  return CNN_OK;
}

int cnn_wide_set_params(cnn_wide* w, const float* h_params) {
  CNN_REQUIRE(w && h_params, "cnn_wide_set_params: NULL argument");
  // same ordering as cnn_net_set_params: nothing in flight reads the old values, and the upload
  // has landed before a launch on a non-blocking stream
  CNN_CUDA(cudaDeviceSynchronize());
  CNN_CUDA(cudaMemcpy(w->d_params, h_params, sizeof(float) * w->d.n_params, cudaMemcpyHostToDevice));
  CNN_CUDA(cudaDeviceSynchronize());
  return CNN_OK;
}

int cnn_wide_get_params(cnn_wide* w, float* h_params) {
  CNN_REQUIRE(w && h_params, "cnn_wide_get_params: NULL argument");
  CNN_CUDA(cudaMemcpy(h_params, w->d_params, sizeof(float) * w->d.n_params, cudaMemcpyDeviceToHost));
  return CNN_OK;
}

int cnn_wide_set_option(cnn_wide* w, const char* key, int value) {
  CNN_REQUIRE(w && key, "cnn_wide_set_option: NULL argument");
  if (std::strcmp(key, "fast_sigmoid") == 0) { w->flavour = (value == 2) ? 2 : (value ? 1 : 0); return CNN_OK; }
  if (std::strcmp(key, "conv") == 0) {
    CNN_REQUIRE(value >= 0 && value <= 2, "cnn_wide_set_option: conv is 0 (fp32 SIMT), 1 (tensor cores, one fp16 pass) or 2 (three passes)");
    w->conv_mode = value;
    return CNN_OK;
  }
  set_error("cnn_wide_set_option: unknown option '%s'", key);
  return CNN_ERR_INVALID;
}

int cnn_wide_status(cnn_wide* w, int* status) {
  CNN_REQUIRE(w && status, "cnn_wide_status: NULL argument");
  CNN_CUDA(cudaDeviceSynchronize());
  CNN_CUDA(cudaMemcpy(status, w->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  if (*status != 0) {
    set_error("a bounded device-side wait ran out (status %d)", *status);
    int zero = 0;
    CNN_CUDA(cudaMemcpy(w->d_status, &zero, sizeof(int), cudaMemcpyHostToDevice));
    return CNN_ERR_TIMEOUT;
  }
  return CNN_OK;
}

int cnn_wide_forward(cnn_wide* w, const float* d_images, long n, float* d_out, int* d_argmax, void* stream) {
  CNN_REQUIRE(w != nullptr, "cnn_wide_forward: NULL handle");
  CNN_REQUIRE(n >= 0 && n <= 65535L * 32, "cnn_wide_forward: bad image count");
  if (n == 0) return CNN_OK;
  CNN_REQUIRE(d_images != nullptr, "cnn_wide_forward: NULL images");
  WideWork k;
  const bool tc = wide_on_tc(w, d_images);
  int rc = wide_reserve(w, n, false, tc, k);
  if (rc != CNN_OK) return rc;
  return wide_forward_dispatch(w, k, tc, d_images, nullptr, n, d_out, d_argmax, false, as_stream(stream));
}

int cnn_wide_grad_batch(cnn_wide* w, const float* d_images, const unsigned int* d_labels, long n, float* d_grad,
                        void* stream) {
  CNN_REQUIRE(w && d_grad, "cnn_wide_grad_batch: NULL argument");
  CNN_REQUIRE(n >= 0 && n <= 65535L * 32, "cnn_wide_grad_batch: bad image count");
  cudaStream_t st = as_stream(stream);
  const WideDims& d = w->d;
  if (n == 0) {
    CNN_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(float) * d.n_padded, st));
    return CNN_OK;
  }
  CNN_REQUIRE(d_images && d_labels, "cnn_wide_grad_batch: NULL images or labels");
  WideWork k;
  const bool tc = wide_on_tc(w, d_images);
  int rc = wide_reserve(w, n, true, tc, k);
  if (rc != CNN_OK) return rc;
  if ((rc = wide_forward_dispatch(w, k, tc, d_images, d_labels, n, nullptr, nullptr, true, st)) != CNN_OK) return rc;
  const int bp_blocks = wide_bp_fc_blocks(d);
  cudaError_t e = launch_pdl(k_wide_bp_fc, dim3(bp_blocks, kWideFcSplit), dim3(128), 0, st, d, n, (const float*)k.as,
                             (const float*)k.delta_f, (const float*)(tc ? k.wf_t : w->d_params + d.o_wf), k.ds, k.part_f, k.ds_max);
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_bp_fc launch");
  const int weight_blocks = (kOut * d.S + 255) / 256;
  if (tc) {
    int ctas = 0;
    if ((rc = wide_tc_backward(w, k, d_images, n, bp_blocks * kWideFcSplit, &ctas, st)) != CNN_OK) return rc;
    const int groups = d.F / kTwF, filter_blocks = groups * 5 * (kTwF / 4), value_blocks = (d.F + 18 + kOut + 7) / 8;
    e = launch_pdl(k_wide_reduce<true>, dim3(value_blocks + filter_blocks + weight_blocks), dim3(256), 0, st, d, n, (long)ctas,
                   (long)ctas * groups, (const float*)k.part_g, (const float*)k.part_b, (const float*)k.part_f, (const float*)k.delta_f,
                   (const float*)k.err, value_blocks, filter_blocks, d_grad);
  } else {
    const int pairs = (d.F + 1) / 2;
    const long slices = wide_grad_slices(d, n);
    const bool vec = d.H % 4 == 0 && (reinterpret_cast<uintptr_t>(d_images) & 15u) == 0;
    e = launch_pdl(vec ? k_wide_grad_win<true> : k_wide_grad_win<false>, dim3(pairs, (unsigned)slices), dim3(kWideWinThreads), 0, st, d, n,
                   d_images, (const float*)k.ac, (const float*)k.ds, (const float*)w->d_params, k.part_c, k.part_s);
    if (e != cudaSuccess) return cuda_fail(e, "k_wide_grad_win launch");
    const int value_blocks = (d.F * 26 + 18 + kOut + 7) / 8;       // one warp each
    e = launch_pdl(k_wide_reduce<false>, dim3(value_blocks + weight_blocks), dim3(256), 0, st, d, n, slices, slices * pairs,
                   (const float*)k.part_c, (const float*)k.part_s, (const float*)k.part_f, (const float*)k.delta_f, (const float*)k.err,
                   value_blocks, 0, d_grad);
  }
  if (e != cudaSuccess) return cuda_fail(e, "wide backward launch");
  return CNN_OK;
}

int cnn_wide_apply_update(cnn_wide* w, const float* d_grad, float scale, void* stream) {
  CNN_REQUIRE(w && d_grad, "cnn_wide_apply_update: NULL argument");
  k_wide_update<<<(w->d.n_params + 255) / 256, 256, 0, as_stream(stream)>>>(w->d.n_params, w->d_params, d_grad, scale);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_wide_update launch");
  return CNN_OK;
}

}  // extern "C"
