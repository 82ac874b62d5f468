// Fused forward + backward kernels.
//
//  * k_grad_partials  -- minibatch mode: every block walks a strided subset of the batch, keeps the
//    gradient of its images in registers, reduces it inside the block with warp shuffles / shared
//    memory (no atomics) and writes one partial row; k_reduce_rows adds the rows in fixed order and
//    optionally applies the update.  Replaces, per image, forward_pass + makeError + back_pass
//    (main.cu:67-88, 147-153, 99-119: 17 memsets, 23 launches, one blocking norm).
//  * k_train_persample -- the reference's learn() loop (main.cu:125-170) as ONE persistent block
//    (the fallback; the default is the six-CTA cluster kernel of persample_cluster8.cu, this one
//    is selected with the "persample_kernel" option set to 0 and needs no cluster launch):
//    parameters live in shared memory, one SGD step per image in file order, same update
//    semantics (output delta without sigmoid derivative, every backward product from pre-update
//    weights, biases and weights stepped by dt), per-epoch mean of ||delta_f||_2, early stop.
//
// Decomposition of k_train_persample: thread (f, window) owns one 4x4 subsample window of one feature
// map: 16 conv outputs (400 FMA forward, 400 FMA for the conv weight gradient), so conv
// activations, their deltas and the 25 weight-gradient partials stay in registers.  216 threads
// are live in a 224-thread block.
//
// Arithmetic notes (all within fp32 rounding of the reference, which itself sums with atomics in
// a run-dependent order): sums use FMA; the per-term divisions by 576 / 216 of layer.cu:379, 397,
// 320 become one multiplication of the delta by the reciprocal constant.
#include <type_traits>

#include "net.cuh"

namespace cnn {

constexpr int kTrThreads = 224;  // 7 warps; threads 216..223 carry zeros
constexpr int kTrWarps = kTrThreads / 32;
constexpr int kRedStride = 27;   // 25 conv-weight partials + 1 conv-bias partial + pad (odd stride)

struct TrSmem {
  float img[2][kImg];
  float wc[kF][28];
  float bc[8];
  float ws[16];
  float bs[4];
  float wf[kOut][kS];
  float bf[12];
  float fc_part[kTrWarps][12];
  float delta_f[12];
  float red_c[kS][kRedStride];
  float red_s[kTrWarps][20];
  unsigned long long full[2];
  int flag[4];
};

__device__ __forceinline__ void load_params_to_smem(TrSmem& sm, const float* params, int tid) {
  for (int i = tid; i < kF * 28; i += kTrThreads) {
    const int f = i / 28, t = i % 28;
    sm.wc[f][t] = (t < 25) ? params[kOffWc + f * 25 + t] : 0.f;
  }
  if (tid < kF) sm.bc[tid] = params[kOffBc + tid];
  if (tid < 16) sm.ws[tid] = params[kOffWs + tid];
  if (tid == 0) sm.bs[0] = params[kOffBs];
  for (int i = tid; i < kOut * kS; i += kTrThreads) sm.wf[i / kS][i % kS] = params[kOffWf + i];
  if (tid < kOut) sm.bf[tid] = params[kOffBf + tid];
}

// Per-thread state of one image's forward pass.
struct FwdRegs {
  float patch[8][8];
  float a[4][4];   // conv activations of the window
  float as;        // subsample activation
  float wfv[kOut]; // this thread's column of the FC weights
};

template <int FAST>
__device__ __forceinline__ void thread_forward(const TrSmem& sm, const float* img, int f, int p, int q,
                                               int s, bool live, FwdRegs& r, float (&pk)[kOut]) {
  if (live) {
    const float* base = img + (4 * p) * kH + 4 * q;
#pragma unroll
    for (int y = 0; y < 8; ++y) {
      const float4 lo = *reinterpret_cast<const float4*>(base + y * kH);
      const float4 hi = *reinterpret_cast<const float4*>(base + y * kH + 4);
      r.patch[y][0] = lo.x; r.patch[y][1] = lo.y; r.patch[y][2] = lo.z; r.patch[y][3] = lo.w;
      r.patch[y][4] = hi.x; r.patch[y][5] = hi.y; r.patch[y][6] = hi.z; r.patch[y][7] = hi.w;
    }
  } else {
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
      for (int x = 0; x < 8; ++x) r.patch[y][x] = 0.f;
  }
  float wr[28];
#pragma unroll
  for (int t = 0; t < 7; ++t) {
    const float4 v = *reinterpret_cast<const float4*>(&sm.wc[f][4 * t]);
    wr[4 * t] = v.x; wr[4 * t + 1] = v.y; wr[4 * t + 2] = v.z; wr[4 * t + 3] = v.w;
  }
  const float b = sm.bc[f];
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < 5; ++j)
#pragma unroll
        for (int i = 0; i < 5; ++i) acc = fmaf(wr[i * 5 + j], r.patch[y + i][x + j], acc);
      r.a[y][x] = sigmoidf<FAST>(acc + b);
    }
  float zs = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) zs = fmaf(sm.ws[i * 4 + j], r.a[i][j], zs);
  r.as = sigmoidf<FAST>(zs + sm.bs[0]);
#pragma unroll
  for (int k = 0; k < kOut; ++k) {
    r.wfv[k] = sm.wf[k][s];
    pk[k] = live ? r.wfv[k] * r.as : 0.f;
  }
}

// Sum each of n values over the 32 lanes (butterfly); every lane ends with the total.
template <int N>
__device__ __forceinline__ void warp_sum(float (&v)[N]) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], m);
}

// Backward of one image for this thread, given delta_f in shared memory.  Produces the thread's
// contributions: gws[16] (subsample weight), gbs (subsample bias term), gwc[25] (conv weight, already
// divided by 576), gbc (conv bias term, divided by 576), and das-derived delta_s.
__device__ __forceinline__ void thread_backward(const TrSmem& sm, const FwdRegs& r, bool live,
                                                const float (&df)[kOut], float& delta_s,
                                                float (&gws)[16], float (&gwc)[25], float& gbc) {
  float das = 0.f;
#pragma unroll
  for (int k = 0; k < kOut; ++k) das = fmaf(r.wfv[k], df[k], das);
  delta_s = live ? das * r.as * (1.f - r.as) : 0.f;
  float dc[4][4];
  const float inv_c = 1.0f / (float)(kC * kC);
  gbc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      gws[i * 4 + j] = delta_s * r.a[i][j];
      const float dac = sm.ws[i * 4 + j] * delta_s;
      const float d = dac * r.a[i][j] * (1.f - r.a[i][j]);
      dc[i][j] = d * inv_c;
      gbc += dc[i][j];
    }
#pragma unroll
  for (int u = 0; u < 5; ++u)
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      float acc = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) acc = fmaf(dc[y][x], r.patch[y + u][x + v], acc);
      gwc[u * 5 + v] = acc;
    }
}

// After the call lane l holds, for the index scatter8_index(l), the sum of v[index] over the lanes that agree with it in bit 0
// (lane bits 4, 3 and 2 pick the index, bit 1 is summed last; lanes that differ in bit 1 hold the same sum).
__device__ __forceinline__ float reduce_scatter8(float (&v)[8], int lane) {
#pragma unroll
  for (int keep = 4; keep >= 1; keep >>= 1) {
    const int mask = keep << 2;          // 16, 8, 4
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < keep; ++i) {
      const float send = upper ? v[i] : v[i + keep], stay = upper ? v[i + keep] : v[i];
      v[i] = stay + __shfl_xor_sync(0xffffffffu, send, mask);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 2);
}
__device__ __forceinline__ int scatter8_index(int lane) { return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1); }

// ----------------------------------------------------------------------------------------------
// Minibatch gradient: one partial row per block.
// Row layout (kRowStride floats): arena-ordered gradient [0, 2343), zero padding, and at
// kRowErr the sum over the block's images of ||delta_f||_2.
//
// One or two teams of seven warps per block, an image each at a time.  Thread (window, map pair, half) of a team owns two
// rows of a 4x4 subsample window for two maps, which sit in the halves of packed fp32 registers: 8 x 2 conv outputs on a
// 6x8 patch (200 packed FMAs forward, 200 for the conv weight gradient), half of the window's ten FC terms.  One barrier
// per image: the FC sums of the team's warps meet in shared memory, and every warp computes the output layer for itself.
// The gradient of a team's images stays in registers (26 pairs of conv taps and bias, five pairs of FC weights, eight
// subsample taps) until the block's reduction at the end (shuffles and shared memory, fixed order, no atomics).
//
// Batches of up to 2,047 images; k_grad_left below does what grad_tc.cu leaves.  Small batches are a chain of latencies, large ones are bound by the FMA pipe (852 cycles
// of it per warp and image; 318 us for 60,000 images).  Measured: a step of 256 images in a training loop 15.4 -> 8.8 us (of which the
// parameters 0.7, forward 1.9, backward 1.5, this kernel's reduction 1.2, the row sums 1.2 and the two hand-overs 1.5 us),
// the gradient of 60,000 images 1,030 -> 643 us.  (Before: a thread per window and map, scalar, two blocks of seven warps per SM at 128 registers
// with the patch and all gradient terms in registers, two barriers per image, a row per image up to 296; then, until 9.5 us, taps from shared
// memory for every image and patch loads that took two turns each.)
// ----------------------------------------------------------------------------------------------
constexpr int kGrThreads = 224;                 // threads of a team: 216 with work
constexpr int kGrWarps = kGrThreads / 32;
constexpr int kGrStages = 3;                    // image buffers of a team
constexpr int kGrRed = 27;                      // pairs per thread in the reduction: 25 taps + bias, padded to an odd number

template <int TEAMS>
struct GrSmem {
  alignas(16) float img[TEAMS][kGrStages][kImg];
  alignas(16) float ws[16];
  alignas(16) f32x2 red[TEAMS * kS][kGrRed];    // conv gradient of every thread
  alignas(8) float wf[kOut][36][kF];            // FC weights as [k][window][map]
  alignas(8) float wc[25][kF];                  // taps as [tap][map]
  alignas(8) float bc[8];
  float bs[4], bf[12];
  float part[TEAMS][2][kGrWarps][12];           // FC sums of a warp, by parity of the turn: outputs 0..4 at 0..4, 5..9 at 6..10
  float red_s[TEAMS * kGrWarps][20];            // subsample-filter gradient of a warp: 16 taps and the bias term
  float red_f[kS][kOut];                        // two teams: FC gradient of the second
  float red_b[TEAMS][12];                       // FC bias gradient and error sum of a team
  unsigned long long full[TEAMS][kGrStages];
};

// Barrier of one team's threads.
template <int TEAMS>
__device__ __forceinline__ void team_sync(int team) {
  if (TEAMS == 1) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kGrThreads) : "memory");
}

// The images of one team, by turn.  Those of a batch go round the teams of all blocks.
struct BatchImages {
  const float* images;
  const unsigned* labels;
  long n, first, step;
  __device__ bool has(int i) const { return first + i * step < n; }
  __device__ long number(int i) const { return first + i * step; }
};
// What the tensor-core kernel has left of a share (`images` and `labels` are the share's): listed images of the tiles that it left out, then those from `from` on.
template <int TEAMS>
struct LeftImages {
  const float* images;
  const unsigned* labels;
  int n, team, listed, from;
  const int* tile;
  __device__ bool has(int i) const { return team + i * TEAMS < n; }
  __device__ long number(int i) const {
    const int im = team + i * TEAMS;
    if (listed == 0) return from + im;
    return im < listed ? kGradTile * tile[im / kGradTile] + im % kGradTile : from + (im - listed);
  }
};

template <int TEAMS, class Images>
__device__ __forceinline__ void copy_image(GrSmem<TEAMS>& sm, int team, const Images& src, int i) {
  if (!src.has(i)) return;
  unsigned long long* bar = &sm.full[team][i % kGrStages];
  mbar_expect_tx(bar, kImg * sizeof(float));
  bulk_g2s(&sm.img[team][i % kGrStages][0], src.images + src.number(i) * kImg, kImg * sizeof(float), bar);
}

template <int TEAMS>
__device__ __forceinline__ void init_image_barriers(GrSmem<TEAMS>& sm, int team) {
  for (int s = 0; s < kGrStages; ++s) mbar_init(&sm.full[team][s], 1);
  mbar_fence_init();
}

// A thread's share of the parameters: every load is under way before the first of them is stored (one L2 latency, not one per
// group of loads: 2.4 -> 0.75 us of a step).
template <int FAST, int TEAMS>
struct ParamShare {
  const float *of_fc, *of_small;
  float wf[kOut / TEAMS], small;
  __device__ __forceinline__ ParamShare(const float* params, int team, int tid)
      : of_fc(params + kOffWf + team * (kOut / TEAMS) * kS + (tid < kS ? tid : 0)),
        of_small(params + (tid < kOffWf ? tid : kOffBf + (tid - kOffWf < kOut ? tid - kOffWf : 0))) {}
  __device__ __forceinline__ void load(int team) {
#pragma unroll
    for (int k = 0; k < kOut / TEAMS; ++k) wf[k] = of_fc[k * kS];
    if (team == 0) small = *of_small;
  }
  __device__ __forceinline__ void store(GrSmem<TEAMS>& sm, int team, int tid) const {
    constexpr float kPre = (FAST == 1) ? -1.4426950408889634f : 1.0f;   // the short sigmoid form's factor, folded into the conv weights
    const int k0 = team * (kOut / TEAMS);
    if (tid < kS) {
#pragma unroll
      for (int k = 0; k < kOut / TEAMS; ++k) sm.wf[k0 + k][tid % 36][tid / 36] = wf[k];
    }
    if (team == 0) {
      if (tid < kOffBc) sm.wc[tid % 25][tid / 25] = kPre * small;
      else if (tid < kOffWs) sm.bc[tid - kOffBc] = kPre * small;
      else if (tid < kOffBs) sm.ws[tid - kOffWs] = small;
      else if (tid == kOffBs) sm.bs[0] = small;
      else if (tid < kOffWf + kOut) sm.bf[tid - kOffWf] = small;
    }
  }
};

// The work of a thread: half of window w's outputs (two rows) of a map pair.  (The eight idle threads shadow thread 0 and add zeros.)
struct ThreadWindow {
  int half, pr, w, patch;
  __device__ __forceinline__ explicit ThreadWindow(int tid) {
    half = tid & 1;
    const int unit = (tid < kS ? tid : 0) >> 1;
    // Eight neighbouring threads, four windows, read 16 bytes each of rows of seven at a time: (4 p + 6 half + q) mod 8 is the bank group.  Of
    // twelve windows (two rows) four with columns 0, 1, 4, 5 of the first row, four of the second, and columns 2, 3 of both ask eight different ones
    // (in the windows' own order every load took two turns: a third of this kernel's shared-memory cycles).
    const int twelve = unit % 36 / 12, quad = unit % 12 / 4, in_quad = unit % 4;
    const int p = 2 * twelve + (quad < 2 ? quad : in_quad >> 1), q = quad < 2 ? in_quad + (in_quad & 2) : 2 + (in_quad & 1);
    pr = unit / 36;
    w = 6 * p + q;
    patch = (4 * p + 2 * half) * kH + 4 * q;
  }
};

// Gradient of both teams' images (the first kGrStages of each are on their way) into the block's row, or added to what is there.
// ONCE: no team has more than one image (one team never has).  Then the gradient's registers are free during the forward pass and hold the taps (which two teams
// otherwise read from shared memory as they go: a quarter of a small batch's shared-memory cycles).
template <int FAST, int TEAMS, bool ONCE, class Images>
__device__ __forceinline__ void grad_images(GrSmem<TEAMS>& sm, const Images& src, const ThreadWindow& at, int team, int tid, float* row, bool add, int* status) {
  const int warp = tid >> 5, lane = threadIdx.x & 31;
  const bool live = tid < kS;
  const int half = at.half, pr = at.pr, w = at.w, patch_at = at.patch;

  f32x2 wt[ONCE ? 25 : 1];
  if (ONCE) {
#pragma unroll
    for (int t = 0; t < 25; ++t) wt[ONCE ? t : 0] = *reinterpret_cast<const f32x2*>(&sm.wc[t][2 * pr]);
  }

  f32x2 g[26], gf[5];
  float gs[8], g_bs = 0.f, g_bf = 0.f, err = 0.f;
#pragma unroll
  for (int t = 0; t < 26; ++t) g[t] = pack2(0.f, 0.f);
#pragma unroll
  for (int t = 0; t < 5; ++t) gf[t] = pack2(0.f, 0.f);
#pragma unroll
  for (int t = 0; t < 8; ++t) gs[t] = 0.f;
  const f32x2 one2 = pack2(1.f, 1.f), minus2 = pack2(-1.f, -1.f);
  const float inv_c = 1.0f / (float)(kC * kC);

  bool gave_up = false;
  for (int it = 0; src.has(it); ++it) {
    unsigned label = 0;
    if (lane < kOut) label = src.labels[src.number(it)];
    mbar_wait_bounded(&sm.full[team][it % kGrStages], (unsigned)(it / kGrStages) & 1u, status, gave_up);
    const float* patch = &sm.img[team][it % kGrStages][0] + patch_at;

    // ---- forward ------------------------------------------------------------------------------
    f32x2 a[2][4];
    {
      const f32x2 bias2 = *reinterpret_cast<const f32x2*>(&sm.bc[2 * pr]);
#pragma unroll
      for (int x = 0; x < 4; ++x) a[0][x] = a[1][x] = bias2;
    }
#pragma unroll
    for (int r = 0; r < 6; ++r) {          // patch rows: eight pixels, each in both halves of a register pair
      const float4 lo = *reinterpret_cast<const float4*>(patch + r * kH), hi = *reinterpret_cast<const float4*>(patch + r * kH + 4);
      const f32x2 v[8] = {pack2(lo.x, lo.x), pack2(lo.y, lo.y), pack2(lo.z, lo.z), pack2(lo.w, lo.w),
                          pack2(hi.x, hi.x), pack2(hi.y, hi.y), pack2(hi.z, hi.z), pack2(hi.w, hi.w)};
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int i = r - y;               // tap row
        if (i < 0 || i > 4) continue;
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          const f32x2 tap = ONCE ? wt[ONCE ? i * 5 + j : 0] : *reinterpret_cast<const f32x2*>(&sm.wc[i * 5 + j][2 * pr]);
#pragma unroll
          for (int x = 0; x < 4; ++x) a[y][x] = fma2(tap, v[x + j], a[y][x]);
        }
      }
    }
    f32x2 zy[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float4 wrow = *reinterpret_cast<const float4*>(&sm.ws[4 * (2 * half + y)]);
      const float ws[4] = {wrow.x, wrow.y, wrow.z, wrow.w};
      zy[y] = pack2(0.f, 0.f);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float u0, u1;
        unpack2(a[y][x], u0, u1);
        a[y][x] = (FAST == 1) ? pack2(rcp_approx(1.0f + exp2f_approx(u0)), rcp_approx(1.0f + exp2f_approx(u1)))
                              : pack2(sigmoidf<FAST>(u0), sigmoidf<FAST>(u1));
        zy[y] = fma2(pack2(ws[x], ws[x]), a[y][x], zy[y]);
      }
    }
    float z0, z1;
    unpack2(add2(zy[0], zy[1]), z0, z1);
    z0 += __shfl_xor_sync(0xffffffffu, z0, 1);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 1);
    const float as0 = live ? sigmoidf<FAST>(z0 + sm.bs[0]) : 0.f, as1 = live ? sigmoidf<FAST>(z1 + sm.bs[0]) : 0.f;
    // FC: output 5 half + j of this window and pair, added over the warp (lane bits 4, 3 and 2 pick one of eight values)
    float v[8];
    float2 wk[5];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = 0.f;
      if (j < 5) {
        wk[j] = *reinterpret_cast<const float2*>(&sm.wf[5 * half + j][w][2 * pr]);
        v[j] = fmaf(wk[j].x, as0, wk[j].y * as1);
      }
    }
    float (&part)[kGrWarps][12] = sm.part[team][it & 1];
    const float mine = reduce_scatter8(v, lane);
    const int idx = scatter8_index(lane);
    if ((lane & 2) == 0 && idx < 5) part[warp][6 * half + idx] = mine;
    team_sync<TEAMS>(team);       // the team's sums are in shared memory; every thread is done with the previous image
    if (!ONCE && tid == 0 && it > 0) copy_image(sm, team, src, it + kGrStages - 1);

    // ---- output layer on lanes 0..9 of every warp -------------------------------------------------
    float delta = 0.f;
    if (lane < kOut) {
      float z = 0.f;
#pragma unroll
      for (int ww = 0; ww < kGrWarps; ++ww) z += part[ww][lane < 5 ? lane : lane + 1];
      const float o = sigmoidf<FAST>(z + sm.bf[lane]);
      delta = ((label == (unsigned)lane) ? 1.0f : 0.0f) - o;       // makeError
    }
    if (warp == 0) {
      g_bf += delta;
      float sq = delta * delta;                                    // zero on lanes >= 10
#pragma unroll
      for (int m = 8; m > 0; m >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, m);
      err += sqrtf(sq);                                            // (lane 0's is used)
    }

    // ---- backward -------------------------------------------------------------------------------
    float das0 = 0.f, das1 = 0.f;
    const f32x2 as2 = pack2(as0, as1);
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const float d = __shfl_sync(0xffffffffu, delta, 5 * half + j);
      das0 = fmaf(wk[j].x, d, das0);
      das1 = fmaf(wk[j].y, d, das1);
      gf[j] = fma2(pack2(d, d), as2, gf[j]);
    }
    das0 += __shfl_xor_sync(0xffffffffu, das0, 1);
    das1 += __shfl_xor_sync(0xffffffffu, das1, 1);
    const float ds0 = das0 * as0 * (1.f - as0), ds1 = das1 * as1 * (1.f - as1);      // zero in idle threads (as = 0)
    if (half == 0) g_bs += ds0 + ds1;
    const f32x2 dsc = pack2(ds0 * inv_c, ds1 * inv_c);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float4 wrow = *reinterpret_cast<const float4*>(&sm.ws[4 * (2 * half + y)]);
      const float ws[4] = {wrow.x, wrow.y, wrow.z, wrow.w};
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float a0, a1;
        unpack2(a[y][x], a0, a1);
        gs[4 * y + x] = fmaf(ds1, a1, fmaf(ds0, a0, gs[4 * y + x]));
        a[y][x] = mul2(mul2(pack2(ws[x], ws[x]), dsc), mul2(a[y][x], fma2(a[y][x], minus2, one2)));    // the conv delta / 576
        g[25] = add2(g[25], a[y][x]);
      }
    }
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const float4 lo = *reinterpret_cast<const float4*>(patch + r * kH), hi = *reinterpret_cast<const float4*>(patch + r * kH + 4);
      const f32x2 u[8] = {pack2(lo.x, lo.x), pack2(lo.y, lo.y), pack2(lo.z, lo.z), pack2(lo.w, lo.w),
                          pack2(hi.x, hi.x), pack2(hi.y, hi.y), pack2(hi.z, hi.z), pack2(hi.w, hi.w)};
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int i = r - y;               // tap row
        if (i < 0 || i > 4) continue;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int j = 0; j < 5; ++j) g[i * 5 + j] = fma2(a[y][x], u[x + j], g[i * 5 + j]);
      }
    }
    if (ONCE) break;
  }

  // ---- block-level reduction, fixed order ----------------------------------------------------
  auto put = [&](float* dst, float v) { *dst = add ? *dst + v : v; };
  if (live) {
#pragma unroll
    for (int t = 0; t < 26; ++t) sm.red[team * kS + tid][t] = g[t];
  }
  {
    const float mine = reduce_scatter8(gs, lane);
    if ((lane & 2) == 0) sm.red_s[team * kGrWarps + warp][8 * half + scatter8_index(lane)] = mine;
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) g_bs += __shfl_xor_sync(0xffffffffu, g_bs, m);
    if (lane == 0) sm.red_s[team * kGrWarps + warp][16] = g_bs * (1.0f / (float)kS);
  }
  if (warp == 0 && lane < kOut) sm.red_b[team][lane] = g_bf;
  if (tid == 0) sm.red_b[team][10] = err;
  if (TEAMS == 2 && team == 1 && live) {
#pragma unroll
    for (int j = 0; j < 5; ++j) unpack2(gf[j], sm.red_f[tid][2 * j], sm.red_f[tid][2 * j + 1]);
  }
  __syncthreads();
  if (team == 0 && live) {
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      float f0, f1;
      unpack2(gf[j], f0, f1);
      if (TEAMS == 2) { f0 += sm.red_f[tid][2 * j]; f1 += sm.red_f[tid][2 * j + 1]; }
      float* dst = row + kOffWf + (5 * half + j) * kS + 2 * pr * 36 + w;
      put(dst, f0);
      put(dst + 36, f1);
    }
  }
  // conv taps and biases: 78 pair columns, 2 TEAMS neighbouring threads each, 36 rows per thread
  constexpr int kPer = 2 * TEAMS;
  const unsigned group = __ballot_sync(0xffffffffu, threadIdx.x < 3 * 26 * kPer);
  if (threadIdx.x < 3 * 26 * kPer) {        // (whole warps or none of the shuffled groups: 3 * 26 * kPer is a multiple of kPer)
    const int col = threadIdx.x / kPer, part = threadIdx.x % kPer;
    const int cp = col / 26, t = col % 26;
    const int r0 = (part / 2) * kS + cp * 72 + (part % 2) * 36;      // 72 threads of a team share a pair
    f32x2 s0 = pack2(0.f, 0.f), s1 = s0, s2 = s0, s3 = s0;
#pragma unroll
    for (int r = 0; r < 36; r += 4) {
      s0 = add2(s0, sm.red[r0 + r][t]);
      s1 = add2(s1, sm.red[r0 + r + 1][t]);
      s2 = add2(s2, sm.red[r0 + r + 2][t]);
      s3 = add2(s3, sm.red[r0 + r + 3][t]);
    }
    float lo, hi;
    unpack2(add2(add2(s0, s1), add2(s2, s3)), lo, hi);
#pragma unroll
    for (int m = kPer / 2; m > 0; m >>= 1) {
      lo += __shfl_xor_sync(group, lo, m);
      hi += __shfl_xor_sync(group, hi, m);
    }
    if (part == 0) {
      float* dst = t < 25 ? row + kOffWc + 2 * cp * 25 + t : row + kOffBc + 2 * cp;
      put(dst, lo);
      put(dst + (t < 25 ? 25 : 1), hi);
    }
  } else if (threadIdx.x >= kGrThreads * TEAMS - 32) {      // the last warp: subsample filter and bias, FC biases, error sum, padding
    if (lane < 17) {
      float sum = 0.f;
#pragma unroll
      for (int ww = 0; ww < TEAMS * kGrWarps; ++ww) sum += sm.red_s[ww][lane];
      put(row + (lane < 16 ? kOffWs + lane : kOffBs), sum);
    } else if (lane < 28) {
      const float sum = TEAMS == 2 ? sm.red_b[0][lane - 17] + sm.red_b[1][lane - 17] : sm.red_b[0][lane - 17];
      put(row + (lane < 27 ? kOffBf + lane - 17 : kRowErr), sum);
    }
    // zero the padding so that reductions and collectives over the padded row stay finite
    for (int i = kNParams + lane; i < kRowStride; i += 32)
      if (i != kRowErr) row[i] = 0.f;
  }
}

// The looping kernel gets 128 registers, what 512 threads would have: with the 144 that it could get it is slower (2,048 images 30.1 us instead of 29.0;
// with 120 and fewer what is spilled costs more, 60,000 images 652 us and up instead of 643).
template <int FAST, int TEAMS, bool ONCE>
__global__ void __launch_bounds__(ONCE ? kGrThreads * TEAMS : 512, 1)
k_grad_partials(const float* images, const unsigned* labels, long n,
                const float* params, float* __restrict__ rows, int* __restrict__ status, int chained) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  GrSmem<TEAMS>& sm = *reinterpret_cast<GrSmem<TEAMS>*>(smem_raw);
  const int team = TEAMS == 1 ? 0 : threadIdx.x / kGrThreads, tid = threadIdx.x - team * kGrThreads;
  const BatchImages src = {images, labels, n, (long)blockIdx.x + (long)team * gridDim.x, (long)TEAMS * gridDim.x};
  // Where everything lies is worked out in the shadow of the kernel before: behind the wait it took 0.2 us of every step (256 images 9.12 -> 8.85 us).
  const ThreadWindow window(tid);
  float* const row = rows + (size_t)blockIdx.x * kRowStride;
  ParamShare<FAST, TEAMS> share(params, team, tid);
  if (chained) pdl_launch_dependents();
  if (tid == 0) {
    init_image_barriers(sm, team);
    // In a training loop the kernel before this one is the previous step's reduce + update kernel, which does not touch
    // the images: their copies may leave while it still runs.  Whatever wrote the images is complete by then, because the loop's
    // first gradient kernel (the one that is not chained) lets its successors start only behind its own wait; kernels that
    // triggered before their waits could otherwise all start while the writer still runs.
    if (chained)
      for (int i = 0; i < kGrStages; ++i) copy_image(sm, team, src, i);
  }
  pdl_wait();      // the parameters (and the row buffer this kernel writes at its end) belong to the predecessor until here
  if (!chained) pdl_launch_dependents();
  if (tid == 0 && !chained)
    for (int i = 0; i < kGrStages; ++i) copy_image(sm, team, src, i);
  share.load(team);
  share.store(sm, team, tid);
  __syncthreads();
  grad_images<FAST, TEAMS, ONCE>(sm, src, window, team, tid, row, false, status);
}

// What the tensor-core kernel (grad_tc.cu) has left, added to the rows that it wrote.  A block takes the share that is next in the queue of those with
// something left, as a rule before that kernel is complete (an SM is free for this block because one of its blocks has finished), else, and for good if there
// is none, when it is.  So shares that are left as a whole are under way beside the others' tiles, and a batch without a byte image takes 4 us longer than
// on k_grad_partials (7 to 23 us when this kernel waited for the other's end and wrote rows of its own).  Parameters and images may be read before the wait: the kernel before this
// one writes neither, and lets this one start only when whatever did is complete.
template <int FAST>
__global__ void __launch_bounds__(512, 1)
k_grad_left(const float* images, const unsigned* labels, GradShares shares,
            const float* params, float* __restrict__ rows, int* __restrict__ status, GradLeft* left, int* pushed) {
  constexpr int TEAMS = 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  GrSmem<TEAMS>& sm = *reinterpret_cast<GrSmem<TEAMS>*>(smem_raw);
  __shared__ int next;
  const int team = threadIdx.x / kGrThreads, tid = threadIdx.x - team * kGrThreads;
  ParamShare<FAST, TEAMS> share(params, team, tid);
  share.load(team);
  if (tid == 0) init_image_barriers(sm, team);
  auto take = [&] {
    if (threadIdx.x == 0) {
      int b;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(b) : "l"(&left[blockIdx.x].next) : "memory");
      next = b;
    }
    __syncthreads();
    return next - 1;
  };
  int b = take();
  if (b < 0) {
    pdl_wait();
    __syncthreads();      // (everybody has looked)
    b = take();
  }
  pdl_launch_dependents();
  if (b >= 0) {
    const long img0 = shares.first(b);
    const GradLeft& mine = left[b];
    const int imgs = shares.size(b), skips = mine.skips, from = mine.from;
    int listed = 0;
    if (skips > 0) {
      const int last = kGradTile * (mine.tile[skips - 1] + 1);      // (the share's last tile may be short)
      listed = kGradTile * skips - (last > imgs ? last - imgs : 0);
    }
    const LeftImages<TEAMS> src = {images + img0 * kImg, labels + img0, listed + imgs - from, team, listed, from, mine.tile};
    if (tid == 0)
      for (int i = 0; i < kGrStages; ++i) copy_image(sm, team, src, i);
    share.store(sm, team, tid);
    __syncthreads();
    grad_images<FAST, TEAMS, false>(sm, src, ThreadWindow(tid), team, tid, rows + (size_t)b * kRowStride, mine.written != 0, status);
    if (threadIdx.x == 0) left[blockIdx.x].next = 0;
    pdl_wait();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *pushed = 0;      // behind the wait: all blocks have pushed what they push
}

// G[i] = sum over rows (fixed order: thirty-two interleaved row groups, then a fixed tree over the
// groups) and, if params is given, params[i] += scale * G[i].  Element kRowErr carries the error sum;
// if mean_err is given, *mean_err += err_scale * that sum.  Block: 1,024 threads = 32 columns x 32 groups.
// (The data-parallel exchange kernel adds a rank's rows in exactly this order.)
constexpr int kRedGroups = 32;

__global__ void __launch_bounds__(32 * kRedGroups)
k_reduce_rows(const float* rows, int n_rows, float* __restrict__ G,
              float* __restrict__ params, float scale, float* __restrict__ mean_err, float err_scale) {
  __shared__ float part[kRedGroups][33];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  pdl_launch_dependents();   // the next step's gradient kernel may set itself up now
  pdl_wait();                // the rows are complete
  float acc = 0.f, p_old = 0.f;
  if (col < kRowStride) {
    if (params && g == 0 && col < kNParams) p_old = params[col];      // under the row loads
    acc = sum_rows<kRedGroups>(rows, n_rows, col, g);
  }
  part[g][lane] = acc;
  __syncthreads();
  if (g == 0 && col < kRowStride) {
    float q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      q[i] = (part[4 * i][lane] + part[4 * i + 1][lane]) + (part[4 * i + 2][lane] + part[4 * i + 3][lane]);
    const float total = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
    if (G) G[col] = total;
    if (params && col < kNParams) params[col] = fmaf(scale, total, p_old);
    if (mean_err && col == kRowErr) *mean_err += err_scale * total;
  }
}

__global__ void k_apply_update(float* __restrict__ params, const float* G, float scale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (i < kNParams) params[i] = fmaf(scale, G[i], params[i]);
}

// ----------------------------------------------------------------------------------------------
// Per-sample SGD, one persistent block.
// ----------------------------------------------------------------------------------------------
template <int FAST>
__global__ void __launch_bounds__(kTrThreads, 1)
k_train_persample(const float* images, const unsigned* labels, long n,
                  int epochs, float dt, float threshold, float* __restrict__ params,
                  float* __restrict__ mean_err, int* __restrict__ epochs_run, int* __restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TrSmem& sm = *reinterpret_cast<TrSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool live = tid < kS;
  const int s = live ? tid : kS - 1;
  const int f = s / 36, w = s % 36, p = w / 6, q = w % 6;

  load_params_to_smem(sm, params, tid);
  if (tid == 0) {
    mbar_init(&sm.full[0], 1);
    mbar_init(&sm.full[1], 1);
    mbar_fence_init();
    sm.flag[0] = 0;
  }
  __syncthreads();

  const long total = (long)epochs * n;
  auto issue = [&](int stage, long step) {
    mbar_expect_tx(&sm.full[stage], kImg * sizeof(float));
    bulk_g2s(&sm.img[stage][0], images + (step % n) * kImg, kImg * sizeof(float), &sm.full[stage]);
  };
  if (tid == 0) {
    if (total > 0) issue(0, 0);
    if (total > 1) issue(1, 1);
  }

  bool gave_up = false;
  float err = 0.f;  // thread 0: running sum of the epoch, a float like main.cu:130
  int done_epochs = 0;
  unsigned next_label = 0;
  if (warp == 0 && lane < kOut && total > 0) next_label = labels[0];

  long step = 0;
  for (int e = 0; e < epochs; ++e) {
    for (long i = 0; i < n; ++i, ++step) {
      const int stage = (int)(step & 1);
      mbar_wait_bounded(&sm.full[stage], (unsigned)(step >> 1) & 1u, status, gave_up);
      const unsigned label = next_label;
      if (warp == 0 && lane < kOut && step + 1 < total) next_label = labels[(step + 1) % n];

      FwdRegs r;
      float pk[kOut];
      thread_forward<FAST>(sm, &sm.img[stage][0], f, p, q, s, live, r, pk);
      warp_sum(pk);
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < kOut; ++k) sm.fc_part[warp][k] = pk[k];
      }
      __syncthreads();  // (A)
      if (tid == 0 && step + 2 < total) issue(stage, step + 2);
      if (warp == 0) {
        float d = 0.f;
        if (lane < kOut) {
          float z = 0.f;
#pragma unroll
          for (int ww = 0; ww < kTrWarps; ++ww) z += sm.fc_part[ww][lane];
          z += sm.bf[lane];
          const float o = sigmoidf<FAST>(z);
          d = ((label == (unsigned)lane) ? 1.0f : 0.0f) - o;  // makeError
          sm.delta_f[lane] = d;
          sm.bf[lane] = fmaf(dt, d, sm.bf[lane]);              // bp_bias_f
        }
        float sq = d * d;
#pragma unroll
        for (int m = 8; m > 0; m >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, m);
        if (lane == 0) err += sqrtf(sq);                        // the norm of main.cu:153-154
      }
      __syncthreads();  // (B)
      float df[kOut];
#pragma unroll
      for (int k = 0; k < kOut; ++k) df[k] = sm.delta_f[k];
      float delta_s, gws[16], gwc[25], gbc;
      thread_backward(sm, r, live, df, delta_s, gws, gwc, gbc);
      if (live) {
        // bp_weight_f then apply_grad on this thread's own column of the FC weights.
#pragma unroll
        for (int k = 0; k < kOut; ++k) sm.wf[k][s] = fmaf(dt, df[k] * r.as, r.wfv[k]);
#pragma unroll
        for (int i = 0; i < 25; ++i) sm.red_c[s][i] = gwc[i];
        sm.red_c[s][25] = gbc;
      }
      {
        float v[17];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = gws[i];
        v[16] = delta_s * (1.0f / (float)kS);
        warp_sum(v);
        if (lane == 0) {
#pragma unroll
          for (int i = 0; i < 17; ++i) sm.red_s[warp][i] = v[i];
        }
      }
      __syncthreads();  // (C) all backward reads of ws / wc are done; partials visible
      if (tid < kF * 26) {
        const int ff = tid / 26, t = tid % 26;
        float sum = 0.f;
#pragma unroll 6
        for (int ww = 0; ww < 36; ++ww) sum += sm.red_c[ff * 36 + ww][t];
        if (t < 25) sm.wc[ff][t] = fmaf(dt, sum, sm.wc[ff][t]);  // apply_grad (c1)
        else sm.bc[ff] = fmaf(dt, sum, sm.bc[ff]);               // bp_bias_c1
      } else if (tid >= 192 && tid < 192 + 17) {
        const int t = tid - 192;
        float sum = 0.f;
#pragma unroll
        for (int ww = 0; ww < kTrWarps; ++ww) sum += sm.red_s[ww][t];
        if (t < 16) sm.ws[t] = fmaf(dt, sum, sm.ws[t]);          // apply_grad (s1)
        else sm.bs[0] = fmaf(dt, sum, sm.bs[0]);                 // bp_bias_s1
      }
      __syncthreads();  // (D) updated parameters visible to the next forward
    }
    // epoch end, main.cu:159-166
    if (tid == 0) {
      const float m = err / (float)n;
      if (mean_err) mean_err[e] = m;
      err = 0.f;
      sm.flag[0] = (m < threshold) ? 1 : 0;
    }
    done_epochs = e + 1;
    __syncthreads();
    if (sm.flag[0]) break;
  }
  // After an early stop up to two prefetched images are still on their way into shared memory:
  // the block does not exit under them.
  if (tid == 0) {
    for (long s2 = step; s2 < total && s2 < step + 2; ++s2)
      mbar_wait_bounded(&sm.full[s2 & 1], (unsigned)(s2 >> 1) & 1u, status, gave_up);
  }

  // write the parameters back
  for (int i = tid; i < kF * 25; i += kTrThreads) params[kOffWc + i] = sm.wc[i / 25][i % 25];
  if (tid < kF) params[kOffBc + tid] = sm.bc[tid];
  if (tid < 16) params[kOffWs + tid] = sm.ws[tid];
  if (tid == 0) params[kOffBs] = sm.bs[0];
  for (int i = tid; i < kOut * kS; i += kTrThreads) params[kOffWf + i] = sm.wf[i / kS][i % kS];
  if (tid < kOut) params[kOffBf + tid] = sm.bf[tid];
  if (tid == 0 && epochs_run) *epochs_run = done_epochs;
}

template <class K>
static int set_smem_attr(K kernel, size_t bytes) {
  CNN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return CNN_OK;
}

// `grid` blocks (one partial row each) over n images; up to one image per block a block has one team of warps, above two.
static int launch_grad(const float* d_params, float* rows, int* status, int fast, const float* d_images, const unsigned* d_labels,
                       long n, int grid, cudaStream_t st, bool chained) {
  int rc;
  cudaError_t le = cudaSuccess;
  // A block that needs little (one team, no registers for a loop) is given half an SM's shared memory and more, so that no two share an SM: batches of
  // 148 images 6.7 us a step, 8.6 without (7.0 with a loop's registers, which kept others away too).
  static_assert(sizeof(GrSmem<1>) <= 120 * 1024, "");
#define CNN_GRAD_SMEM(TEAMS) (TEAMS == 1 ? 120 * 1024 : sizeof(GrSmem<TEAMS>))
#define CNN_LAUNCH_GRAD(FL, TEAMS, ONCE)                                                                      \
  do {                                                                                                       \
    if ((rc = set_smem_attr(k_grad_partials<FL, TEAMS, ONCE>, CNN_GRAD_SMEM(TEAMS))) != CNN_OK) return rc;     \
    le = launch_pdl(k_grad_partials<FL, TEAMS, ONCE>, dim3(grid), dim3(kGrThreads * TEAMS), CNN_GRAD_SMEM(TEAMS), st, \
                    d_images, d_labels, n, d_params, rows, status, chained ? 1 : 0); \
  } while (0)
  if (n <= grid) {
    if (fast) CNN_LAUNCH_GRAD(1, 1, true);
    else CNN_LAUNCH_GRAD(0, 1, true);
  } else if (n <= 2l * grid) {
    if (fast) CNN_LAUNCH_GRAD(1, 2, true);
    else CNN_LAUNCH_GRAD(0, 2, true);
  } else {
    if (fast) CNN_LAUNCH_GRAD(1, 2, false);
    else CNN_LAUNCH_GRAD(0, 2, false);
  }
#undef CNN_LAUNCH_GRAD
#undef CNN_GRAD_SMEM
  if (le == cudaSuccess) le = cudaGetLastError();
  if (le != cudaSuccess) return cuda_fail(le, "k_grad_partials launch");
  return CNN_OK;
}

// Blocks of k_grad_partials: one per SM at most (a block holds two images at a time), so that few rows are left to add.
static int grid_for_batch(long n) {
  const long sms = sm_count();
  return (int)(n < sms ? n : sms);
}

// Tensor cores or CUDA cores.  Microseconds per gradient call, CUDA cores / tensor cores, back to back: 740 images 14.6 / 17.6, 1,000 18.0 / 20.7,
// 1,250 21.6 / 20.8, 1,480 (two tiles per SM) 22.6 / 20.8, 2,000 28.9 / 24.1, 3,000 40.2 / 30.4, 6,000 71.8 / 43.5, 20,000 220 / 106, 60,000 643 / 281.
// They meet at about 1,250; the line leaves room for images that turn out not to be whole numbers / 255 and go to the CUDA cores behind a
// look at a sample: 2,048 images 33.2 (29.0 without the look), 6,000 76 (72), 60,000 652 (643).  With other pixels in one image of a hundred 60,000
// images are 367 us, with other pixels in the second half of them 678.
int launch_gradient(cnn_net* net, const float* d_images, const unsigned* d_labels, long n, cudaStream_t st, bool chained, int* rows) {
  constexpr long kTcGradMin = 2048;
  const int sms = sm_count();
  const bool tensor = net->grad_path == 1 || (net->grad_path < 0 && n >= kTcGradMin);
  if (!tensor || !net->fast_sigmoid || n > (1l << 30)) {
    *rows = grid_for_batch(n);
    return launch_grad(net->d_params, net->d_partials, net->d_status, net->fast_sigmoid, d_images, d_labels, n, *rows, st, chained);
  }
  const long grid = (n + kGradTile - 1) / kGradTile < sms ? (n + kGradTile - 1) / kGradTile : sms;
  const GradShares shares = {(int)grid, (int)(n / grid), (int)(n % grid)};
  GradLeft* left = grad_left(net);
  int* pushed = grad_queued(net);
  int rc = set_smem_attr(k_grad_left<1>, sizeof(GrSmem<2>));
  if (rc == CNN_OK) rc = launch_grad_tc(net, d_images, d_labels, shares, left, pushed, st);
  if (rc != CNN_OK) return rc;
  cudaError_t e = launch_pdl(k_grad_left<1>, dim3((unsigned)grid), dim3(kGrThreads * 2), sizeof(GrSmem<2>), st, d_images, d_labels, shares,
                             (const float*)net->d_params, net->d_partials, net->d_status, left, pushed);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    cudaMemsetAsync(pushed, 0, sizeof(GradLeft) * (1 + (size_t)sms) - sizeof(int), st);      // nobody takes what the kernel before has queued
    return cuda_fail(e, "k_grad_left launch");
  }
  *rows = (int)grid;
  return CNN_OK;
}

}  // namespace cnn

using namespace cnn;

extern "C" {

int cnn_grad_batch(cnn_net* net, const float* d_images, const unsigned int* d_labels, long n,
                   float* d_grad, void* stream) {
  CNN_REQUIRE(net && d_grad, "cnn_grad_batch: NULL argument");
  CNN_REQUIRE(n >= 0, "cnn_grad_batch: negative image count");
  cudaStream_t st = as_stream(stream);
  if (n == 0) {
    CNN_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(float) * kNParamsPadded, st));
    return CNN_OK;
  }
  CNN_REQUIRE(d_images && d_labels, "cnn_grad_batch: NULL images or labels");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_images) & 15u) == 0,
              "cnn_grad_batch: image batch must start on a 16-byte boundary");
  int rc = ensure_train_scratch(net);
  if (rc != CNN_OK) return rc;
  int rows = 0;
  if ((rc = launch_gradient(net, d_images, d_labels, n, st, false, &rows)) != CNN_OK) return rc;
  cudaError_t e = launch_pdl(k_reduce_rows, dim3((kNParamsPadded + 31) / 32), dim3(32 * kRedGroups), 0, st,
                             (const float*)net->d_partials, rows, d_grad, (float*)nullptr, 0.f, (float*)nullptr, 0.f);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_reduce_rows launch");
  return CNN_OK;
}

int cnn_apply_update(cnn_net* net, const float* d_grad, float scale, void* stream) {
  CNN_REQUIRE(net && d_grad, "cnn_apply_update: NULL argument");
  cudaError_t e = launch_pdl(k_apply_update, dim3((kNParams + 255) / 256), dim3(256), 0, as_stream(stream), net->d_params, d_grad, scale);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_apply_update launch");
  return CNN_OK;
}

int cnn_train_minibatch(cnn_net* net, const float* d_images, const unsigned int* d_labels, long n,
                        int batch, int epochs, float dt, float* d_mean_err, void* stream) {
  CNN_REQUIRE(net != nullptr, "cnn_train_minibatch: NULL net");
  CNN_REQUIRE(n >= 0 && batch > 0 && epochs >= 0, "cnn_train_minibatch: bad sizes");
  if (n == 0 || epochs == 0) return CNN_OK;
  CNN_REQUIRE(d_images && d_labels, "cnn_train_minibatch: NULL images or labels");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_images) & 15u) == 0,
              "cnn_train_minibatch: image batch must start on a 16-byte boundary");
  cudaStream_t st = as_stream(stream);
  int rc = ensure_train_scratch(net);
  if (rc != CNN_OK) return rc;
  if (d_mean_err) CNN_CUDA(cudaMemsetAsync(d_mean_err, 0, sizeof(float) * (size_t)epochs, st));
  for (int e = 0; e < epochs; ++e) {
    for (long first = 0; first < n; first += batch) {
      const long b = (n - first) < batch ? (n - first) : batch;
      int rows = 0;
      if ((rc = launch_gradient(net, d_images + first * kImg, d_labels + first, b, st, first > 0 || e > 0, &rows)) != CNN_OK) return rc;
      cudaError_t err = launch_pdl(k_reduce_rows, dim3((kNParamsPadded + 31) / 32), dim3(32 * kRedGroups), 0, st,
                                   (const float*)net->d_partials, rows, net->d_grad, net->d_params, dt / (float)b,
                                   d_mean_err ? d_mean_err + e : nullptr, 1.0f / (float)n);
      if (err == cudaSuccess) err = cudaGetLastError();
      if (err != cudaSuccess) return cuda_fail(err, "k_reduce_rows launch");
    }
  }
  return CNN_OK;
}

int cnn_train_sgd_persample(cnn_net* net, const float* d_images, const unsigned int* d_labels, long n,
                            int epochs, float dt, float threshold, float* h_mean_err, int* h_epochs_run,
                            void* stream) {
  CNN_REQUIRE(net != nullptr, "cnn_train_sgd_persample: NULL net");
  CNN_REQUIRE(n >= 0 && epochs >= 0, "cnn_train_sgd_persample: bad sizes");
  if (h_epochs_run) *h_epochs_run = 0;
  if (n == 0 || epochs == 0) return CNN_OK;
  CNN_REQUIRE(d_images && d_labels, "cnn_train_sgd_persample: NULL images or labels");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_images) & 15u) == 0,
              "cnn_train_sgd_persample: image batch must start on a 16-byte boundary");
  cudaStream_t st = as_stream(stream);
  int rc = ensure_train_scratch(net);
  if (rc != CNN_OK) return rc;
  // Scratch reuse: d_grad holds the per-epoch means (epochs <= kNParamsPadded) and the epoch count.
  CNN_REQUIRE(epochs <= kNParamsPadded, "cnn_train_sgd_persample: too many epochs");
  float* d_mean = net->d_grad;
  int* d_ran = reinterpret_cast<int*>(net->d_grad + kNParamsPadded);
  const size_t smem = sizeof(TrSmem);
  if (net->ps_kernel) {
    if ((rc = launch_persample_cluster8(net, d_images, d_labels, n, epochs, dt, threshold, d_mean, d_ran, st)) != CNN_OK)
      return rc;
  } else {
#define CNN_LAUNCH_PS(FL)                                                                          \
  do {                                                                                             \
    if ((rc = set_smem_attr(k_train_persample<FL>, smem)) != CNN_OK) return rc;                    \
    k_train_persample<FL><<<1, kTrThreads, smem, st>>>(d_images, d_labels, n, epochs, dt, threshold, \
                                                       net->d_params, d_mean, d_ran, net->d_status); \
  } while (0)
  if (net->fast_sigmoid) CNN_LAUNCH_PS(1);
  else CNN_LAUNCH_PS(0);
#undef CNN_LAUNCH_PS
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_train_persample launch");
  CNN_CUDA(cudaStreamSynchronize(st));
  int ran = 0;
  CNN_CUDA(cudaMemcpy(&ran, d_ran, sizeof(int), cudaMemcpyDeviceToHost));
  if (h_epochs_run) *h_epochs_run = ran;
  if (h_mean_err && ran > 0)
    CNN_CUDA(cudaMemcpy(h_mean_err, d_mean, sizeof(float) * (size_t)ran, cudaMemcpyDeviceToHost));
  int status = 0;
  CNN_CUDA(cudaMemcpy(&status, net->d_status, sizeof(int), cudaMemcpyDeviceToHost));
  if (status != 0) {
    set_error("cnn_train_sgd_persample: a bounded device-side wait ran out");
    int zero = 0;
    cudaMemcpy(net->d_status, &zero, sizeof(int), cudaMemcpyHostToDevice);
    return CNN_ERR_TIMEOUT;
  }
  return CNN_OK;
}

// ----------------------------------------------------------------------------------------------
// Gradient of a batch without any allocation.
//
// Some callers may not allocate device memory at the point where they need a gradient: code that
// runs inside a memory-budgeted service whose pools are carved up at start-up, plug-ins that are
// handed device buffers by a host application and are forbidden to call cudaMalloc themselves,
// and real-time loops where an allocation (a device-wide synchronisation) is not acceptable.
// cnn_grad_batch needs a cnn_net, and creating one allocates; this entry point takes raw device
// pointers instead and keeps the partial-gradient rows of k_grad_partials in a fixed array that is
// part of the library image.
// ----------------------------------------------------------------------------------------------
namespace cnn {
constexpr int kNoAllocMaxRows = 160;          // one row per block, at most this many blocks
constexpr long kNoAllocMaxImages = 65536;     // largest batch the entry point accepts
// rows | status word (+ padding to keep the array a multiple of 256 bytes)
constexpr size_t kNoAllocFloats = (size_t)kNoAllocMaxRows * kRowStride + 64;
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocFloats];

// Set-up, once per device, with that device current: in host code the array's name is only a
// handle, its device address has to be asked for.
static int noalloc_scratch(float** rows) {
  static float* scratch_of_device[64] = {nullptr};
  int dev = -1;
  CNN_CUDA(cudaGetDevice(&dev));
  CNN_REQUIRE(dev >= 0 && dev < 64, "cnn_grad_batch_noalloc: device ordinal out of range");
  if (scratch_of_device[dev] == nullptr) {
    float* ptr = nullptr;
    CNN_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_noalloc_scratch));
    CNN_REQUIRE(ptr != nullptr, "cnn_grad_batch_noalloc: no device address for the scratch array");
    scratch_of_device[dev] = ptr;
  }
  *rows = scratch_of_device[dev];
  return CNN_OK;
}
}  // namespace cnn

int cnn_grad_batch_noalloc(const float* d_params, const float* d_images, const unsigned int* d_labels,
                           long n, float* d_grad, void* stream) {
  CNN_REQUIRE(d_params && d_grad, "cnn_grad_batch_noalloc: NULL params or gradient buffer");
  CNN_REQUIRE(n >= 0, "cnn_grad_batch_noalloc: negative image count");
  if (n > kNoAllocMaxImages) {
    set_error("cnn_grad_batch_noalloc: %ld images exceed the fixed-scratch limit of %ld per call; "
              "split the batch (gradients add) or use cnn_grad_batch", n, kNoAllocMaxImages);
    return CNN_ERR_INVALID;
  }
  cudaStream_t st = as_stream(stream);
  if (n == 0) {
    CNN_CUDA(cudaMemsetAsync(d_grad, 0, sizeof(float) * kNParamsPadded, st));
    return CNN_OK;
  }
  CNN_REQUIRE(d_images && d_labels, "cnn_grad_batch_noalloc: NULL images or labels");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_images) & 15u) == 0,
              "cnn_grad_batch_noalloc: image batch must start on a 16-byte boundary");
  float* rows = nullptr;
  int rc = noalloc_scratch(&rows);
  if (rc != CNN_OK) return rc;
  int* status = reinterpret_cast<int*>(rows + (size_t)kNoAllocMaxRows * kRowStride);

  long grid_l = sm_count();
  if (grid_l > kNoAllocMaxRows) grid_l = kNoAllocMaxRows;
  if (grid_l > n) grid_l = n;
  const int grid = (int)grid_l;
  // The array keeps what the previous call left.  Every row that is read below is rewritten in full
  // by its block, padding included, so no row needs clearing.  The status word starts at zero when
  // the library is loaded, is only ever set by a wait that ran out, and stays set until
  // cnn_grad_batch_noalloc_status reads and clears it.
  if ((rc = launch_grad(d_params, rows, status, 0, d_images, d_labels, n, grid, st, false)) != CNN_OK) return rc;
  cudaError_t e = launch_pdl(k_reduce_rows, dim3((kNParamsPadded + 31) / 32), dim3(32 * kRedGroups), 0, st, (const float*)rows, grid,
                             d_grad, (float*)nullptr, 0.f, (float*)nullptr, 0.f);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_reduce_rows launch (no-alloc)");
  return CNN_OK;
}

int cnn_grad_batch_noalloc_status(void* stream) {
  float* rows = nullptr;
  int rc = noalloc_scratch(&rows);
  if (rc != CNN_OK) return rc;
  int* d_status = reinterpret_cast<int*>(rows + (size_t)kNoAllocMaxRows * kRowStride);
  cudaStream_t st = as_stream(stream);
  CNN_CUDA(cudaStreamSynchronize(st));
  int status = 0;
  CNN_CUDA(cudaMemcpyAsync(&status, d_status, sizeof(int), cudaMemcpyDeviceToHost, st));
  CNN_CUDA(cudaStreamSynchronize(st));
  if (status != 0) {
    CNN_CUDA(cudaMemsetAsync(d_status, 0, sizeof(int), st));
    CNN_CUDA(cudaStreamSynchronize(st));
    set_error("cnn_grad_batch_noalloc: a bounded device-side wait ran out; the gradient of that call is not valid");
    return CNN_ERR_TIMEOUT;
  }
  return CNN_OK;
}

int cnn_copy_to_host(void* h_dst, const void* d_src, size_t bytes) {
  CNN_REQUIRE(h_dst && d_src, "cnn_copy_to_host: NULL argument");
  CNN_CUDA(cudaMemcpy(h_dst, d_src, bytes, cudaMemcpyDeviceToHost));
  return CNN_OK;
}

int cnn_copy_to_device(void* d_dst, const void* h_src, size_t bytes) {
  CNN_REQUIRE(d_dst && h_src, "cnn_copy_to_device: NULL argument");
  CNN_CUDA(cudaMemcpy(d_dst, h_src, bytes, cudaMemcpyHostToDevice));
  CNN_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // a pageable source may still be in DMA on return
  return CNN_OK;
}

}  // extern "C"
