// Batched forward of the reference's 28x28 net with the convolution (fp_preact_c1, layer.cu:116-133:
// 94 % of the forward MACs) on the 5th-generation tensor cores (tcgen05, accumulators in tensor
// memory), and everything after it -- bias, sigmoid, shared 4x4 subsample, sigmoid, FC 216->10,
// sigmoid, argmax -- done by the epilogue warps straight out of tensor memory.  Selected with the
// option "forward_path" = 1 (two passes, three where pixels leave a remainder, fp32-level accuracy; the default for large batches, fp32 images
// or uint8 pixels) or 2 (one pass and a tanh.approx sigmoid: an explicitly reduced-precision inference mode).
//
// The convolution as a GEMM WITHOUT an im2col copy.  For kernel row i the conv is a product of image rows
// with a banded (Toeplitz) weight matrix,
//     out[y][x][f] = sum_i sum_c R[y + i][c] * T_i[c][x][f],   T_i[c][x][f] = Wc[f][i][c - x] (0 <= c-x < 5),
// so the A operand of kernel row i is the SAME tile of image rows, started i rows further down: in the
// un-swizzled K-major shared-memory layout a row is 16 bytes inside each 16-byte column chunk
// ([chunk][row][8 fp16]), and a matrix descriptor may start at any row.  M is made of groups of 8 output
// rows (the layout's core matrices); a group keeps the 12 input rows it needs, so the group stride is
// 12 rows and an image's 24 output rows are exactly three groups: no output row is computed for nothing.
// (Stacking whole images, 28 rows each, wasted 4 rows in 28 of everything below: tensor work, sigmoids, epilogue.)
// The band is cut into two blocks of 12 output columns (16 input columns, K = 16 per kernel row = one MMA),
// and because the weights are shift-invariant both blocks use the same B operand: 5 x [80 x 16] values.
// Column chunks are kept at columns 0-7, 8-15, 12-19, 20-27, so that both blocks start on a chunk.
// One tile of 16 groups (5.33 images) costs 10 MMAs of 128 x 80 x 16 per pass.
//
// Accuracy.  Path 1 splits both operands into an fp16 high part and an fp16 remainder and issues hi*hi + hi*lo +
// lo*hi (fp32 accumulation): 22-23 significant bits of either operand take part, what is left out is lo*lo,
// about 2^-24 relative.  fp16 instead of tf32 halves the MMAs (K = 16 per instruction at the same operand bytes,
// and operand bytes are what an MMA of this shape costs) at one more bit of mantissa.  Its range does not cover
// fp32's, so weights and pixels are scaled with powers of two that follow the largest weight w (undone, exactly, in the
// epilogue's bias FMA): weights so that w lies between 256 and 512, pixels by more than 25 w, which keeps what a pixel's
// parts lose (2^-25 of the scaled value, absolute) below 2^-24 in any pre-activation, whatever the pixels.
// Besides the power of two a pixel is multiplied by 255, and the weights by 1 / 255 (in two parts, so that it costs them
// nothing): a pixel that is a byte / 255, as image files have them, then is a whole number below 256 times a power of two, in fp32
// arithmetic exactly, its high part all of it and its remainder zero.  A tile of such images takes two passes instead
// of three; the third would add zeros, so what an image gives does not depend on its neighbours.  (65,536 images: 138 -> 115 us; images
// of other numbers 134 -> 127 us, by the loader alone.)  Such a pixel kept as a byte needs no table: fp16(byte) is two instructions per pair.
// Another pixel's product with 255 is rounded, which does not show: outputs of noise and of normalised noise, eight nets as drawn, are 7.0e-8 and 7.1e-8
// of their norm from fp64 with the power of two alone, with 255, and with the remainder of the exact product (146 us).
// An image with a scaled pixel of 65,520 or more (a pixel of 1,000 to 2,000 where w = 1: its pre-activations are no longer
// of order one) is noticed by the loader, and a finisher warp computes it in plain fp32 instead (slow, 0.1 ms per image; no
// image data is expected there).  uint8 pixels reach that limit only where w is above 1,000: the finishers look for themselves
// then.  With a weight or a conv bias of 1e27 or more, or one that is not finite, all images go that way.
// Path 2 uses the high parts only (11 significant bits, as tf32) and one special-function operation
// per activation: outputs within about 1e-4, argmax equal wherever the top-two margin is clear of that.
//
// Pipeline (one CTA per SM, 20 warps, everything handed over through mbarriers with bounded waits):
//   warps 4-7   fetch the tile's rows -- consecutive in HBM -- by one bulk copy per tile, three tiles ahead (path 2: warp 3 does), convert
//               them to fp16 high and low parts and store them in the operand layout, 16 bytes per store.  A copy into registers
//               one tile ahead left its latency, 2,300 cycles per tile, in the path: cost 4 us of 136;
//   warp 3      issues the tile's MMAs into one of three 160-column accumulators and commits to
//               mbarriers (the whole warp runs the loop, an elected lane issues: see wide_tc.cuh);
//   warps 8-19  three epilogue groups of four warps (one per 32-lane quarter of tensor memory), one
//               tile each: tcgen05.ld of 8 columns (one window row of two maps) at a time, software
//               pipelined; bias, sigmoid, the window row's four subsample taps; the four rows of a
//               window are four adjacent lanes (reduce-scatter by shuffles); subsample sigmoid; the
//               activation into the image's slot in shared memory, window rows counted on its mbarrier;
//   warps 0-2   finish images in order, three at a time in turn: FC 216 -> 10 (lane = every 32nd subsample
//               output, so the weights are read once for three images), reduce-scatter, output
//               sigmoid, argmax (lowest index wins ties), 44 bytes per image to HBM.
//
// Measured on a B200 (three passes whatever the pixels, a table for uint8 before, now): 65,536 fp32 images 138 -> 114 us, 30,011 uint8 images
// 65 -> 53 us, path 2 on 65,536 images 98 -> 91 us (loader without bank conflicts).  What bounds it now, per tile of 5.33 images
// (2,400 cycles): the shared-memory data pipe (20 MMAs fetch 130 KB of operands, 1,040 cycles, the other warps and the copies take 900),
// and next the special-function unit (1,600 cycles) and instruction issue (1,400); path 2: the same pipe, 88 % busy, then the special-function unit, 64 %.
#include <type_traits>

#include "banded_conv.cuh"
#include "cluster_exchange.cuh"
#include "net.cuh"
#include "wide_tc.cuh"
#include "phase_clocks.cuh"

namespace cnn {

constexpr int kTfThreads = 640;
constexpr int kTfSlabsTotal = 6;             // operand slabs in shared memory: path 1 uses them as 3 (high, low)
                                             // pairs, path 2 as 6
constexpr int kTfRaw = 4;                    // tiles of raw image rows in shared memory
constexpr int kTfAcc = 3;                    // accumulators in tensor memory
constexpr int kTfGroups = 16;                // groups of 8 output rows per tile (M = 128)
constexpr int kTfGroupsImg = 3;              // groups per image
constexpr int kTfGroupRows = 12;             // input rows a group keeps: 8 + 4
constexpr unsigned kTfGroupStride = kTfGroupRows * 16;                       // 192 B
constexpr unsigned kTfChunkStride = kTfGroups * kTfGroupStride + 16;         // 3,088 B: the 16 B put the four chunks of the rows
                                                                             // r and r + 4 into different banks for the loader
constexpr int kTfSlabBytes = 4 * kTfChunkStride;                             // 12,352
constexpr int kTfBN = 80;                    // MMA N of one 12-column block: 72 used, padded to 16n
constexpr unsigned kTfBChunk = kTfBN * 16;   // 1,280 B between the two K chunks of a kernel row
constexpr unsigned kTfBRow = 2 * kTfBChunk;  // 2,560 B per kernel row (K = 16)
constexpr int kTfBBytes = 5 * kTfBRow;       // 12,800
constexpr int kTfDCols = 2 * kTfBN;          // 160 accumulator columns per tile
constexpr int kTfSlots = 32;                 // images whose FC sums may be in flight (ring)
constexpr int kTfRange = 128;                // ring of out-of-range marks: more images than can be between loader and finisher
constexpr int kTfFinishers = 3;
constexpr int kTfMmaWarp = 3;
constexpr int kTfLoadWarp0 = 4, kTfLoaders = 128;
constexpr int kTfUnits = kTfGroups * kTfGroupRows * 4 / kTfLoaders;   // 6 chunk rows (8 pixels) per loader thread and tile
constexpr int kTfEpiWarp0 = 8;
constexpr float kTfMaxExp = 31.f;            // (1 + 2^31)^4 is still finite
constexpr int kTfFcIn = 7;                   // subsample outputs per lane of a finisher warp: 216 = 6.75 x 32
constexpr int kTfAsStride = 32 * kTfFcIn;    // 224

constexpr int kTfRawPixels = kTfGroups * 8 * kH + 6 * 4 * kH;   // a tile meets six images at most, four halo rows each

struct TfSmem {
  alignas(128) float raw[kTfRaw][kTfRawPixels];               // image rows as they lie in HBM (fp32, or uint8 in the first quarter)
  alignas(128) unsigned char slab[kTfSlabsTotal][kTfSlabBytes];   // path 1: slab s = high part, slab s + 3 = low part
  alignas(128) unsigned char b_hi[kTfBBytes];
  alignas(128) unsigned char b_lo[kTfBBytes];                 // path 1 only
  alignas(16) float wf[kTfFcIn][3][32][4];    // FC weights of subsample output 32 j + lane: ten, padded to twelve
  alignas(16) float as[kTfSlots][kTfAsStride];   // subsample activations of an image: [window row][6 * window column + map]
  float bc[8], ws[16], bs[4], bf[12];
  unsigned long long raw_full[kTfRaw], raw_free[kTfRaw];
  unsigned long long a_full[kTfSlabsTotal], a_free[kTfSlabsTotal], d_full[2 * kTfAcc], d_free[2 * kTfAcc], img_done[kTfSlots];
  unsigned char out_of_range[kTfRange];
  alignas(4) unsigned char has_low[kTfSlabsTotal][4];    // per slab and loader warp: some pixel of the tile has a remainder
  int finished[kTfFinishers];                            // image triples that each finisher warp has written out (slot reuse guard)
  unsigned tmem_base;
  long long clock_base;                       // phase clocks only
};

CNN_PHASE_TABLE(g_phase_clocks_tc, 20)

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Group g of a CTA starts 224 g + 112 (g / 3) pixels into its images: 8 rows further per group, 12 more per image.
__device__ __forceinline__ int group_pixel(int g) { return 8 * kH * g + 4 * kH * (g / kTfGroupsImg); }

// Bounded spin on a counter in shared memory (same limit and status convention as mbar_wait_bounded).
__device__ __forceinline__ void wait_counter_bounded(const int* counter, int at_least, int* status, bool& gave_up) {
  if (gave_up) return;
  if (*reinterpret_cast<const volatile int*>(counter) >= at_least) return;
  const long long t0 = clock64();
  while (*reinterpret_cast<const volatile int*>(counter) < at_least) {
    if (clock64() - t0 > 4000000000LL) {
      gave_up = true;
      if (status) atomicExch(status, 1);
      return;
    }
  }
}

// FC sums (without bias) of one image in plain fp32 by one warp, lane k < 10 returns sum k: the way out for images whose
// pixels do not fit fp16.  Lanes own windows; kept out of line and rolled so that it costs the hot code nothing.
template <int SIG, typename Pixel>
__device__ __noinline__ float image_fc_plain(const Pixel* image, const float* params, int lane) {
  auto pixel = [](Pixel v) { return sizeof(Pixel) == 1 ? (float)((double)v / 255.0) : (float)v; };
  float mine = 0.f;
#pragma unroll 1
  for (int w0 = 0; w0 < 36; w0 += 32) {
    const int w = w0 + lane;
    const bool live = w < 36;
    const Pixel* base = image + (live ? (4 * (w / 6)) * kH + 4 * (w % 6) : 0);
#pragma unroll 1
    for (int f = 0; f < kF; ++f) {
      float zs = params[kOffBs];
#pragma unroll 1
      for (int o = 0; o < 16; ++o) {
        float acc = params[kOffBc + f];
#pragma unroll 1
        for (int t = 0; t < 25; ++t)
          acc = fmaf(params[kOffWc + f * 25 + t], pixel(base[(o / 4 + t / 5) * kH + o % 4 + t % 5]), acc);
        zs = fmaf(params[kOffWs + o], sigmoidf<SIG>(acc), zs);
      }
      const float as = live ? sigmoidf<SIG>(zs) : 0.f;
#pragma unroll 1
      for (int k = 0; k < kOut; ++k) {
        float v = live ? params[kOffWf + k * kS + f * 36 + w] * as : 0.f;
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
        if (lane == k) mine += v;
      }
    }
  }
  return mine;
}

// uint8 pixels where the parameters ask for the way out: white, at the scale that the weights set, is beyond fp16 (weights above 1,000), or, `all`,
// the parameters are.  FC sums of the three images from `base` on (of a CTA's images; lane 10 j + k: sum k), `z` where the tensor core's
// are right.  As the fp32 images' loader does, all images of a tile with a pixel out of range are taken -- noticed here, because in the
// loader it cost 5 % of every call.
template <int SIG>
__device__ __noinline__ float finish_plain_u8(const unsigned char* pixels, const float* params, float level, int base, int imgs, bool all,
                                              float z, int lane) {
  for (int j = 0; j < 3 && base + j < imgs; ++j) {
    const int g = (base + j) * kTfGroupsImg, end = imgs * kTfGroupsImg;
    const int g0 = g / kTfGroups * kTfGroups, g1 = min(((g + kTfGroupsImg - 1) / kTfGroups + 1) * kTfGroups, end) - 1;      // of its tiles
    unsigned most = 0;
    for (int i = group_pixel(g0) / 4 + lane; i < (group_pixel(g1) + kTfGroupRows * kH) / 4; i += 32)
      most = __vmaxu4(most, reinterpret_cast<const unsigned*>(pixels)[i]);
    most = __reduce_max_sync(0xffffffffu, max(max(most & 255u, (most >> 8) & 255u), max((most >> 16) & 255u, most >> 24)));
    if (!all && (float)most * level < 65520.f) continue;      // its high part is finite
    const float s = image_fc_plain<SIG>(pixels + (size_t)(base + j) * kImg, params, lane);
    const float sk = __shfl_sync(0xffffffffu, s, lane % 10);
    if (lane / 10 == j) z = sk;
  }
  return z;
}

// PATH 1: two or three passes, sigmoid flavour SIG (0 or 1).  PATH 2: one pass, tanh sigmoid.  U8: `images` points at
// uint8 pixels and the kernel applies the reference's ingest, float(pixel / 255.0) (mnist.h:145, main.cu:57-65).
template <int PATH, int SIG, bool U8>
__global__ void __launch_bounds__(kTfThreads, 1)
k_forward_tc(const void* images, long n, long imgs_per_cta, const float* params,
             float* __restrict__ out, int* __restrict__ argmax, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  TfSmem& sm = *reinterpret_cast<TfSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool kPrecise = (PATH == 1);
  constexpr bool kLow = kPrecise && !U8;                                   // pixels may have a remainder
  constexpr int kTfSlabs = kLow ? kTfSlabsTotal / 2 : kTfSlabsTotal;       // slabs in flight
  // Path 2 computes tanh(v / 2): conv weights and bias are halved.  Path 1 with the short sigmoid form folds
  // the form's multiplication by -log2(e) into them.
  constexpr bool kShort = kPrecise && (SIG == 1);
  constexpr float kPre = kPrecise ? (kShort ? -1.4426950408889634f : 1.0f) : 0.5f;

  const long img0 = (long)blockIdx.x * imgs_per_cta;
  const long imgs_here_l = (n - img0) < imgs_per_cta ? (n - img0) : imgs_per_cta;
  const int imgs_here = imgs_here_l > 0 ? (int)imgs_here_l : 0;
  const int n_groups = imgs_here * kTfGroupsImg;
  const int n_tiles = (n_groups + kTfGroups - 1) / kTfGroups;

  // ---- set-up that touches nothing of the kernel before this one ------------------------------------
  pdl_launch_dependents();
  if (tid == 32 * kTfMmaWarp) {
    for (int s = 0; s < kTfRaw; ++s) {
      mbar_init(&sm.raw_full[s], 1);
      mbar_init(&sm.raw_free[s], kTfLoaders / 32);
    }
    for (int s = 0; s < kTfSlabs; ++s) {
      mbar_init(&sm.a_full[s], kTfLoaders / 32);
      mbar_init(&sm.a_free[s], 1);
    }
    for (int s = 0; s < 2 * kTfAcc; ++s) {      // one pair per column block of an accumulator
      mbar_init(&sm.d_full[s], 1);
      mbar_init(&sm.d_free[s], 4);
    }
    for (int s = 0; s < kTfSlots; ++s) mbar_init(&sm.img_done[s], 6);
    mbar_fence_init();
    for (int w = 0; w < kTfFinishers; ++w) sm.finished[w] = 0;
  }
  if (tid < kTfRange) sm.out_of_range[tid] = 0;
  if (kLow)      // no remainders yet (written by the first tiles instead: 1.3 us more per call)
    for (int i = tid; i < kTfSlabsTotal / 2 * kTfSlabBytes / 16; i += kTfThreads)
      reinterpret_cast<uint4*>(sm.slab[kTfSlabsTotal / 2])[i] = make_uint4(0, 0, 0, 0);
  if (tid < 8 * kTfSlots) sm.as[tid >> 3][216 + (tid & 7)] = 0.f;     // the padding meets zero weights and has to be finite
  if (warp == kTfMmaWarp) tc::tmem_alloc(&sm.tmem_base, 512);
  pdl_wait();

  // ---- loaders: the first copies leave now ------------------------------------------------------------------
  const int lt = tid - 32 * kTfLoadWarp0;
  const bool loader = lt >= 0 && lt < kTfLoaders;
  // One thread: the rows of tile k, from its first group's first to its last group's twelfth (source offset, size), by one bulk copy.
  constexpr unsigned kPixelBytes = U8 ? 1u : 4u;
  auto fetch_extent = [&](int k, unsigned& bytes) {
    const int g0 = k * kTfGroups, g1 = min(g0 + kTfGroups, n_groups) - 1;
    const int first = group_pixel(g0);
    bytes = (unsigned)(group_pixel(g1) + kTfGroupRows * kH - first) * kPixelBytes;
    return static_cast<const unsigned char*>(images) + (size_t)(img0 * kImg + first) * kPixelBytes;
  };
  auto fetch = [&](int k, const unsigned char* src, unsigned bytes) {
    unsigned long long* bar = &sm.raw_full[k % kTfRaw];
    mbar_expect_tx(bar, bytes);
    bulk_g2s(sm.raw[k % kTfRaw], src, bytes, bar);
  };

  if (tid == 32 * kTfMmaWarp)        // the thread that initialised the barriers
    for (int k = 0; k < kTfRaw && k < n_tiles; ++k) {
      unsigned bytes;
      const unsigned char* src = fetch_extent(k, bytes);
      fetch(k, src, bytes);
    }

  // ---- set-up: weight scale, B operand (banded weights), FC table, small parameters -------------------------
  // Every load of a thread is under way before the first value is used: one wait for L2 instead of three in a row.
  constexpr int kBRows = 5 * 2 * kTfBN, kBTurns = (kBRows + kTfThreads - 1) / kTfThreads;      // 16-byte rows of the B operand
  float bw[kBTurns][5], wfc[kOut], small;
#pragma unroll
  for (int t = 0; t < kBTurns; ++t) {
    const int e = min(tid + t * kTfThreads, kBRows - 1), nn = e % kTfBN;
    const int at = nn < 72 ? kOffWc + band_map(nn) * 25 + e / (2 * kTfBN) * 5 : 0;
#pragma unroll
    for (int d = 0; d < 5; ++d) bw[t][d] = params[at + d];
  }
  {
    const int u = min(tid, kS - 1), p = u / 36, q = (u % 36) / 6, f = u % 6, t = tid - 256;
#pragma unroll
    for (int k = 0; k < kOut; ++k) wfc[k] = params[kOffWf + k * kS + f * 36 + p * 6 + q];
    small = params[t < 0 || t > 40 ? 0 : (t < 16 ? kOffWs + t : (t < 28 ? kOffBf + min(t - 16, kOut - 1) : (t < 28 + kF ? kOffBc + t - 28 : kOffBs)))];
  }
  float wmax = 0.f;
  bool finite = true;
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int e = lane + 32 * j;      // the 150 weights and 6 biases
    if (e < kOffBc + kF) {
      const float a = fabsf(params[e]);
      finite = finite && (a <= 1e27f);      // (below 2^90: the weights' exponent is not clamped)
      if (e < kOffBc) wmax = fmaxf(wmax, a);
    }
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, m));
  const bool plain = !__all_sync(0xffffffffu, finite);    // parameters that fp16 cannot stand in for: every image in plain fp32
  // With 2^E <= max |kPre * w| < 2^(E+1) weights are scaled by 2^(16-E) / 255 and pixels by 255 * 2^(E-3): the accumulator carries 2^13.
  int wexp = (int)((__float_as_uint(fabsf(kPre) * wmax) >> 23) & 255u) - 127;
  wexp = wexp > 90 ? 90 : (wexp < -90 ? -90 : wexp);
  const float w_scale = __int_as_float((127 + 16 - wexp) << 23), px_scale = 255.f * __int_as_float((127 - 3 + wexp) << 23);
  constexpr float w_unscale = 1.0f / 8192.0f;

#pragma unroll
  for (int turn = 0; turn < kBTurns; ++turn) {     // one 16-byte row of a chunk: 8 columns of one accumulator column
    const int e = tid + turn * kTfThreads;
    if (e >= kBRows) break;
    const int i = e / (2 * kTfBN), rem = e % (2 * kTfBN);
    const int ch = rem / kTfBN, nn = rem % kTfBN, x = band_column(nn);
    float w[5];
#pragma unroll
    for (int d = 0; d < 5; ++d) w[d] = (nn < 72) ? w_scale * bw[turn][d] : 0.f;
    __half2 hi[4], lo[4];
    constexpr TwoPart kFactor = two_part((double)kPre / 255.0);
    band_row(w, 8 * ch - x, kFactor, hi, lo);
    const unsigned off = (unsigned)i * kTfBRow + (unsigned)ch * kTfBChunk + (unsigned)nn * 16u;
    *reinterpret_cast<uint4*>(sm.b_hi + off) = *reinterpret_cast<uint4*>(hi);
    if (kPrecise) *reinterpret_cast<uint4*>(sm.b_lo + off) = *reinterpret_cast<uint4*>(lo);
  }
  if (tid < kTfAsStride) {       // FC table
    float w[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) w[k] = (tid < kS && k < kOut) ? wfc[k < kOut ? k : 0] : 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      *reinterpret_cast<float4*>(sm.wf[tid >> 5][k][tid & 31]) = make_float4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
  } else if (tid >= 256 && tid < 256 + 64) {
    const int t = tid - 256;
    if (t < 16) sm.ws[t] = small;
    else if (t < 28) sm.bf[t - 16] = (t - 16 < kOut) ? small : 0.f;
    else if (t < 28 + kF) sm.bc[t - 28] = kPre * small;
    else if (t == 40) sm.bs[0] = small;
  }
  tc::fence_async_smem();      // the B operand was written through the generic proxy
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const unsigned tmem_base = sm.tmem_base;

  bool gave_up = false;
  CNN_PHASE_BEGIN(blockIdx.x == 0, sm.clock_base)

  if (warp < kTfFinishers) {
    // ================= finishers: images in order, three at a time in turn ===========================
    const int li = lane / 10, k = lane % 10;
    for (int base = 3 * warp, turn = 0; base < imgs_here; base += 3 * kTfFinishers) {
      const int img = base + li;
      const bool active = (lane < 30) && (img < imgs_here);
      CNN_PHASE(0);
      const float* as[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int slot = (base + j) & (kTfSlots - 1);
        as[j] = &sm.as[slot][lane];
        if (base + j < imgs_here) mbar_wait_bounded(&sm.img_done[slot], (unsigned)((base + j) / kTfSlots) & 1u, status, gave_up);
      }
      CNN_PHASE(1);
      f32x2 fc2[3][kOut / 2];
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int kk = 0; kk < kOut / 2; ++kk) fc2[j][kk] = pack2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kTfFcIn; ++i) {
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(sm.wf[i][0][lane]);
        const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(sm.wf[i][1][lane]);
        const f32x2 w4 = *reinterpret_cast<const f32x2*>(sm.wf[i][2][lane]);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float a = as[j][32 * i];
          const f32x2 a2 = pack2(a, a);
          fc2[j][0] = fma2(w0.x, a2, fc2[j][0]); fc2[j][1] = fma2(w0.y, a2, fc2[j][1]); fc2[j][2] = fma2(w1.x, a2, fc2[j][2]);
          fc2[j][3] = fma2(w1.y, a2, fc2[j][3]); fc2[j][4] = fma2(w4, a2, fc2[j][4]);
        }
      }
      float sums[32];
      sums[30] = sums[31] = 0.f;
#pragma unroll
      for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int kk = 0; kk < kOut / 2; ++kk) unpack2(fc2[j][kk], sums[10 * j + 2 * kk], sums[10 * j + 2 * kk + 1]);
      float z = warp_reduce_scatter32(sums, lane);      // lane 10 li + k: sum k of image base + li
      if constexpr (U8) {
        if (plain || px_scale >= 65520.f)
          z = finish_plain_u8<SIG>(static_cast<const unsigned char*>(images) + img0 * kImg, params, px_scale * (1.0f / 255.0f), base, imgs_here, plain, z, lane);
      }
      const bool bad = !U8 && active && (plain || sm.out_of_range[img & (kTfRange - 1)] != 0);
      if (!U8 && __any_sync(0xffffffffu, bad)) {
        for (int j = 0; j < 3; ++j) {
          if (!__shfl_sync(0xffffffffu, (int)bad, 10 * j)) continue;
          const float s = image_fc_plain<kPrecise ? SIG : 1>(static_cast<const float*>(images) + (img0 + base + j) * kImg, params, lane);
          const float sk = __shfl_sync(0xffffffffu, s, k);
          if (li == j) z = sk;
        }
        if (bad && k == 0) sm.out_of_range[img & (kTfRange - 1)] = 0;
      }
      z += sm.bf[k];
      const float o = kPrecise ? sigmoidf<SIG>(z) : fmaf(0.5f, tanh_approx(0.5f * z), 0.5f);
      __syncwarp();
      // classify(): strict '<' scan from index 0, so the lowest index wins ties.
      float bv = __shfl_sync(0xffffffffu, o, li * 10);
      int best = 0;
#pragma unroll
      for (int kk = 1; kk < kOut; ++kk) {
        const float v = __shfl_sync(0xffffffffu, o, li * 10 + kk);
        if (bv < v) { bv = v; best = kk; }
      }
      if (active) {
        if (out) out[(img0 + img) * kOut + k] = o;
        if (argmax && k == 0) argmax[img0 + img] = best;
      }
      __syncwarp();
      if (lane == 0) *reinterpret_cast<volatile int*>(&sm.finished[warp]) = ++turn;   // these slots may be reused
      CNN_PHASE(2);
    }
  } else if (warp == kTfMmaWarp) {
    // ================= MMA issue: the whole warp runs the loop, one elected lane issues ============
    const unsigned idesc = tc::idesc_f16(128, kTfBN);
    // descriptors differ only in their 14-bit start-address field: base + (byte offset >> 4)
    const unsigned long long bd_hi = tc::smem_desc(smem_u32(sm.b_hi), kTfBChunk, 128);
    const unsigned long long bd_lo = tc::smem_desc(smem_u32(sm.b_lo), kTfBChunk, 128);
    for (int k = 0; k < n_tiles; ++k) {
      const int s = k % kTfSlabs, b = k % kTfAcc;
      CNN_PHASE(0);
      unsigned bytes = 0;
      const unsigned char* src = kPrecise ? nullptr : fetch_extent(k + kTfRaw, bytes);
      mbar_wait_bounded(&sm.a_full[s], (unsigned)(k / kTfSlabs) & 1u, status, gave_up);
      CNN_PHASE(1);
      // Issuing a bulk copy takes 300 cycles.  With one pass this warp has them to spare, with two or three the loaders do (path 2 by the
      // loaders: 94 instead of 91 us; path 1 by this warp: 118 instead of 116).
      if (!kPrecise && lane == 0 && k + kTfRaw < n_tiles) fetch(k + kTfRaw, src, bytes);     // the loaders are done with tile k's buffer
      __syncwarp();
      CNN_PHASE(2);
      const bool low = kLow && *reinterpret_cast<const volatile unsigned*>(sm.has_low[s]) != 0;
      const unsigned long long ad_hi = tc::smem_desc(smem_u32(sm.slab[s]), kTfChunkStride, kTfGroupStride);
      const unsigned long long ad_lo = tc::smem_desc(smem_u32(sm.slab[(s + kTfSlabsTotal / 2) % kTfSlabsTotal]), kTfChunkStride, kTfGroupStride);
      const unsigned d_tile = tmem_base + (unsigned)(b * kTfDCols);
      // Four roles share this SM's instruction cache, so the loop over the two column blocks stays rolled; the MMAs
      // of one block are written out (with dependent address arithmetic between two MMAs they cost 76-91 cycles
      // each instead of 53).
#pragma unroll 1
      for (int xb = 0; xb < 2; ++xb) {
        // The two column blocks of an accumulator are handed over and freed one by one: while an epilogue group works on
        // the second block of its tile, the first block of its next tile (three tiles on) is computed, so it never
        // waits for its own MMAs.
        mbar_wait_bounded(&sm.d_free[2 * b + xb], ((unsigned)(k / kTfAcc) & 1u) ^ 1u, status, gave_up);
        __syncwarp();
        tc::fence_after_sync();
        const unsigned d_blk = d_tile + (unsigned)(xb * kTfBN);
        const unsigned a_blk = ((unsigned)(2 * xb) * kTfChunkStride) >> 4;
#pragma unroll
        for (int pass = 0; pass < (kPrecise ? 3 : 1); ++pass) {
          if (pass == 2 && !low) continue;
          const unsigned long long a_d = ((pass == 2) ? ad_lo : ad_hi) + a_blk;
          const unsigned long long b_d = (pass == 1) ? bd_lo : bd_hi;
#pragma unroll
          for (int i = 0; i < 5; ++i)
            tc::mma_f16_elect(d_blk, a_d + (unsigned)i, b_d + (unsigned)i * (kTfBRow >> 4), idesc, (pass | i) ? 1u : 0u);
        }
        tc::mma_commit_elect(&sm.d_full[2 * b + xb]);    // the block is complete ...
      }
      tc::mma_commit_elect(&sm.a_free[s]);               // ... and after both the slab may be overwritten
      CNN_PHASE(3);
    }
  } else if (loader) {
    // ================= loaders: image rows -> operand slabs ==========================================
    // A thread converts eight pixels (one column chunk) of six rows of one group: rows j + 4 * sub (j < 4), j + 4 + 2 * sub (j = 4, 5).  Eight
    // consecutive lanes are the four chunks of two rows, four rows apart as a rule: neither their 16-byte loads (rows of 28 floats) nor
    // their stores meet in a bank then (two rows that are neighbours took two turns per load: 200 cycles per tile).
    typedef typename std::conditional<U8, unsigned, float4>::type Piece;     // four pixels
    const int chunk = lane & 3, sub = (lane >> 2) & 1, group = 4 * (warp - kTfLoadWarp0) + (lane >> 3);
    const int column = 2 * chunk - (chunk >> 1);                              // columns 0, 8, 12, 20
    const unsigned slab_at = (unsigned)chunk * kTfChunkStride + (unsigned)(group * kTfGroupRows) * 16u;
    auto row_of = [&](int j) { return j < 4 ? j + 4 * sub : j + 4 + 2 * sub; };
    // uint8 pixels: fp16 1024 + pixel is the byte below 0x64; times 2^e1, minus 1024 * 2^e1, is exact; 2^e2 (as a rule 1) finishes the scale where
    // fp16 could not hold its factors, and rounds, overflows or vanishes as the conversion of an fp32 image's scaled pixel does.
    const int e1 = min(max(wexp - 3, -24), 5), e2 = min(max(wexp - 3 - e1, -25), 15);
    const __half2 s1 = __float2half2_rn(__int_as_float((127 + e1) << 23)), s2 = __float2half2_rn(__int_as_float((127 + e2) << 23));
    const __half2 base1 = __float2half2_rn(-1024.f * __int_as_float((127 + e1) << 23));
    const f32x2 px_scale2 = pack2(px_scale, px_scale);
    unsigned stale = 0;      // slabs whose low part, this warp's share of it, is not all zeros
    bool expect_low = false;
    for (int k = 0; k < n_tiles; ++k) {
      const int s = k % kTfSlabs, r = k % kTfRaw;
      CNN_PHASE(0);
      mbar_wait_bounded(&sm.raw_full[r], (unsigned)(k / kTfRaw) & 1u, status, gave_up);
      CNN_PHASE(1);
      mbar_wait_bounded(&sm.a_free[s], ((unsigned)(k / kTfSlabs) & 1u) ^ 1u, status, gave_up);
      CNN_PHASE(2);
      // Groups past the last image read what the buffer held before: their output rows are never looked at.
      const Piece* raw = reinterpret_cast<const Piece*>(sm.raw[r]) + (group_pixel(k * kTfGroups + group) - group_pixel(k * kTfGroups)) / 4 + column;
      const bool live = k * kTfGroups + group < n_groups;
      unsigned char* hi_s = sm.slab[s];
      unsigned char* lo_s = sm.slab[(s + kTfSlabsTotal / 2) % kTfSlabsTotal];
      float top = 0.f;
      // Stores the high parts and, LOW, the low parts; says whether some pixel of this thread's has (or, without LOW, may have) a remainder.
      auto convert = [&](auto low_too) {
        [[maybe_unused]] constexpr bool LOW = decltype(low_too)::value;
        unsigned bits = 0;
        Piece v[kTfUnits][2];
#pragma unroll
        for (int j = 0; j < kTfUnits; ++j) {
          const Piece* p = raw + row_of(j) * (kH / 4);
          v[j][0] = p[0];
          v[j][1] = p[1];
        }
#pragma unroll
        for (int j = 0; j < kTfUnits; ++j) {
          unsigned hi[4];
          const unsigned o = slab_at + (unsigned)row_of(j) * 16u;
          if constexpr (U8) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const unsigned two = __byte_perm(v[j][c >> 1], 0x64646464u, (c & 1) ? 0x4342 : 0x4140);
              __half2 x = __hfma2(*reinterpret_cast<const __half2*>(&two), s1, base1);
              if (e2 != 0) x = __hmul2(x, s2);
              hi[c] = *reinterpret_cast<unsigned*>(&x);
            }
          } else {
            float x[8], big = 0.f;
            unpack2(mul2(pack2(v[j][0].x, v[j][0].y), px_scale2), x[0], x[1]);
            unpack2(mul2(pack2(v[j][0].z, v[j][0].w), px_scale2), x[2], x[3]);
            unpack2(mul2(pack2(v[j][1].x, v[j][1].y), px_scale2), x[4], x[5]);
            unpack2(mul2(pack2(v[j][1].z, v[j][1].w), px_scale2), x[6], x[7]);
            [[maybe_unused]] unsigned lo[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const __half2 h = __floats2half2_rn(x[2 * c], x[2 * c + 1]);
              hi[c] = *reinterpret_cast<const unsigned*>(&h);
              big = max_abs_nan(big, x[2 * c], x[2 * c + 1]);
              if constexpr (LOW) {
                const float2 b = __half22float2(h);
                const __half2 l = __floats2half2_rn(x[2 * c] - b.x, x[2 * c + 1] - b.y);
                lo[c] = *reinterpret_cast<const unsigned*>(&l);
                bits |= lo[c];
              } else {
                bits |= (__float_as_uint(x[2 * c]) | __float_as_uint(x[2 * c + 1])) & 0x1fffu;      // eleven significant bits leave no remainder
              }
            }
            if constexpr (LOW) *reinterpret_cast<uint4*>(lo_s + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            if (live) top = max_abs_nan(top, big, big);
          }
          *reinterpret_cast<uint4*>(hi_s + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        }
        return bits != 0;
      };
      if constexpr (kLow) {
        // Without remainders (uint8 / 255, as image files have them) the low part is not multiplied; it is written only where it was not all zeros
        // before.  The tile before says which of the two conversions to try first.
        bool low = expect_low || __any_sync(0xffffffffu, convert(std::false_type()));
        if (low || ((stale >> s) & 1u)) {
          low = __any_sync(0xffffffffu, convert(std::true_type()));
          stale = (stale & ~(1u << s)) | ((unsigned)low << s);
        }
        expect_low = low;
        if (lane == 0) *reinterpret_cast<volatile unsigned char*>(&sm.has_low[s][warp - kTfLoadWarp0]) = low;
      } else {
        convert(std::false_type());
      }
      if constexpr (!U8) {
        // fp16 holds magnitudes below 65,520: a larger scaled pixel (or one that is not a number) marks the tile's images
        if (!(top < 65520.f)) {
          const int first = (k * kTfGroups) / kTfGroupsImg, last = (k * kTfGroups + kTfGroups - 1) / kTfGroupsImg;
          for (int im = first; im <= last; ++im)
            if (im < imgs_here) sm.out_of_range[im & (kTfRange - 1)] = 1;
        }
      }
      tc::fence_async_smem();    // generic-proxy writes -> visible to the tensor core's operand reads
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm.raw_free[r]);
        mbar_arrive(&sm.a_full[s]);
      }
      if (kPrecise && lt == 0 && k + kTfRaw < n_tiles) {
        unsigned bytes;
        const unsigned char* src = fetch_extent(k + kTfRaw, bytes);
        mbar_wait_bounded(&sm.raw_free[r], (unsigned)(k / kTfRaw) & 1u, status, gave_up);
        fetch(k + kTfRaw, src, bytes);
      }
      __syncwarp();
      CNN_PHASE(3);
    }
  } else if (warp >= kTfEpiWarp0) {
    // ================= epilogue ====================================================================
    const int group = (warp - kTfEpiWarp0) >> 2;   // accumulator / tile residue this group owns
    const int quarter = warp & 3;                  // tensor-memory lanes 32 * quarter ..
    const int rsub = lane & 3;                     // row of the 4x4 window
    f32x2 ws2[4], bc2[kF / 2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float w = (kPrecise ? 1.0f : 0.5f) * sm.ws[rsub * 4 + j];
      ws2[j] = pack2(w, w);
    }
#pragma unroll
    for (int f = 0; f < kF; f += 2) bc2[f / 2] = pack2(sm.bc[f], sm.bc[f + 1]);
    const f32x2 unscale2 = pack2(w_unscale, w_unscale), one2 = pack2(1.f, 1.f);
    // path 2: sum_j ws * (0.5 + 0.5 t) = sum_j (0.5 ws) t + 0.5 * sum(ws); the constant goes into the bias
    float bs_eff = sm.bs[0];
    if (!kPrecise) {
      float sw = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) sw += sm.ws[j];
      bs_eff = fmaf(0.5f, sw, bs_eff);
    }
    const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;

    for (int k = group; k < n_tiles; k += kTfAcc) {
      CNN_PHASE(0);
      const int g = k * kTfGroups + quarter * 4 + (lane >> 3);     // group of 8 output rows this lane's row belongs to
      const int img_l = g / kTfGroupsImg;
      const int p = 2 * (g - img_l * kTfGroupsImg) + ((lane >> 2) & 1);   // window row
      const bool valid = img_l < imgs_here;
      const unsigned t0 = tmem_base + (unsigned)(group * kTfDCols) + ((unsigned)(quarter * 32) << 16);
      const int slot = img_l & (kTfSlots - 1);
      {   // the slots of this quarter's two or three images are free again: the images that had them, kTfSlots ago, lie in
          // the triple of the last one and the triple before it, of different finisher warps
        const int t = ((k * kTfGroups + quarter * 4 + 3) / kTfGroupsImg - kTfSlots) / 3;
        if (k * kTfGroups + quarter * 4 + 3 >= kTfGroupsImg * kTfSlots) {
          wait_counter_bounded(&sm.finished[t % kTfFinishers], t / kTfFinishers + 1, status, gave_up);
          if (t > 0) wait_counter_bounded(&sm.finished[(t - 1) % kTfFinishers], (t - 1) / kTfFinishers + 1, status, gave_up);
        }
      }
      // after the reduce-scatter lane r = rsub holds sums 9 (r & 1) + 5 (r >> 1) + i of a block, i < 5 - (r >> 1)
      float* as_dst = &sm.as[slot][p * 36 + (b0 ? 9 : 0) + (b1 ? 5 : 0)];
      CNN_PHASE(1);
      // (the column-block loop stays rolled to keep the epilogue's code inside the instruction cache)
#pragma unroll 1
      for (int xb = 0; xb < 2; ++xb) {              // one 12-column block = three window columns
        mbar_wait_bounded(&sm.d_full[2 * group + xb], (unsigned)(k / kTfAcc) & 1u, status, gave_up);
        if (xb == 0) CNN_PHASE(2); else CNN_PHASE(5);
        __syncwarp();
        tc::fence_after_sync();
        unsigned nxt[8];
        tc::tmem_ld8_nowait(t0 + (unsigned)(xb * kTfBN), nxt);
        tc::tmem_wait8(nxt);
        float z[18];
        f32x2 d2[4];               // the row's four activations before the reciprocal (of two maps), one step behind
        // Step ch turns 8 accumulator columns (window column ch / 3, maps 2 * (ch % 3) + {0, 1}) into exponentials and
        // finishes the columns of step ch - 1, so that two chains of dependent instructions are always under way.
#pragma unroll
        for (int ch = 0; ch < 10; ++ch) {
          f32x2 e2[4];
          if (ch < 9) {
            if (ch > 0) tc::tmem_wait8(nxt);
            // the window row's four columns of two maps: t = unscale * acc + bias
#pragma unroll
            for (int j = 0; j < 4; ++j)
              e2[j] = fma2(pack2(__uint_as_float(nxt[2 * j]), __uint_as_float(nxt[2 * j + 1])), unscale2, bc2[ch % 3]);
            if (ch < 8) {
              tc::tmem_ld8_nowait(t0 + (unsigned)(xb * kTfBN + (ch + 1) * 8), nxt);
            } else {
              // the last columns of this block are in registers: hand it back to the MMA warp
              tc::fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&sm.d_free[2 * group + xb]);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, y;
              unpack2(e2[j], x, y);
              if (kShort) e2[j] = pack2(exp2f_approx(fminf(x, kTfMaxExp)), exp2f_approx(fminf(y, kTfMaxExp)));
              else if (kPrecise) e2[j] = pack2(sigmoidf<SIG>(x), sigmoidf<SIG>(y));
              else e2[j] = pack2(tanh_approx(x), tanh_approx(y));
            }
          }
          if (ch > 0) {
            f32x2 z2;
            if constexpr (kShort) {
              // sum_j ws_j / d_j with d_j = 1 + 2^t_j over one common denominator: one reciprocal for four activations
              // (the special-function unit would bound the kernel: 1.25 operations per activation instead of 2).
              // t is capped at 31 so that the product of four stays finite: an activation below 4.7e-10 counts as 4.7e-10,
              // far below the rounding of the sum it enters.
              const f32x2 d01 = mul2(d2[0], d2[1]), d23 = mul2(d2[2], d2[3]);
              float x, y;
              unpack2(mul2(d01, d23), x, y);
              const f32x2 n01 = fma2(ws2[0], d2[1], mul2(ws2[1], d2[0])), n23 = fma2(ws2[2], d2[3], mul2(ws2[3], d2[2]));
              z2 = mul2(pack2(rcp_approx(x), rcp_approx(y)), fma2(n01, d23, mul2(n23, d01)));
            } else {
              z2 = fma2(ws2[3], d2[3], fma2(ws2[2], d2[2], fma2(ws2[1], d2[1], mul2(ws2[0], d2[0]))));
            }
            unpack2(z2, z[2 * (ch - 1)], z[2 * (ch - 1) + 1]);    // sums 6 * (window column) + map
          }
          if (ch < 9) {
#pragma unroll
            for (int j = 0; j < 4; ++j) d2[j] = kShort ? add2(e2[j], one2) : e2[j];
          }
        }
        if (xb == 0) CNN_PHASE(3); else CNN_PHASE(6);
        // ---- the window's four rows are lanes 4g..4g+3: reduce-scatter the block's 18 sums -----------
        // step 1 (lane bit 0): 9 each; step 2 (lane bit 1): 5 / 4 (+ one empty slot)
        float w9[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const float send = b0 ? z[i] : z[i + 9];
          const float keep = b0 ? z[i + 9] : z[i];
          w9[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
        float u[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const float hi9 = (i < 4) ? w9[i + 5] : 0.f;
          const float send = b1 ? w9[i] : hi9;
          const float keep = b1 ? hi9 : w9[i];
          u[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
        // ---- subsample sigmoid into the image's slot ----------------------------------------------------
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const float zs = u[i] + bs_eff;
          const float as = kPrecise ? sigmoidf<SIG>(zs) : fmaf(0.5f, tanh_approx(0.5f * zs), 0.5f);
          if (valid && (i < 4 || !b1)) as_dst[18 * xb + i] = as;
        }
        if (xb == 0) CNN_PHASE(4); else CNN_PHASE(7);
      }
      __syncwarp();
      if (valid && rsub == 0) mbar_arrive(&sm.img_done[slot]);   // one of the image's six window rows (release)
      CNN_PHASE(8);
    }
  }
  CNN_PHASE_END(g_phase_clocks_tc);

  tc::fence_before_sync();
  __syncthreads();
  if (warp == kTfMmaWarp) tc::tmem_dealloc(tmem_base, 512);
}

template <int PATH, int SIG, bool U8>
static int launch_forward_tc(cnn_net* net, const void* d_images, long n, float* d_out, int* d_argmax,
                             cudaStream_t stream) {
  // Every CTA owns a contiguous range of whole images (an image's window rows meet in shared memory).
  long grid = sm_count();
  const long min_imgs = 16;
  if (grid * min_imgs > n) grid = (n + min_imgs - 1) / min_imgs;
  const long per_cta = (n + grid - 1) / grid;
  grid = (n + per_cta - 1) / per_cta;
  const size_t smem = sizeof(TfSmem) + 128;
  CNN_CUDA(cudaFuncSetAttribute(k_forward_tc<PATH, SIG, U8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaError_t e = launch_pdl(k_forward_tc<PATH, SIG, U8>, dim3((unsigned)grid), dim3(kTfThreads), smem, stream, d_images, n,
                             per_cta, (const float*)net->d_params, d_out, d_argmax, net->d_status);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_forward_tc launch");
  return CNN_OK;
}

int forward_device_tc(cnn_net* net, int path, const float* d_images, long n, float* d_out, int* d_argmax,
                      cudaStream_t stream) {
  if (path == 2) return launch_forward_tc<2, 2, false>(net, d_images, n, d_out, d_argmax, stream);
  // Path 1 with fast_sigmoid set uses the short sigmoid form (ex2.approx, rcp.approx): over the 65,536 images of
  // benchmark configuration 2 the outputs are as close to the oracle with it as with the refined form.
  return net->fast_sigmoid ? launch_forward_tc<1, 1, false>(net, d_images, n, d_out, d_argmax, stream)
                           : launch_forward_tc<1, 0, false>(net, d_images, n, d_out, d_argmax, stream);
}

int forward_device_tc_u8(cnn_net* net, const unsigned char* d_pixels, long n, float* d_out, int* d_argmax,
                         cudaStream_t stream) {
  return net->fast_sigmoid ? launch_forward_tc<1, 1, true>(net, d_pixels, n, d_out, d_argmax, stream)
                           : launch_forward_tc<1, 0, true>(net, d_pixels, n, d_out, d_argmax, stream);
}

}  // namespace cnn

#ifdef CNN_PHASE_CLOCKS
// Sums of the SM clock at each stamp for the 20 warps of CTA 0 of the last launch (tuning builds only).
extern "C" int cnn_debug_phase_clocks_tc(long long* out /* [20][16] */) {
  return cudaMemcpyFromSymbol(out, cnn::g_phase_clocks_tc, sizeof(cnn::g_phase_clocks_tc)) == cudaSuccess ? 0 : 2;
}
#endif
