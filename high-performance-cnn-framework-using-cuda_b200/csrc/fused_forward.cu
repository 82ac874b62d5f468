// Fused batched forward: conv 6x5x5 + bias + sigmoid, shared 4x4/stride-4 subsample + bias +
// sigmoid, FC 216->10 + bias + sigmoid and argmax in ONE kernel.  Replaces, for n images at once,
// the reference's forward_pass launch sequence (main.cu:67-88: 8 memsets, one H2D copy and nine
// <<<64,64>>> launches per image) and classify's D2H + host argmax (main.cu:181-189).
//
// Exact fp32 on the CUDA cores: batches below kTcMinBatch images, and whatever asks for it.  Two maps at a time sit in the
// halves of packed fp32 registers throughout: a packed FMA takes two cycles of the FMA pipe but one issue slot, which
// leaves the other slots to everything else.  Images are contiguous 3,136-byte records that come into shared memory by
// 1-D bulk copies (cp.async.bulk, no multicast), double-buffered behind mbarriers; the only other HBM traffic is the 44
// bytes of results per image.  Two kernels share the work by size (forward_kernel_for):
//
//  * k_forward_one, a few hundred images at most: one image per block and turn, so that an image is as short a chain as
//    possible.  Thread (window, map pair, half) owns two rows of a 4x4 subsample window for two maps: 8 x 2 conv
//    outputs on a 6x8 patch, 200 packed FMAs, the 25 tap pairs in registers for the whole launch.  The two halves of a window
//    meet in one shuffle, each computes five of the ten FC partial sums, which are added up over the warp by a
//    shuffle reduce-scatter and over the block's seven warps through shared memory.  Bound by the chain launch -
//    parameters - patch - 25 x 8 FMAs - two sigmoids - sums - sigmoid: 1 image 10.2 -> 4.0 us, 300 images 10.6 -> 4.4 us
//    (before: the next kernel's shape at every size, scalar; until 4.5 us the parameters were loaded in several groups, one wait for L2 each).
//  * k_forward_tiles: tiles of up to seven images, thread = window for all six maps (three packed pairs one after another), FC
//    partial sums in registers, one barrier pair per tile.  Bound by the FMA pipe (92,016 FMAs = 719 SM-cycles per
//    image; 65 % of it at 6,143 images): 1,000 images 10.5 -> 6.6 us (tiles of equal length), 2,000 images 16.4 -> 10.5 us, 6,143 images
//    34.9 -> 26.5 us (scalar FMAs on a patch in registers before).
#include "net.cuh"

namespace cnn {

constexpr int kFwPairs = kF / 2;                              // map pairs
constexpr int kFwLive = 36 * kFwPairs * 2;                    // 216 threads with work
constexpr int kFwThreads = (kFwLive + 31) / 32 * 32;          // 224 = 7 warps
constexpr int kFwWarps = kFwThreads / 32;
constexpr int kFwBlocksPerSm = 2;
constexpr int kFwStages = 2;
constexpr int kForwardOne = 3;             // what forward_kernel_for calls k_forward_one

struct FwSmem {
  alignas(16) float img[kFwStages][kImg];   // filled by bulk copies (uint8 pixels: the first quarter)
  alignas(16) float pix[kImg];              // uint8 input only: the current image as fp32
  alignas(16) float wf[kOut][36][kF];       // FC weights as [k][window][map]: a pair is one 64-bit read
  alignas(8) float wc[25][kF];                       // taps as [tap][map]
  alignas(16) float ws[16];                 // read 16 bytes at a time
  alignas(8) float bc[8];                   // read as pairs
  float bs[4], bf[12];
  float part[2][kFwWarps][12];              // FC sums of a warp, by parity of the turn: outputs 0..4 at 0..4, 5..9 at 6..10
  float lut[256];                           // uint8 pixel -> float(pixel / 255.0), uint8 input only
  unsigned long long full[kFwStages];
};

// U8 = false: images are fp32 [n][28][28].  U8 = true: `images` points at uint8 pixels [n][28][28]
// (the storage of the IDX files the reference reads) and the kernel applies the reference's ingest,
// float(pixel / 255.0) (mnist.h:145 then main.cu:57-65), through a 256-entry table.
template <int FAST, bool U8>
__global__ void __launch_bounds__(kFwThreads, kFwBlocksPerSm)
k_forward_one(const void* images, long n, const float* params,
                float* __restrict__ out, int* __restrict__ argmax, int* __restrict__ status) {
  __shared__ FwSmem sm;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // With the short sigmoid form its multiplication by -log2(e) is folded into the conv weights and bias.
  constexpr float kPre = (FAST == 1) ? -1.4426950408889634f : 1.0f;
  constexpr unsigned kImageBytes = (U8 ? 1u : 4u) * (unsigned)kImg;

  pdl_launch_dependents();
  auto issue = [&](int stage, long im) {
    mbar_expect_tx(&sm.full[stage], kImageBytes);
    bulk_g2s(&sm.img[stage][0], static_cast<const unsigned char*>(images) + (size_t)im * kImageBytes, kImageBytes, &sm.full[stage]);
  };
  if (tid == 0) {
    for (int s = 0; s < kFwStages; ++s) mbar_init(&sm.full[s], 1);
    mbar_fence_init();
  }
  if (U8)
    for (int i = tid; i < 256; i += kFwThreads) sm.lut[i] = (float)((double)i / 255.0);
  pdl_wait();
  if (tid == 0) {
    for (int s = 0; s < kFwStages; ++s) {
      const long im = (long)blockIdx.x + (long)s * gridDim.x;
      if (im < n) issue(s, im);
    }
  }
  // Parameters: 9.4 KB, L2-resident after the first block.  Every load of a thread is under way before the first is stored (one wait for L2).
  {
    const int at = tid < kS ? tid : kS - 1;
    float wf[kOut];
#pragma unroll
    for (int k = 0; k < kOut; ++k) wf[k] = params[kOffWf + k * kS + at];
    const float small = params[tid < kOffWf ? tid : kOffBf + (tid - kOffWf < kOut ? tid - kOffWf : 0)];
    if (tid < kS) {
#pragma unroll
      for (int k = 0; k < kOut; ++k) sm.wf[k][tid % 36][tid / 36] = wf[k];
    }
    if (tid < kOffBc) sm.wc[tid % 25][tid / 25] = kPre * small;
    else if (tid < kOffWs) sm.bc[tid - kOffBc] = kPre * small;
    else if (tid < kOffBs) sm.ws[tid - kOffWs] = small;
    else if (tid == kOffBs) sm.bs[0] = small;
    else if (tid < kOffWf + kOut) sm.bf[tid - kOffWf] = small;
  }
  __syncthreads();

  // thread -> (window, pair, half): half fastest, so that a window's halves are neighbouring lanes
  const bool live = tid < kFwLive;
  const int half = tid & 1, unit = (live ? tid : 0) >> 1;
  // (the order of the windows keeps eight neighbouring threads' 16-byte reads out of one another's banks: see k_grad_partials)
  const int pr = unit / 36, twelve = unit % 36 / 12, quad = unit % 12 / 4, in_quad = unit % 4;
  const int p = 2 * twelve + (quad < 2 ? quad : in_quad >> 1), q = quad < 2 ? in_quad + (in_quad & 2) : 2 + (in_quad & 1);
  const int w = 6 * p + q;
  f32x2 wt[25];
#pragma unroll
  for (int t = 0; t < 25; ++t) wt[t] = *reinterpret_cast<const f32x2*>(&sm.wc[t][2 * pr]);
  const f32x2 bias2 = *reinterpret_cast<const f32x2*>(&sm.bc[2 * pr]);
  bool gave_up = false;

  int it = 0;
  for (long im = blockIdx.x; im < n; im += gridDim.x, ++it) {
    const int stage = it % kFwStages;
    mbar_wait_bounded(&sm.full[stage], (unsigned)(it / kFwStages) & 1u, status, gave_up);
    const float* img = &sm.img[stage][0];
    if constexpr (U8) {
      // the previous image's patches were read before the barrier of its turn
      if (tid < kImg / 4) {
        const unsigned v = reinterpret_cast<const unsigned*>(&sm.img[stage][0])[tid];
        *reinterpret_cast<float4*>(&sm.pix[4 * tid]) =
            make_float4(sm.lut[v & 0xFFu], sm.lut[(v >> 8) & 0xFFu], sm.lut[(v >> 16) & 0xFFu], sm.lut[v >> 24]);
      }
      __syncthreads();
      img = sm.pix;
    }
    const float* base = img + (4 * p + 2 * half) * kH + 4 * q;

    f32x2 acc[2][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) acc[0][x] = acc[1][x] = bias2;
#pragma unroll
    for (int r = 0; r < 6; ++r) {          // patch rows: eight pixels, each in both halves of a register pair
      const float4 lo = *reinterpret_cast<const float4*>(base + r * kH), hi = *reinterpret_cast<const float4*>(base + r * kH + 4);
      const f32x2 v[8] = {pack2(lo.x, lo.x), pack2(lo.y, lo.y), pack2(lo.z, lo.z), pack2(lo.w, lo.w),
                          pack2(hi.x, hi.x), pack2(hi.y, hi.y), pack2(hi.z, hi.z), pack2(hi.w, hi.w)};
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int i = r - y;               // tap row
        if (i < 0 || i > 4) continue;
#pragma unroll
        for (int j = 0; j < 5; ++j)
#pragma unroll
          for (int x = 0; x < 4; ++x) acc[y][x] = fma2(wt[i * 5 + j], v[x + j], acc[y][x]);
      }
    }
    f32x2 z = pack2(0.f, 0.f);
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      const float4 wrow = *reinterpret_cast<const float4*>(&sm.ws[4 * (2 * half + y)]);
      const float ws[4] = {wrow.x, wrow.y, wrow.z, wrow.w};
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float u0, u1;
        unpack2(acc[y][x], u0, u1);
        const f32x2 a = (FAST == 1) ? pack2(rcp_approx(1.0f + exp2f_approx(u0)), rcp_approx(1.0f + exp2f_approx(u1)))
                                    : pack2(sigmoidf<FAST>(u0), sigmoidf<FAST>(u1));
        z = fma2(pack2(ws[x], ws[x]), a, z);
      }
    }
    float z0, z1;
    unpack2(z, z0, z1);
    z0 += __shfl_xor_sync(0xffffffffu, z0, 1);
    z1 += __shfl_xor_sync(0xffffffffu, z1, 1);
    const float as0 = live ? sigmoidf<FAST>(z0 + sm.bs[0]) : 0.f, as1 = live ? sigmoidf<FAST>(z1 + sm.bs[0]) : 0.f;
    // FC: output 5 half + j of this window and pair, added over the warp's 16 windows and pairs (lane bits 4 and 3 pick
    // two of the eight values, bits 2 and 1 the rest of the sum)
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = 0.f;
      if (j < 5) {
        const float2 wk = *reinterpret_cast<const float2*>(&sm.wf[5 * half + j][w][2 * pr]);
        v[j] = fmaf(wk.x, as0, wk.y * as1);
      }
    }
#pragma unroll
    for (int keep = 4; keep >= 1; keep >>= 1) {
      const int mask = keep << 2;          // 16, 8, 4
      const bool upper = (lane & mask) != 0;
#pragma unroll
      for (int i = 0; i < keep; ++i) {
        const float send = upper ? v[i] : v[i + keep], mine = upper ? v[i + keep] : v[i];
        v[i] = mine + __shfl_xor_sync(0xffffffffu, send, mask);
      }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    const int j = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    float (&part)[kFwWarps][12] = sm.part[it & 1];
    if ((lane & 2) == 0 && j < 5) part[warp][6 * half + j] = v[0];
    __syncthreads();    // the sums are in shared memory, and every thread has taken its patch: the stage may be refilled
    if (tid == 0) {
      const long next = im + (long)kFwStages * gridDim.x;
      if (next < n) issue(stage, next);
    }
    // one warp per turn finishes the image while the others go on (the sums alternate with the turn's parity: a warp is
    // never two barriers ahead of another)
    if (warp == it % kFwWarps) {
      float o = 0.f;
      if (lane < kOut) {
        float s = 0.f;
#pragma unroll
        for (int ww = 0; ww < kFwWarps; ++ww) s += part[ww][lane < 5 ? lane : lane + 1];
        o = sigmoidf<FAST>(s + sm.bf[lane]);
      }
      // classify(): strict '<' scan from index 0, so the lowest index wins ties.
      float bv = __shfl_sync(0xffffffffu, o, 0);
      int best = 0;
#pragma unroll
      for (int kk = 1; kk < kOut; ++kk) {
        const float u = __shfl_sync(0xffffffffu, o, kk);
        if (bv < u) { bv = u; best = kk; }
      }
      if (lane < kOut && out) out[im * kOut + lane] = o;
      if (lane == 0 && argmax) argmax[im] = best;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Tiles of seven images: 252 of a block's 256 threads own a window, and two 8-warp blocks per SM may use 128 registers
// per thread.  (Eight images = 288 threads are allocated as ten warps, which caps two blocks per SM at 96 registers.)
constexpr int kFtImgs = 7;                                    // images per tile
constexpr int kFtThreads = (kFtImgs * 36 + 31) / 32 * 32;     // 256 = 8 warps
constexpr int kFtBlocksPerSm = 2;
constexpr int kFtPartStride = 37;           // 36 windows + 1 pad: conflict-free column reads
constexpr int kFtTaps = 26;                 // 25 tap pairs, padded to an even number for 128-bit reads

struct FtSmem {
  alignas(16) float img[kFwStages][kFtImgs][kImg];   // filled by bulk copies; uint8 pixels: [0] the tile as fp32, [1] both raw tiles
  alignas(16) float wc[kFwPairs][kFtTaps][2];        // tap pairs
  alignas(16) float ws[16][2];                       // subsample taps, both halves
  alignas(16) float wf[kFwPairs][36][2][12];         // FC weights as [pair][window][map of the pair][output]
  float bc[8], bs[4], bf[12];
  float part[2][kFtImgs][kOut][kFtPartStride];       // by parity of the turn
  float lut[256];                                    // uint8 pixel -> float(pixel / 255.0), uint8 input only
  unsigned long long full[kFwStages];
};

// ONE_ROUND: a tile per block, per_tile images each and one more in the first `more`; otherwise tiles of seven, the last one of what is left.
template <int FAST, bool U8, bool ONE_ROUND>
__global__ void __launch_bounds__(kFtThreads, kFtBlocksPerSm)
k_forward_tiles(const void* images, long n, int per_tile, int more, const float* params,
                float* __restrict__ out, int* __restrict__ argmax, int* __restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  FtSmem& sm = *reinterpret_cast<FtSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long n_tiles = ONE_ROUND ? gridDim.x : (n + kFtImgs - 1) / kFtImgs;
  auto first_of = [&](long tile) -> long { return ONE_ROUND ? tile * per_tile + (tile < more ? tile : more) : tile * kFtImgs; };
  auto count_of = [&](long tile) -> int {
    if (ONE_ROUND) return per_tile + (tile < more ? 1 : 0);
    const long left = n - tile * kFtImgs;
    return left < kFtImgs ? (int)left : kFtImgs;
  };
  constexpr float kPre = (FAST == 1) ? -1.4426950408889634f : 1.0f;
  constexpr unsigned kImageBytes = (U8 ? 1u : 4u) * (unsigned)kImg;

  pdl_launch_dependents();
  auto raw = [&](int stage) -> unsigned char* {
    return U8 ? reinterpret_cast<unsigned char*>(&sm.img[1][0][0]) + stage * (kFtImgs * kImg) : reinterpret_cast<unsigned char*>(&sm.img[stage][0][0]);
  };
  auto issue = [&](int stage, long tile) {
    const long first = first_of(tile);
    const unsigned bytes = (unsigned)count_of(tile) * kImageBytes;
    mbar_expect_tx(&sm.full[stage], bytes);
    bulk_g2s(raw(stage), static_cast<const unsigned char*>(images) + (size_t)first * kImageBytes, bytes, &sm.full[stage]);
  };
  if (tid == 0) {
    for (int s = 0; s < kFwStages; ++s) mbar_init(&sm.full[s], 1);
    mbar_fence_init();
  }
  if (U8) sm.lut[tid] = (float)((double)tid / 255.0);
  pdl_wait();
  if (tid == 0) {
    for (int s = 0; s < kFwStages; ++s) {
      const long t = (long)blockIdx.x + (long)s * gridDim.x;
      if (t < n_tiles) issue(s, t);
    }
  }
  // Parameters: every load of a thread is under way before the first is stored (one wait for L2).
  {
    const int f = tid / 36, w = tid % 36, tap_f = tid / kFtTaps, tap = tid % kFtTaps;
    float wf[kOut];
#pragma unroll
    for (int k = 0; k < kOut; ++k) wf[k] = params[kOffWf + k * kS + (tid < kS ? tid : kS - 1)];
    const float taps = params[kOffWc + (tap_f < kF && tap < 25 ? tap_f * 25 + tap : 0)];
    const float small = params[tid < 216 ? 0 : (tid < 232 ? kOffWs + tid - 216 : (tid < 242 ? kOffBf + tid - 232 : (tid < 248 ? kOffBc + tid - 242 : kOffBs)))];
    if (tid < kS) {                       // 216 threads, ten FC weights each
      float* dst = sm.wf[f >> 1][w][f & 1];
#pragma unroll
      for (int k = 0; k < kOut; ++k) dst[k] = wf[k];
    } else if (tid < 232) {
      sm.ws[tid - 216][0] = sm.ws[tid - 216][1] = small;
    } else if (tid < 242) {
      sm.bf[tid - 232] = small;
    } else if (tid < 248) {
      sm.bc[tid - 242] = kPre * small;
    } else if (tid == 248) {
      sm.bs[0] = small;
    }
    if (tid < kF * kFtTaps) sm.wc[tap_f >> 1][tap][tap_f & 1] = (tap < 25) ? kPre * taps : 0.f;
  }
  __syncthreads();

  // Eight neighbouring threads read 16 bytes each at a time, of rows of seven: (4 p + q) mod 8 (plus 4 in every other image) is the bank group.  Twelve
  // threads own two rows of windows; columns 0-3 of both ask eight different ones, columns 4, 5 of both together with columns 2, 3 of the next
  // two rows, too, and what remains of those takes two turns: 4 turns for 24 windows, the least there is (in the windows' own order 6).
  const int twelve = tid / 12, t12 = tid % 12, img = twelve / 3;
  const bool odd12 = (twelve & 1) != 0;
  const int sub = t12 & 3, third = t12 >> 2;
  const int second_row = odd12 ? (third == 0 ? sub >> 1 : third - 1) : (third < 2 ? third : sub >> 1);
  const int q = odd12 ? (third == 0 ? 2 + (sub & 1) : sub + (sub & 2)) : (third < 2 ? sub : 4 + (sub & 1));
  const int p = 2 * (twelve % 3) + second_row, w = 6 * p + q;
  bool gave_up = false;
  int it = 0;
  for (long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++it) {
    const int stage = it % kFwStages;
    mbar_wait_bounded(&sm.full[stage], (unsigned)(it / kFwStages) & 1u, status, gave_up);
    const long first = first_of(tile);
    const int imgs_here = count_of(tile);
    const bool live = img < imgs_here;
    // Warps without an image leave the pipes to the others.  (uint8 pixels in several rounds: the test costs 2 %, and few warps have none.)
    const bool work = (U8 && !ONE_ROUND) || __any_sync(0xffffffffu, live);
    const int at = (live ? img : 0) * kImg + (4 * p) * kH + 4 * q;         // first pixel of the thread's patch
    if constexpr (U8) {                    // (the previous tile's patches were read before its barriers)
      const unsigned* src = reinterpret_cast<const unsigned*>(raw(stage));
      for (int i = tid; i < imgs_here * (kImg / 4); i += kFtThreads) {
        const unsigned v = src[i];
        reinterpret_cast<float4*>(&sm.img[0][0][0])[i] =
            make_float4(sm.lut[v & 0xFFu], sm.lut[(v >> 8) & 0xFFu], sm.lut[(v >> 16) & 0xFFu], sm.lut[v >> 24]);
      }
      __syncthreads();
    }

    f32x2 fc[kOut / 2];                    // pairs of outputs
#pragma unroll
    for (int k = 0; k < kOut / 2; ++k) fc[k] = pack2(0.f, 0.f);
#pragma unroll 1
    for (int pr = work ? 0 : kFwPairs; pr < kFwPairs; ++pr) {
      int again = at;                      // hidden from the compiler: keeping the 8x8 patch over the pairs would spill
      asm volatile("" : "+r"(again));
      const float* base = &sm.img[U8 ? 0 : stage][0][0] + again;
      f32x2 wt[kFtTaps], acc[4][4];
#pragma unroll
      for (int t = 0; t < kFtTaps; t += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(sm.wc[pr][t]);
        wt[t] = v.x; wt[t + 1] = v.y;
      }
      const f32x2 bias2 = pack2(sm.bc[2 * pr], sm.bc[2 * pr + 1]);
      f32x2 z = pack2(0.f, 0.f);
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] = bias2;
#pragma unroll
      for (int r = 0; r < 8; ++r) {        // patch rows: eight pixels, each in both halves of a register pair
        const float4 lo = *reinterpret_cast<const float4*>(base + r * kH), hi = *reinterpret_cast<const float4*>(base + r * kH + 4);
        const f32x2 v[8] = {pack2(lo.x, lo.x), pack2(lo.y, lo.y), pack2(lo.z, lo.z), pack2(lo.w, lo.w),
                            pack2(hi.x, hi.x), pack2(hi.y, hi.y), pack2(hi.z, hi.z), pack2(hi.w, hi.w)};
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          const int i = r - y;             // tap row
          if (i < 0 || i > 4) continue;
#pragma unroll
          for (int j = 0; j < 5; ++j)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[y][x] = fma2(wt[i * 5 + j], v[x + j], acc[y][x]);
        }
        // output row r - 4 is complete: its sigmoids (special-function unit) go under the next rows' FMAs
        if (r >= 4) {
          const int y = r - 4;
#pragma unroll
          for (int x = 0; x < 4; x += 2) {
            const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(sm.ws[4 * y + x]);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float u0, u1;
              unpack2(acc[y][x + e], u0, u1);
              const f32x2 a = (FAST == 1) ? pack2(rcp_approx(1.0f + exp2f_approx(u0)), rcp_approx(1.0f + exp2f_approx(u1)))
                                          : pack2(sigmoidf<FAST>(u0), sigmoidf<FAST>(u1));
              z = fma2(e == 0 ? w2.x : w2.y, a, z);
            }
          }
        }
      }
      float zz[2];
      unpack2(z, zz[0], zz[1]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float as = sigmoidf<FAST>(zz[e] + sm.bs[0]);
        const f32x2 as2 = pack2(as, as);
        const float* wr = sm.wf[pr][w][e];
        const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(wr), w1 = *reinterpret_cast<const ulonglong2*>(wr + 4);
        fc[0] = fma2(w0.x, as2, fc[0]); fc[1] = fma2(w0.y, as2, fc[1]); fc[2] = fma2(w1.x, as2, fc[2]);
        fc[3] = fma2(w1.y, as2, fc[3]); fc[4] = fma2(*reinterpret_cast<const f32x2*>(wr + 8), as2, fc[4]);
      }
    }
    if (live && tid < kFtImgs * 36) {
#pragma unroll
      for (int k = 0; k < kOut / 2; ++k) {
        float a, b;
        unpack2(fc[k], a, b);
        sm.part[it & 1][img][2 * k][w] = a;
        sm.part[it & 1][img][2 * k + 1][w] = b;
      }
    }
    __syncthreads();    // the sums are in shared memory, and every thread is done with its patch: the stage may be refilled
    if (tid == 0) {
      const long next = tile + (long)kFwStages * gridDim.x;
      if (next < n_tiles) issue(stage, next);
    }
    // Three warps in turn finish the tile while the others go on (the sums alternate with the turn's parity: a warp is
    // never two barriers ahead of another), three images each on lanes 0..29: lane = 10*local_image + k.
    const int fin = (warp + kFtThreads / 32 * 3 - 3 * it % (kFtThreads / 32)) % (kFtThreads / 32);
    if (fin < (kFtImgs + 2) / 3) {
      const int li = lane / 10, k = lane % 10;
      const int im = fin * 3 + li;
      const bool valid = (lane < 30) && (im < imgs_here);
      float z = 0.f;
      if (valid) {
        float zq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ww = 0; ww < 36; ++ww) zq[ww & 3] += sm.part[it & 1][im][k][ww];
        z = ((zq[0] + zq[1]) + (zq[2] + zq[3])) + sm.bf[k];
      }
      const float o = sigmoidf<FAST>(z);
      // classify(): strict '<' scan from index 0, so the lowest index wins ties.
      float bv = __shfl_sync(0xffffffffu, o, li * 10);
      int best = 0;
#pragma unroll
      for (int kk = 1; kk < kOut; ++kk) {
        const float v = __shfl_sync(0xffffffffu, o, li * 10 + kk);
        if (bv < v) { bv = v; best = kk; }
      }
      if (valid) {
        const long gi = first + im;
        if (out) out[gi * kOut + k] = o;
        if (argmax && k == 0) argmax[gi] = best;
      }
    }
  }
}

template <int FAST, bool U8>
static int launch_variant(cnn_net* net, int path, const void* d_images, long n, float* d_out, int* d_argmax,
                          cudaStream_t stream) {
  cudaError_t e;
  if (path == kForwardOne) {
    const long resident = (long)kFwBlocksPerSm * sm_count();
    e = launch_pdl(k_forward_one<FAST, U8>, dim3((unsigned)(n < resident ? n : resident)), dim3(kFwThreads), 0, stream, d_images, n,
                   (const float*)net->d_params, d_out, d_argmax, net->d_status);
  } else {
    // One round of tiles: a tile per block, of equal length to one image, because a round takes as long as its longest tile and warps without an image
    // leave the pipes to the others (tiles of seven: 889 images 10.5 us, 1,036 6.7, 1,184 10.5, 2,072 10.7; equal ones 6.5, 6.6, 8.7, 10.5).  Up to
    // seven images per SM that is a block on each SM: fewer would leave SMs idle that take two blocks of the next launch.  With more rounds
    // tiles of seven, but for the last one, are the better ones (2,500 images 14.4 against 16.2 us, 5,000 22.7 against 26.2; 3,000 18.9 against 17.7).
    const long sms = sm_count(), resident = kFtBlocksPerSm * sms;
    const bool one_round = n <= resident * kFtImgs;
    const long most = n <= sms * kFtImgs ? sms : resident, n_tiles = one_round ? (n < most ? n : most) : (n + kFtImgs - 1) / kFtImgs;
    const long grid = n_tiles < resident ? n_tiles : resident;
    auto* const kernel = one_round ? k_forward_tiles<FAST, U8, true> : k_forward_tiles<FAST, U8, false>;
    CNN_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FtSmem)));
    e = launch_pdl(kernel, dim3((unsigned)grid), dim3(kFtThreads), sizeof(FtSmem), stream, d_images, n, (int)(n / n_tiles), (int)(n % n_tiles),
                   (const float*)net->d_params, d_out, d_argmax, net->d_status);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fused forward launch");
  return CNN_OK;
}

// The kernel a call over n_total images uses: 0 = k_forward_tiles, kForwardOne = k_forward_one, 1 / 2 = forward_tc.cu.
// Default (-1): the tensor-core kernel in two or three passes for batches of kTcMinBatch images and more, this file's below.  The line is the one
// that the interface promises (the two sides differ in their last bits); it is not where the kernels meet.  That is at one round of
// tiles, 14 images per SM: 2,072 images 10.5 us here, 10.3 on the tensor cores; 2,073 images 11.9 and 10.3; 4,144: 18.6 and 13.8; 6,143: 26.5 and
// 16.7 (uint8: 10.8 / 9.5, 14.8 / 9.5, 20.8 / 12.7, 29.7 / 15.2).
// uint8 pixels follow the same rule, so that they give the same bits as the fp32
// images they stand for (the reduced-precision path 2 is for fp32 images only).  All keep the 1e-5 parity bar.
// With the reference's sigmoid expression asked for (fast_sigmoid = 0) the default stays in this file.
// One-image kernel / a tile on each SM, fp32 and uint8: 148 images 3.4 / 4.6 us and 3.3 / 4.6, 350 images 4.5 / 4.6 and 4.7 / 4.9, 444 images
// 5.7 / 4.7 and 5.8 / 4.9 (up to three images a tile's warps have a scheduler each), 445 images 5.7 / 6.1 and 5.8 / 6.7, 660 images 6.3 / 6.5 and
// 6.5 / 6.9, 700 images 7.3 / 6.5 and 7.7 / 6.9, 888 images 7.5 / 6.5 and 7.9 / 6.8: the lines lie at 2.5, 3 and 4.5 images per SM.
int forward_kernel_for(const cnn_net* net, long n_total, bool u8) {
  constexpr long kTcMinBatch = 6144;
  int path = net->forward_path;
  if (path < 0 || (u8 && path == 2)) path = (net->fast_sigmoid && n_total >= kTcMinBatch) ? 1 : 0;
  const long sms = sm_count();
  return (path == 0 && (2 * n_total <= 5 * sms || (n_total > 3 * sms && 2 * n_total <= 9 * sms))) ? kForwardOne : path;
}

// `path` as returned by forward_kernel_for: callers that cut a request into chunks decide once for the
// whole request, so that every image of it goes through the same kernel.
int forward_device(cnn_net* net, int path, const float* d_images, long n, float* d_out, int* d_argmax,
                   cudaStream_t stream) {
  if (path == 1 || path == 2) return forward_device_tc(net, path, d_images, n, d_out, d_argmax, stream);
  return net->fast_sigmoid ? launch_variant<1, false>(net, path, d_images, n, d_out, d_argmax, stream)
                           : launch_variant<0, false>(net, path, d_images, n, d_out, d_argmax, stream);
}

int forward_device_u8(cnn_net* net, int path, const unsigned char* d_pixels, long n, float* d_out, int* d_argmax,
                      cudaStream_t stream) {
  if (path == 1) return forward_device_tc_u8(net, d_pixels, n, d_out, d_argmax, stream);
  return net->fast_sigmoid ? launch_variant<1, true>(net, path, d_pixels, n, d_out, d_argmax, stream)
                           : launch_variant<0, true>(net, path, d_pixels, n, d_out, d_argmax, stream);
}

}  // namespace cnn

extern "C" int cnn_forward_batched(cnn_net* net, const float* d_images, long n, float* d_out,
                                   int* d_argmax, void* stream) {
  CNN_REQUIRE(net != nullptr, "cnn_forward_batched: NULL net");
  CNN_REQUIRE(n >= 0, "cnn_forward_batched: negative image count");
  if (n == 0) return CNN_OK;
  CNN_REQUIRE(d_images != nullptr, "cnn_forward_batched: NULL images");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_images) & 15u) == 0,
              "cnn_forward_batched: image batch must start on a 16-byte boundary");
  return cnn::forward_device(net, cnn::forward_kernel_for(net, n, false), d_images, n, d_out, d_argmax, cnn::as_stream(stream));
}

extern "C" int cnn_forward_batched_u8(cnn_net* net, const unsigned char* d_pixels, long n, float* d_out,
                                      int* d_argmax, void* stream) {
  CNN_REQUIRE(net != nullptr, "cnn_forward_batched_u8: NULL net");
  CNN_REQUIRE(n >= 0, "cnn_forward_batched_u8: negative image count");
  if (n == 0) return CNN_OK;
  CNN_REQUIRE(d_pixels != nullptr, "cnn_forward_batched_u8: NULL pixels");
  CNN_REQUIRE((reinterpret_cast<uintptr_t>(d_pixels) & 15u) == 0,
              "cnn_forward_batched_u8: pixel batch must start on a 16-byte boundary");
  return cnn::forward_device_u8(net, cnn::forward_kernel_for(net, n, true), d_pixels, n, d_out, d_argmax, cnn::as_stream(stream));
}
