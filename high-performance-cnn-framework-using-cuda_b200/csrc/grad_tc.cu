// Gradient of a large batch of the reference's 28x28 net with both contractions of the convolution -- forward (fp_preact_c1,
// layer.cu:116-133) and weight gradient (bp_weight_c1, layer.cu:363-381): 91 % of the step's MACs -- on the 5th-generation
// tensor cores, everything else (sigmoids, subsample, FC, error, deltas, the other gradients) in fp32 around them.
// One pass over the images, nothing of an image in HBM but its pixels: the tile's pre-activations stay in tensor memory from the
// convolution until the deltas are done.
//
// A tile is five images: M = 128 of 16 groups of eight output rows, of which 15 are used (three per image), each with the twelve input
// rows it needs, as in forward_tc.cu.  The operand is kept in column chunks of eight fp16 that start at the columns 0, 4, .. 20: [chunk][group
// x 12 + row][8].  It is read twice:
//   convolution   out[y][x][f] = sum_i sum_c R[y + i][c] * T_i[c][x][f], T_i[c][x][f] = Wc[f][i][c - x], in three blocks of eight output
//                 columns (48 accumulator columns each; 24 = 3 x 8 needs no padding of N, and three tiles' accumulators fit): K = 16
//                 columns per kernel row, 128 x 48 x 16 per MMA, weights in fp16 high and low parts;
//   gradient      D[(x, f)][(i, c)] = sum_rows d[row][4 q + x][f] * R[row + i][4 q + c], G[f][i][j] = sum_x D[(x, f)][(i, x + j)], per column q of
//                 windows: K = the tile's rows, M = 64 (24 columns of the deltas' high parts, 24 of their low parts, 16 unused), N = 40
//                 (five kernel rows of eight columns).  All six window columns add to one D.  The deltas are the A operand, M-contiguous as the
//                 epilogue's lanes (rows) have them, the slab is the N-contiguous B operand: a row is 16 bytes, so it may start at any.
//
// Accuracy.  Pixels that are whole numbers / 255 (image files' bytes) are exact in fp16 (forward_tc.cu).  A tile with any other pixel goes through as
// an empty one, and its images are left to k_grad_left (fused_train.cu); so is the whole share of a CTA whose sample of pixels has others in several
// places, what comes behind too many such tiles, and everything where a parameter is not finite or far out of range.  The tensor core truncates its additions, which over a tile's 48 would cost a gradient 1e-6.  Here they are exact: deltas are
// scaled by a power of two so that the tile's bound on them (max |ds| * max |Ws| / 4) lies in [1024, 2048), and cut into a whole
// number, at most 11 bits, and the rest, which in fp16 is good to 2^-24 of the bound.  Products of whole numbers with bytes have 19 bits.  A D adds 720 of
// them: with deltas of one sign and bright pixels up to 2^28, of which truncation took 0.9e-6 on average and 3e-6 at most, always towards zero.  So
// pixels are taken from a level, the whole number next to the mean of a sample of the block's images; what it adds to a pre-activation is in the bias, and
// what it adds to a tap's gradient is the level times the bias gradient, which is summed in fp32.  Sums of centred pixels stay below 2^24: over nets as drawn
// and trained, and nets with deltas of one sign, with strokes, inverted strokes, both mixed, noise and smooth bright images, a tile's
// largest lies between 2^14 and 2^23.5 (without the level up to 2^26.9).
// D is added to fp32 sums in registers after every tile.  Distance of the gradient from fp64 in 1e-8 of its norm, k_grad_partials / here, geometric means: strokes, nets
// as drawn, 12 nets and batches of 2,048 to 60,000 images 4.93 / 4.93, conv weights alone 4.83 / 4.8, conv biases 5.8 / 4.8.  4,000 images and six to ten nets, conv
// weights alone: strokes 4.7 / 4.8, inverted 9.0 / 5.9, bright (200-255) 7.4 / 5.1, strokes and inverted ones 8.3 / 7.4, dim (0-126) 5.9 / 5.1; with deltas of one sign
// 4.9 / 5.1, 7.8 / 7.1, 8.6 / 8.6, 7.4 / 6.8, 6.6 / 6.9 (27 to 51 without the level).  With conv weights 30 times as large, where pre-activations are the limit: strokes
// 11.5 / 12.9, inverted 31 / 19, bright 80 / 64, both 22 / 21, dim 7.3 / 7.4, the whole gradient of strokes 4.8 / 5.4.
//
// Pipeline (one CTA per SM, 20 warps, mbarriers with bounded waits):
//   warps 4-7   one bulk copy per tile, two tiles ahead; pixels -> fp16 operand; drain D of the tile that had the slab before;
//   warp 2      issues the convolution's MMAs, block by block as accumulators become free;
//   warp 3      issues the gradient's, window column by window column;
//   warps 8-19  three groups of four warps, a tile each in turn.  Stage 1: conv activations (kept in tensor memory in the pre-activations' place),
//               window sums, subsample activations to shared memory.  Then the output layer of the five images, its error and the subsample
//               deltas.  Stage 2: conv deltas, subsample-filter and bias gradients, delta operand (its whole parts negated: one instruction less);
//   warps 0-1   FC gradient in registers (a thread owns three or four of the 216 inputs), from what the groups leave in shared memory.
//
// Measured on a B200, 60,000 images with the kernels around it: 643 us (k_grad_partials) -> 282 us.  What bounds it, per tile of five images (6,200 cycles):
// the shared-memory data pipe (operands of the 78 MMAs 2,590 cycles, other warps 3,020: delta operands 580, FC layer
// 700, loader 350, conflicts with the tensor core 570); instruction issue about 60 %, the special-function unit 37 %.  2,048 images are 24.0 us, of which a launch's
// set-up is 3.2 us.
#include "banded_conv.cuh"
#include "cluster_exchange.cuh"
#include "net.cuh"
#include "phase_clocks.cuh"
#include "wide_tc.cuh"

namespace cnn {

constexpr int kGtThreads = 640;
constexpr int kGtImgs = kGradTile;            // images per tile
constexpr int kGtRaw = 2, kGtSlabs = 5;       // tiles of raw images, and of operands, in shared memory
constexpr int kGtSets = 3;                    // groups of epilogue warps, and accumulators
constexpr unsigned kGtGroupStride = 12 * 16;  // a group's twelve rows
constexpr unsigned kGtChunk = 15 * kGtGroupStride + 48;      // 2,928 B: (row - piece) mod 8 picks the loader's 16-byte bank group
constexpr int kGtChunks = 6;
constexpr int kGtSlabBytes = kGtChunks * kGtChunk + 160;     // the sixteenth, unused group reads on behind the last chunk: finite numbers there
constexpr int kGtPieces = kGtImgs * kImg / 4;                // 980 pieces of four pixels
constexpr int kGtLoaders = 128, kGtUnits = (kGtPieces + kGtLoaders - 1) / kGtLoaders;
constexpr int kGtBN = 48;                                    // accumulator columns of a block of eight output columns
constexpr unsigned kGtBChunk = 5 * kGtBN * 16;               // 3,840 B: [kernel row][accumulator column][8 input columns]
constexpr int kGtBPart = 3 * kGtBChunk;                      // K chunks: first, second, and the last block's second (four columns on)
constexpr int kGtWindows = 4;                                // delta operands (one window column of a tile each) in shared memory
constexpr unsigned kGtDeltaBlock = 128 * 16;                 // [eight columns: 4 x, 2 maps][row]
constexpr int kGtDeltaBytes = 6 * kGtDeltaBlock;             // three map pairs, high and low parts
constexpr int kGtGradN = 40, kGtGradCol = kGtSets * 3 * kGtBN;     // D of even and odd tiles behind the accumulators: 432 + 2 * 40 = 512
constexpr int kGtFcThreads = 64, kGtFcRounds = 4;            // 216 = 3 * 64 + 24
// Places of the share that are looked at first, 128 pixels each, and how many with other than whole numbers / 255 leave it to the CUDA cores.  Images of
// strokes that are all of other numbers show them in half of the places or more (a fifth of a canvas is not zero); where one image in ten has them, a tile's worth
// of images in ten tiles is still cheaper left out (an empty tile 3.5 us, five images on the CUDA cores 8).
constexpr int kGtPlaces = 2 * kGtThreads / 32, kGtPlacesOther = 8;
constexpr int kGtWfStride = 234;              // five rows of weights, 10 (mod 32) words apart, by six parts of nine inputs: thirty banks
constexpr float kGtUnscale = 1.0f / 8192.0f;                 // of the convolution's accumulators
constexpr int kGtMaxExp = 100;                               // deltas are scaled by 2^100 at most, where they are zero or nearly so
constexpr float kGtMost = 67108864.f;                        // largest parameter, 2^26: a tap of the subsample filter times that scale is finite
constexpr int kGtConvWarp = 2, kGtGradWarp = 3, kGtLoadWarp0 = 4, kGtEpiWarp0 = 8;

struct GtSmem {
  alignas(128) float raw[kGtRaw][kGtImgs * kImg];
  alignas(128) unsigned char slab[kGtSlabs][kGtSlabBytes];
  alignas(128) unsigned char b[2][kGtBPart];                 // conv weights, high and low parts
  alignas(128) unsigned char delta[kGtWindows][kGtDeltaBytes];      // (M = 64 reads two blocks on: the last one's, whatever follows here)
  alignas(16) float wf[kOut][kGtWfStride];                   // FC weights by slot entry
  alignas(16) float as[kGtSets][kGtImgs][kS];       // subsample activations [window row][6 * window column + map]
  alignas(16) float ds[kGtSets][kGtImgs][kS];                // and deltas
  alignas(16) float df[kGtSets][kGtImgs][12];                // output deltas
  alignas(16) float zeros[36];                               // subsample deltas of the unused group
  float bc[8], ws[16], bs[4], bf[12];
  float most;                                                // largest pixel that is finite in fp16 with and without level and scale
  unsigned ds_max[kGtSets][4];
  float tile_unscale[kGtSlabs];
  unsigned long long raw_full[kGtRaw], a_full[kGtSlabs], a_free[kGtSlabs], d_full[3 * kGtSets], d_free[3 * kGtSets], df_ready[kGtSets], df_free[kGtSets],
      dl_full[kGtWindows], dl_free[kGtWindows], g_free[2];
  int px_sum[kGtThreads / 32];                               // whole pixels of the sample, by warp
  int skips, skipped[kGradSkips];                            // tiles left out: how many, and which
  int empty[kGtSlabs];                                       // the last of them that was in a slab
  int stop;                                                  // tiles that take part
  unsigned tmem_base;
  long long clock_base;                                      // phase clocks only
};

// What the block's gradients are gathered in at its end, in place of the raw images.
struct GtEnd {
  float d[48][kGtGradN + 1];
  float ws[12][16], bc[12][kF], bf[kOut], bs[12], err;
};
static_assert(sizeof(GtEnd) <= sizeof(float) * kGtRaw * kGtImgs * kImg, "");

CNN_PHASE_TABLE(g_phase_clocks_gt, 20)

// Barrier of 128 threads -- the loaders (1) or a group of epilogue warps (2 and up) -- that tells all of them whether any of them says so.
__device__ __forceinline__ bool barrier_any(int id, bool mine) {
  unsigned any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"((unsigned)mine), "r"(id)
      : "memory");
  return any != 0;
}

__device__ __forceinline__ void tmem_st8(unsigned taddr, const f32x2 (&v)[4]) {
  float x[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) unpack2(v[j], x[2 * j], x[2 * j + 1]);
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "f"(x[0]), "f"(x[1]), "f"(x[2]),
               "f"(x[3]), "f"(x[4]), "f"(x[5]), "f"(x[6]), "f"(x[7])
               : "memory");
}

// Barrier of one group of epilogue warps.
__device__ __forceinline__ void group_sync(int set) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(2 + set) : "memory"); }

// Eight bytes to shared memory if `when` is not zero, without a branch.
__device__ __forceinline__ void store_if(unsigned smem_addr, const unsigned (&v)[2], unsigned when) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.shared.v2.b32 [%0], {%1, %2};\n\t}" ::"r"(smem_addr), "r"(v[0]), "r"(v[1]),
               "r"(when)
               : "memory");
}

__device__ __forceinline__ f32x2 ld2(const float* p) { return *reinterpret_cast<const f32x2*>(p); }

// The loaders: tile k has other pixels.  It goes through all the same, with output deltas of zero, if what is in its slab is finite in fp16.
// Returns how many tiles take part: as many as before, or k where the block stops with this one.
__device__ __noinline__ int other_tile(GtSmem& sm, int k, int tiles, float big, int lt) {
  const int skips = sm.skips;
  if (barrier_any(1, !(big <= sm.most)) || skips == kGradSkips || 2 * skips > k + 4) {
    if (lt == 0) *const_cast<volatile int*>(&sm.stop) = k;
    return k;
  }
  if (lt == 0) {
    sm.skipped[skips] = k;
    *const_cast<volatile int*>(&sm.empty[k % kGtSlabs]) = k;
    sm.skips = skips + 1;
  }
  return tiles;
}

// One thread: the images of tile k of a share.
__device__ __forceinline__ void fetch_tile(GtSmem& sm, const float* images, int imgs_here, int k) {
  const unsigned bytes = (unsigned)(min(kGtImgs, imgs_here - k * kGtImgs) * kImg) * (unsigned)sizeof(float);
  mbar_expect_tx(&sm.raw_full[k % kGtRaw], bytes);
  bulk_g2s(sm.raw[k % kGtRaw], images + (long)k * kGtImgs * kImg, bytes, &sm.raw_full[k % kGtRaw]);
}

// The loaders' part (warps 4-7): tiles to operands, and what the gradient's MMAs have added up.  A function of its own, as run_group is: as parts of the
// kernel their registers and schedules changed with every line of the set-up (60,000 images 288 to 321 us, as functions 277 to 281).
__device__ __noinline__ void load_tiles(GtSmem& sm, const float* images, int imgs_here, int n_tiles, int wexp, int level, unsigned tmem_base, int* status) {
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  bool gave_up = false;
  CNN_PHASE_ROLE(blockIdx.x == 0, sm.clock_base)
  const int lt = tid - 32 * kGtLoadWarp0, quarter = warp & 3;
  // Piece i = lt + 128 j: four pixels (column 4 c) of one row, the second half of chunk c - 1 and the first of chunk c, in one group or two.
  // Lanes eight apart write the two halves of 16 bytes in opposite order, so that no bank is asked twice: first to `own + at[0]`, then to
  // `own + at[1]`.  Bits 16 to 19: whether the first place exists, whether a second group has it (64 bytes before), and the same of the second.
  unsigned dst[kGtUnits];
  const int swap = (lane >> 3) & 1;
  const unsigned at[2] = {swap ? 8u - kGtChunk : 0u, swap ? 0u : 8u - kGtChunk};
#pragma unroll
  for (int j = 0; j < kGtUnits; ++j) {
    const int i = lt + kGtLoaders * j, img = i / (kImg / 4), rest = i % (kImg / 4), r = rest / 7, c = rest % 7;
    const int g = min(r >> 3, 2);
    dst[j] = (unsigned)(((3 * img + g) * 12 + (r - 8 * g)) * 16) + (unsigned)c * kGtChunk;
    const unsigned two = g > 0 && r - 8 * g < 4 ? 3u : 1u, own = c < 6 ? two : 0u, before = c > 0 ? two : 0u;
    dst[j] |= i < kGtPieces ? (swap ? before | own << 2 : own | before << 2) << 16 : 0u;
  }
  const __half2 px_scale = __float2half2_rn(__int_as_float((127 + wexp - 3) << 23)), magic = __float2half2_rn(1536.f);
  const __half2 minus_level = __float2half2_rn(-(float)level * __int_as_float((127 + wexp - 3) << 23));
  const f32x2 k255 = pack2(255.f, 255.f);
  f32x2 sum[kGtGradN / 2];
#pragma unroll
  for (int i = 0; i < kGtGradN / 2; ++i) sum[i] = pack2(0.f, 0.f);
  auto drain = [&](int k) {
    mbar_wait_bounded(&sm.a_free[k % kGtSlabs], (unsigned)(k / kGtSlabs) & 1u, status, gave_up);
    __syncwarp();
    if (quarter == 3) return;
    tc::fence_after_sync();
    const float f = *const_cast<const volatile float*>(&sm.tile_unscale[k % kGtSlabs]);
    const f32x2 f2 = pack2(f, f);
    const unsigned t0 = tmem_base + (unsigned)(kGtGradCol + (k & 1) * kGtGradN) + ((unsigned)(quarter * 32) << 16);
#pragma unroll
    for (int c = 0; c < kGtGradN; c += 8) {
      unsigned v[8];
      tc::tmem_ld8_nowait(t0 + (unsigned)c, v);
      tc::tmem_wait8(v);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        sum[c / 2 + i] = fma2(pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), f2, sum[c / 2 + i]);
    }
    tc::fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.g_free[k & 1]);
  };
  int tiles = *const_cast<const volatile int*>(&sm.stop);
  int k = 0, drained = 0;
  for (; k < tiles; ++k) {
    const int s = k % kGtSlabs, r = k % kGtRaw;
    CNN_PHASE(0);
    if (k >= kGtSlabs) drain(drained++);
    CNN_PHASE(1);
    mbar_wait_bounded(&sm.raw_full[r], (unsigned)(k / kGtRaw) & 1u, status, gave_up);
    CNN_PHASE(2);
    const int pieces = min(kGtImgs, imgs_here - k * kGtImgs) * (kImg / 4);
    const unsigned slab = smem_u32(sm.slab[s]);
    unsigned bits = 0, odd = 0;
    float big = 0.f;
#pragma unroll
    for (int j0 = 0; j0 < kGtUnits; j0 += 4) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const float4*>(&sm.raw[r][4 * min(lt + kGtLoaders * (j0 + j), pieces - 1)]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x[4];
        unpack2(mul2(pack2(v[j].x, v[j].y), k255), x[0], x[1]);
        unpack2(mul2(pack2(v[j].z, v[j].w), k255), x[2], x[3]);
        big = max_abs_nan(max_abs_nan(big, x[0], x[1]), x[2], x[3]);
        bits |= __float_as_uint(x[0]) | __float_as_uint(x[1]) | __float_as_uint(x[2]) | __float_as_uint(x[3]);
        unsigned h[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const __half2 p = __floats2half2_rn(x[2 * c], x[2 * c + 1]);
          const __half2 w = __hsub2(__hadd2(p, magic), magic);      // whole numbers below 512 as they are
          odd |= *reinterpret_cast<const unsigned*>(&p) ^ *reinterpret_cast<const unsigned*>(&w);
          const __half2 q = __hfma2(p, px_scale, minus_level);
          h[c] = *reinterpret_cast<const unsigned*>(&q);
        }
        const unsigned to = lt + kGtLoaders * (j0 + j) < pieces ? dst[j0 + j] : 0u, own = slab + (to & 0xffffu);
#pragma unroll
        for (int turn = 0; turn < 2; ++turn) {
          store_if(own + at[turn], h, to & (1u << (16 + 2 * turn)));
          store_if(own + at[turn] - 64u, h, to & (1u << (17 + 2 * turn)));
        }
      }
    }
    tc::fence_async_smem();    // generic-proxy writes -> visible to the tensor core's operand reads
    if (barrier_any(1, (bits & 0x1fffu) != 0 || odd != 0 || !(big <= 255.f))) tiles = other_tile(sm, k, tiles, big, lt);
    if (lt == 0) {
      if (k + kGtRaw < n_tiles) fetch_tile(sm, images, imgs_here, k + kGtRaw);
      mbar_arrive(&sm.a_full[s]);
    }
    __syncwarp();
    CNN_PHASE(3);
  }
  // copies that are still on their way land before their memory is used for anything else
  for (int j = k; j < min(k + kGtRaw, n_tiles); ++j)
    mbar_wait_bounded(&sm.raw_full[j % kGtRaw], (unsigned)(j / kGtRaw) & 1u, status, gave_up);
  for (; drained < tiles; ++drained) drain(drained);      // (`tiles` take part, k may be one more)
  __syncthreads();
  if (quarter < 3 && lane < 16) {
    GtEnd& end = *reinterpret_cast<GtEnd*>(sm.raw);
    float* to = end.d[16 * quarter + lane];
#pragma unroll
    for (int i = 0; i < kGtGradN / 2; ++i) unpack2(sum[i], to[2 * i], to[2 * i + 1]);
  }
  CNN_PHASE_END(g_phase_clocks_gt);
}

// The part of a group of epilogue warps (8-19).
__device__ __noinline__ void run_group(GtSmem& sm, const unsigned* labels, int imgs_here, int n_tiles, float wsmax, unsigned tmem_base, int* status) {
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const volatile int& stop = sm.stop;
  bool gave_up = false;
  CNN_PHASE_ROLE(blockIdx.x == 0, sm.clock_base)
  const int set = (warp - kGtEpiWarp0) >> 2;     // accumulator / tile residue this group owns
  const int quarter = warp & 3;                  // tensor-memory lanes 32 * quarter ..
  const int rsub = lane & 3;                     // row of the 4x4 window
  const int g = quarter * 4 + (lane >> 3);       // group of 8 output rows this lane's row belongs to
  const int img = g / 3, p = 2 * (g % 3) + ((lane >> 2) & 1);      // image of the tile (5: the unused group), window row
  const bool used = img < kGtImgs;
  const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;
  f32x2 bc2[kF / 2], gws[4], gbc[kF / 2];
#pragma unroll
  for (int j = 0; j < 4; ++j) gws[j] = pack2(0.f, 0.f);
#pragma unroll
  for (int f = 0; f < kF; f += 2) {
    bc2[f / 2] = pack2(sm.bc[f], sm.bc[f + 1]);
    gbc[f / 2] = pack2(0.f, 0.f);
  }
  const f32x2 unscale2 = pack2(kGtUnscale, kGtUnscale), one2 = pack2(1.f, 1.f);
  const float bs = sm.bs[0];
  float* const as_slot = used ? &sm.as[set][img][p * 36] : nullptr;
  const float* const ds_slot = used ? &sm.ds[set][img][p * 36] : sm.zeros;
  // FC forward: 54 inputs per warp, lane = nine of them (of six parts) and outputs fk and fk + 5, for all five images
  const int fk = lane < 30 ? lane % 5 : 4, fpart = lane < 30 ? lane / 5 : 5, first_in = 54 * quarter + 9 * fpart;
  const int gt = 32 * quarter + lane;            // thread of the group: inputs gt and gt + 128
  float g_bs = 0.f;
  const unsigned t0 = tmem_base + (unsigned)(set * 3 * kGtBN) + ((unsigned)(quarter * 32) << 16);

  for (int k = set; k < n_tiles; k += kGtSets) {
    const unsigned turn = (unsigned)(k / kGtSets) & 1u;
    bool halt = false;
    // output layer: quarter 0 images 0-2, quarter 1 images 3-4, lane 10 j + o
    const int oj = 3 * quarter + lane / 10, oo = lane % 10;
    const bool outputs = quarter < 2 && lane < (quarter ? 20 : 30);
    unsigned label = ~0u;
    if (outputs && k * kGtImgs + oj < imgs_here) label = labels[k * kGtImgs + oj];
    CNN_PHASE(0);
    if (k >= kGtSets) mbar_wait_bounded(&sm.df_free[set], turn ^ 1u, status, gave_up);      // this group's tile before this one
    {
      f32x2 ws2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float w = sm.ws[rsub * 4 + j];
        ws2[j] = pack2(w, w);
      }
#pragma unroll 1
      for (int xb = 0; xb < 3; ++xb) {              // one block of two window columns
        mbar_wait_bounded(&sm.d_full[3 * set + xb], turn, status, gave_up);
        if (xb == 0) {
          halt = barrier_any(2 + set, k >= stop);      // (all of the group, or none)
          CNN_PHASE(1);
        }
        if (halt) break;
        __syncwarp();
        tc::fence_after_sync();
        unsigned nxt[8];
        tc::tmem_ld8_nowait(t0 + (unsigned)(xb * kGtBN), nxt);
        tc::tmem_wait8(nxt);
        float z[12];
        f32x2 d2[4];               // 1 + 2^t of the row's four columns (of two maps), one step behind
        // Step ch turns 8 accumulator columns (window column ch / 3, maps 2 * (ch % 3) + {0, 1}) into exponentials and
        // finishes the columns of step ch - 1, so that two chains of dependent instructions are always under way.
#pragma unroll
        for (int ch = 0; ch < 7; ++ch) {
          f32x2 e2[4];
          if (ch < 6) {
            if (ch > 0) tc::tmem_wait8(nxt);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              e2[j] = fma2(pack2(__uint_as_float(nxt[2 * j]), __uint_as_float(nxt[2 * j + 1])), unscale2, bc2[ch % 3]);
            if (ch < 5) tc::tmem_ld8_nowait(t0 + (unsigned)(xb * kGtBN + (ch + 1) * 8), nxt);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, y;
              unpack2(e2[j], x, y);
              e2[j] = pack2(exp2f_approx(x), exp2f_approx(y));
            }
          }
          if (ch > 0) {
            f32x2 z2;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x, y;
              unpack2(d2[j], x, y);
              d2[j] = pack2(rcp_approx(x), rcp_approx(y));
              z2 = j == 0 ? mul2(ws2[0], d2[0]) : fma2(ws2[j], d2[j], z2);
            }
            tmem_st8(t0 + (unsigned)(xb * kGtBN + (ch - 1) * 8), d2);      // the activations, for stage 2
            unpack2(z2, z[2 * (ch - 1)], z[2 * (ch - 1) + 1]);
          }
          if (ch < 6) {
#pragma unroll
            for (int j = 0; j < 4; ++j) d2[j] = add2(e2[j], one2);
          }
        }
        // the window's four rows are lanes 4g..4g+3: reduce-scatter the block's 12 sums
        float w6[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const float send = b0 ? z[i] : z[i + 6], keep = b0 ? z[i + 6] : z[i];
          w6[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float send = b1 ? w6[i] : w6[i + 3], keep = b1 ? w6[i + 3] : w6[i];
          const float as = sigmoidf<1>(keep + __shfl_xor_sync(0xffffffffu, send, 2) + bs);
          if (used) as_slot[12 * xb + (b0 ? 6 : 0) + (b1 ? 3 : 0) + i] = as;
        }
      }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    if (halt) {
      if (lane == 0 && quarter < 2) mbar_arrive(&sm.df_ready[set]);
      if (k == stop) {        // the gradient warp waits for this tile's first window: its turn, empty
        const int win = (6 * k) % kGtWindows;
        if (k >= 2) mbar_wait_bounded(&sm.a_free[(k - 2) % kGtSlabs], (unsigned)((k - 2) / kGtSlabs) & 1u, status, gave_up);
        mbar_wait_bounded(&sm.dl_free[win], ((unsigned)(6 * k / kGtWindows) & 1u) ^ 1u, status, gave_up);
        if (lane == 0) mbar_arrive(&sm.dl_full[win]);
      }
      break;
    }
    CNN_PHASE(2);
    // ---- the output layer, its error, and the subsample deltas, by the group's 128 threads ----
    group_sync(set);
    {
      const float *as = &sm.as[set][0][first_in], *w0 = &sm.wf[fk][first_in], *w1 = &sm.wf[fk + 5][first_in];
      f32x2 z[kGtImgs];
#pragma unroll
      for (int jj = 0; jj < kGtImgs; ++jj) z[jj] = pack2(0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const f32x2 w2 = pack2(w0[i], w1[i]);
#pragma unroll
        for (int jj = 0; jj < kGtImgs; ++jj) {
          const float a = as[jj * kS + i];
          z[jj] = fma2(w2, pack2(a, a), z[jj]);
        }
      }
      // parts 3-5 to parts 0-2, the twelve sums of the group to shared memory (where the subsample deltas come later)
      float* part = &sm.ds[set][0][0] + (3 * quarter + fpart) * 50 + fk;
#pragma unroll
      for (int jj = 0; jj < kGtImgs; ++jj) {
        float lo, hi;
        unpack2(z[jj], lo, hi);
        lo += __shfl_down_sync(0xffffffffu, lo, 15);
        hi += __shfl_down_sync(0xffffffffu, hi, 15);
        if (lane < 15) {
          part[10 * jj] = lo;
          part[10 * jj + 5] = hi;
        }
      }
    }
    CNN_PHASE(9);
    group_sync(set);
    CNN_PHASE(10);
    if (quarter < 2) {
      if (outputs) {
        const float* part = &sm.ds[set][0][0] + 10 * oj + oo;
        float z = 0.f;
#pragma unroll
        for (int i = 0; i < 12; i += 4) z += (part[50 * i] + part[50 * i + 50]) + (part[50 * i + 100] + part[50 * i + 150]);
        const float d = (label == (unsigned)oo ? 1.0f : 0.0f) - sigmoidf<1>(z + sm.bf[oo]);       // makeError
        const bool counts = k * kGtImgs + oj < imgs_here && *const_cast<const volatile int*>(&sm.empty[k % kGtSlabs]) != k;
        sm.df[set][oj][oo] = counts ? d : 0.f;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.df_ready[set]);
    }
    CNN_PHASE(11);
    group_sync(set);
    CNN_PHASE(12);
    float most = 0.f;
    {
      f32x2 wk[2][kOut / 2];
      const bool second = gt + 128 < kS;
      const int u[2] = {gt, second ? gt + 128 : gt};
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int kk = 0; kk < kOut / 2; ++kk) wk[r][kk] = pack2(sm.wf[2 * kk][u[r]], sm.wf[2 * kk + 1][u[r]]);
#pragma unroll
      for (int jj = 0; jj < kGtImgs; ++jj) {
        const ulonglong2 e0 = *reinterpret_cast<const ulonglong2*>(&sm.df[set][jj][0]), e1 = *reinterpret_cast<const ulonglong2*>(&sm.df[set][jj][4]);
        const f32x2 e4 = ld2(&sm.df[set][jj][8]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float a = sm.as[set][jj][u[r]];
          float lo, hi;
          unpack2(fma2(wk[r][4], e4, fma2(wk[r][3], e1.y, fma2(wk[r][2], e1.x, fma2(wk[r][1], e0.y, mul2(wk[r][0], e0.x))))), lo, hi);
          const float ds = (lo + hi) * a * (1.f - a);
          if (r == 0 || second) {
            sm.ds[set][jj][u[r]] = ds;
            g_bs += ds;
          }
          most = fmaxf(most, fabsf(ds));
        }
      }
    }
    const unsigned m32 = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
    if (lane == 0) sm.ds_max[set][quarter] = m32;
    group_sync(set);
    CNN_PHASE(3);
    CNN_PHASE(7);
    // The delta operands go round: a window's turn is told by a parity, which is unambiguous while no more than two tiles are at it.
    if (k >= 2) mbar_wait_bounded(&sm.a_free[(k - 2) % kGtSlabs], (unsigned)((k - 2) / kGtSlabs) & 1u, status, gave_up);
    CNN_PHASE(8);
    // |conv delta * 576| <= max |ds| * max |Ws| / 4: scaled by 2^e into [1024, 2048) at most
    const unsigned ds_bits = max(max(sm.ds_max[set][0], sm.ds_max[set][1]), max(sm.ds_max[set][2], sm.ds_max[set][3]));
    const float bound = __uint_as_float(ds_bits) * wsmax * 0.25f;
    const int e = min(max(10 - ((int)(__float_as_uint(bound) >> 23) - 127), -kGtMaxExp), kGtMaxExp);
    const float scale = __int_as_float((127 + e) << 23), unscale = __int_as_float((127 - e) << 23);
    if (quarter == 0 && lane == 0) *const_cast<volatile float*>(&sm.tile_unscale[k % kGtSlabs]) = unscale;
    f32x2 ws2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float w = sm.ws[rsub * 4 + j] * scale;
      ws2[j] = pack2(w, w);
    }
    const f32x2 back2 = pack2(unscale, unscale), minus2 = pack2(-1.f, -1.f);
    const f32x2 magic2 = pack2(12582912.f, 12582912.f);      // 1.5 * 2^23: adding it rounds to a whole number
    unsigned nxt[8];
    tc::tmem_ld8_nowait(t0, nxt);
#pragma unroll 1
    for (int w = 0; w < 6; ++w) {                 // window columns
      const int at = 6 * k + w, win = at % kGtWindows;
      unsigned char* const to = sm.delta[win] + (32 * quarter + lane) * 16;
      CNN_PHASE(5);
      mbar_wait_bounded(&sm.dl_free[win], ((unsigned)(at / kGtWindows) & 1u) ^ 1u, status, gave_up);
      __syncwarp();
      CNN_PHASE(6);
#pragma unroll
      for (int m = 0; m < 3; ++m) {               // map pairs
        tc::tmem_wait8(nxt);
        f32x2 a2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) a2[j] = pack2(__uint_as_float(nxt[2 * j]), __uint_as_float(nxt[2 * j + 1]));
        if (m < 2 || w < 5) tc::tmem_ld8_nowait(t0 + (unsigned)(24 * w + 8 * m + 8), nxt);
        if (m == 2 && (w & 1)) {                   // the last columns of a block are in registers: hand it back to the MMA warp
          tc::fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.d_free[3 * set + (w >> 1)]);
        }
        const f32x2 ds2 = ld2(ds_slot + 6 * w + 2 * m);
        unsigned hi[4], lo[4];
        f32x2 total;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          gws[j] = fma2(ds2, a2[j], gws[j]);
          const f32x2 slope = mul2(a2[j], fma2(a2[j], minus2, one2)), c = mul2(ds2, ws2[j]);      // the delta is their product
          total = j == 0 ? mul2(slope, c) : fma2(slope, c, total);
          const f32x2 whole = fma2(fma2(slope, c, magic2), minus2, magic2);                        // minus the delta, rounded
          float q0, q1, l0, l1;
          unpack2(whole, q0, q1);
          unpack2(fma2(slope, c, whole), l0, l1);
          const __half2 hh = __floats2half2_rn(q0, q1), hl = __floats2half2_rn(l0, l1);
          hi[j] = *reinterpret_cast<const unsigned*>(&hh);
          lo[j] = *reinterpret_cast<const unsigned*>(&hl);
        }
        gbc[m] = fma2(total, back2, gbc[m]);
        *reinterpret_cast<uint4*>(to + m * kGtDeltaBlock) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(to + (3 + m) * kGtDeltaBlock) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
      tc::fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.dl_full[win]);
    }
    CNN_PHASE(4);
  }
  // ---- what this warp has gathered: lanes 0-3 the taps 4 * lane + j, lane 0 the biases ----
  float t[4], b[kF];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float lo, hi;
    unpack2(gws[j], lo, hi);
    t[j] = lo + hi;
#pragma unroll
    for (int m = 4; m <= 16; m <<= 1) t[j] += __shfl_xor_sync(0xffffffffu, t[j], m);
  }
#pragma unroll
  for (int f = 0; f < kF; f += 2) unpack2(gbc[f / 2], b[f], b[f + 1]);
#pragma unroll
  for (int f = 0; f < kF; ++f)
#pragma unroll
    for (int m = 1; m <= 16; m <<= 1) b[f] += __shfl_xor_sync(0xffffffffu, b[f], m);
#pragma unroll
  for (int m = 1; m <= 16; m <<= 1) g_bs += __shfl_xor_sync(0xffffffffu, g_bs, m);
  __syncthreads();
  GtEnd& end = *reinterpret_cast<GtEnd*>(sm.raw);
  if (lane < 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) end.ws[warp - kGtEpiWarp0][4 * lane + j] = t[j];
  }
  if (lane == 0) {
#pragma unroll
    for (int f = 0; f < kF; ++f) end.bc[warp - kGtEpiWarp0][f] = b[f];
    end.bs[warp - kGtEpiWarp0] = g_bs;
  }
  CNN_PHASE_END(g_phase_clocks_gt);
}

// One thread: this block has left something, and has written what, and its row.
__device__ __forceinline__ void push_left(GradLeft* left, int* pushed) {
  __threadfence();
  const int at = atomicAdd(pushed, 1);
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(&left[at].next), "r"((int)blockIdx.x + 1) : "memory");
}

// left[b]: what of block b's share is not in its row.
__global__ void __launch_bounds__(kGtThreads, 1)
k_grad_tc(const float* images, const unsigned* labels, GradShares shares, const float* params, float* __restrict__ rows,
          GradLeft* left, int* pushed, int* __restrict__ status) {
  extern __shared__ unsigned char smem_raw[];
  GtSmem& sm = *reinterpret_cast<GtSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  constexpr float kPre = -1.4426950408889634f;      // the short sigmoid form's factor, in the conv weights and biases
  constexpr double kByteExcess = 2.37e-8;

  const long img0 = shares.first(blockIdx.x);
  const int imgs_here = shares.size(blockIdx.x);
  const int n_tiles = (imgs_here + kGtImgs - 1) / kGtImgs;

  if (tid == 0) {
    for (int s = 0; s < kGtRaw; ++s) mbar_init(&sm.raw_full[s], 1);
    for (int s = 0; s < kGtSlabs; ++s) { mbar_init(&sm.a_full[s], 1); mbar_init(&sm.a_free[s], 1); }
    for (int s = 0; s < 3 * kGtSets; ++s) { mbar_init(&sm.d_full[s], 1); mbar_init(&sm.d_free[s], 4); }
    for (int s = 0; s < kGtSets; ++s) { mbar_init(&sm.df_ready[s], 2); mbar_init(&sm.df_free[s], kGtFcThreads / 32); }
    for (int s = 0; s < kGtWindows; ++s) { mbar_init(&sm.dl_full[s], 4); mbar_init(&sm.dl_free[s], 1); }
    for (int s = 0; s < 2; ++s) mbar_init(&sm.g_free[s], 3);
    mbar_fence_init();
  }
  if (warp == kGtGradWarp) tc::tmem_alloc(&sm.tmem_base, 512);
  pdl_wait();
  pdl_launch_dependents();

  // ---- a sample of the share's pixels, 128 neighbours at each of kGtPlaces places: its mean is the level that pixels are taken from, and images with
  // other pixels than whole numbers / 255 are as a rule many (this block has nothing to do then) ----
  float4 px[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int first = (2 * warp + j) * ((imgs_here * (kImg / 4) - 32) / (kGtPlaces - 1));
    px[j] = reinterpret_cast<const float4*>(images + img0 * kImg)[first + lane];
  }
  // The parameters as well: every load of the set-up is under way before the first value is used.
  constexpr int kBRows = 3 * 5 * kGtBN, kBTurns = (kBRows + kGtThreads - 1) / kGtThreads;      // 16-byte rows of the conv operand
  // The first 80 threads build two of them; the FC table, the small parameters and the biases are others' (all by the first: 0.4 us more per launch).
  constexpr int kFcFrom = 96, kSmallFrom = 320, kBiasWarp = 12;
  constexpr int kAll = (kNParams + kGtThreads - 1) / kGtThreads;
  float bw[kBTurns][5], wfc[kOut], small, share[kAll], taps[5], wsmax;      // (taps: the 150 and the six biases)
#pragma unroll
  for (int t = 0; t < kBTurns; ++t) {
    const int e = min(tid + t * kGtThreads, kBRows - 1), i = e / kGtBN % 5;
#pragma unroll
    for (int d = 0; d < 5; ++d) bw[t][d] = params[kOffWc + band_map(e % kGtBN) * 25 + i * 5 + d];
  }
  {
    const int u = min(max(tid - kFcFrom, 0), kS - 1), t = tid - kSmallFrom;
    const float* wf = params + kOffWf + (u % 6) * 36 + u / 6;      // slot entry u = 36 p + 6 q + f: input 36 f + 6 p + q
#pragma unroll
    for (int k = 0; k < kOut; ++k) wfc[k] = wf[k * kS];
    small = params[t < 0 || t > 28 ? 0 : (t < 16 ? kOffWs + t : (t < 28 ? kOffBf + min(t - 16, kOut - 1) : kOffBs))];
  }
#pragma unroll
  for (int j = 0; j < kAll; ++j) share[j] = params[min(tid + kGtThreads * j, kNParams - 1)];
#pragma unroll
  for (int j = 0; j < 5; ++j) taps[j] = params[min(lane + 32 * j, kOffWs - 1)];
  wsmax = fabsf(params[kOffWs + (lane & 15)]);
  // What no tile of five images writes of a slab: behind each chunk, and behind the last.  The slab of a shorter tile, the share's last, as a whole.
  for (int i = tid; i < kGtSlabs * 28; i += kGtThreads) {
    const int j = i % 28;
    const unsigned off = j < 3 * kGtChunks ? j / 3 * kGtChunk + 15 * kGtGroupStride + j % 3 * 16 : kGtChunks * kGtChunk + (j - 3 * kGtChunks) * 16;
    *reinterpret_cast<uint4*>(sm.slab[i / 28] + off) = make_uint4(0, 0, 0, 0);
  }
  if (imgs_here % kGtImgs != 0)
    for (int i = tid; i < kGtSlabBytes / 16; i += kGtThreads) reinterpret_cast<uint4*>(sm.slab[(n_tiles - 1) % kGtSlabs])[i] = make_uint4(0, 0, 0, 0);
  if (tid < 36) sm.zeros[tid] = 0.f;
  if (tid < kGtSlabs) sm.empty[tid] = -1;
  {
    bool other[2] = {false, false};
    int sum = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float x[4] = {px[j].x * 255.f, px[j].y * 255.f, px[j].z * 255.f, px[j].w * 255.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        other[j] = other[j] || !(x[c] == rintf(x[c]) && fabsf(x[c]) <= 255.f);
        sum += (int)fminf(fmaxf(x[c], 0.f), 255.f);
      }
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) sm.px_sum[warp] = sum;
    const bool first = __any_sync(0xffffffffu, other[0]), second = __any_sync(0xffffffffu, other[1]);
    if (__syncthreads_count((lane == 0 && first) || (lane == 1 && second)) >= kGtPlacesOther) {
      if (tid == 0) {
        left[blockIdx.x].from = left[blockIdx.x].written = left[blockIdx.x].skips = 0;
        push_left(left, pushed);
      }
      if (warp == kGtGradWarp) tc::tmem_dealloc(sm.tmem_base, 512);
      return;
    }
  }
  if (tid == 0)        // the thread that initialised the barriers
    for (int k = 0; k < kGtRaw && k < n_tiles; ++k) fetch_tile(sm, images + img0 * kImg, imgs_here, k);

  // ---- set-up: scales, conv weights, FC table, small parameters ----------------------------------------------
  float wmax = 0.f;
  bool sane = true;
#pragma unroll
  for (int j = 0; j < 5; ++j) wmax = fmaxf(wmax, lane + 32 * j < kOffBc ? fabsf(taps[j]) : 0.f);
#pragma unroll
  for (int j = 0; j < kAll; ++j) sane = sane && fabsf(share[j]) <= kGtMost;
  wmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(wmax)));      // (magnitudes compare as their bits)
  wsmax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(wsmax)));
  // With 2^E <= max |kPre * w| < 2^(E+1) weights are scaled by 2^(16-E) / 255 and pixels by 255 * 2^(E-3): the accumulator carries 2^13.
  int wexp = (int)((__float_as_uint(fabsf(kPre) * wmax) >> 23) & 255u) - 127;
  sane = sane && wexp >= -21 && wexp <= 11;      // fp16 holds 255 * 2^(E-3)
  wexp = min(max(wexp, -21), 11);
  const float w_scale = __int_as_float((127 + 16 - wexp) << 23);
  int level = __reduce_add_sync(0xffffffffu, lane < kGtThreads / 32 ? sm.px_sum[lane] : 0);       // the sample's mean pixel, a whole number
  level = wexp > 10 ? 0 : (level + 128 * kGtPlaces / 2) / (128 * kGtPlaces);      // (a negative pixel may be 510 below it)

#pragma unroll
  for (int turn = 0; turn < kBTurns; ++turn) {     // one 16-byte row: 8 input columns of one accumulator column
    const int e = tid + turn * kGtThreads;
    if (e >= kBRows) break;
    const int variant = e / (5 * kGtBN), i = e / kGtBN % 5, nn = e % kGtBN, x = band_column(nn);
    float w[5];
#pragma unroll
    for (int d = 0; d < 5; ++d) w[d] = w_scale * bw[turn][d];
    __half2 hi[4], lo[4];
    // A byte / 255 in fp32 is kByteExcess of itself too large on average, and the pixels are bytes.  And truncated additions take 4e-8 of a
    // pre-activation: with that the conv weights' gradient is nearest to fp64 (strokes, weights eight times as large: 8.8e-8 without, 7.6e-8, 8.6e-8 with
    // twice as much).
    constexpr TwoPart kFactor = two_part((double)kPre / 255.0 * (1.0 + kByteExcess + 4e-8));
    // Input columns of the block: 0-7, 8-15, or 4-11 of which the first four are in the first chunk.
    band_row(w, (variant == 0 ? 0 : (variant == 1 ? 8 : 4)) - x, kFactor, hi, lo);
    if (variant == 2) hi[0] = hi[1] = lo[0] = lo[1] = __half2half2(__ushort_as_half(0));
    const unsigned off = (unsigned)variant * kGtBChunk + (unsigned)(i * kGtBN + nn) * 16u;
    *reinterpret_cast<uint4*>(sm.b[0] + off) = *reinterpret_cast<uint4*>(hi);
    *reinterpret_cast<uint4*>(sm.b[1] + off) = *reinterpret_cast<uint4*>(lo);
  }
  if (tid >= kFcFrom && tid < kFcFrom + kS) {
#pragma unroll
    for (int k = 0; k < kOut; ++k) sm.wf[k][tid - kFcFrom] = wfc[k];
  } else if (tid >= kSmallFrom && tid <= kSmallFrom + 28) {
    const int t = tid - kSmallFrom;
    if (t < 16) sm.ws[t] = small;
    else if (t < 28) sm.bf[t - 16] = (t - 16 < kOut) ? small : 0.f;
    else sm.bs[0] = small;
  }
  // A map's bias, and what the level adds to its pre-activations: an error here is the same in every window, so it is rounded once (in fp32: the gradient of
  // dense bright images at weights up to 15 three times as far from fp64).
  if (warp >= kBiasWarp && warp < kBiasWarp + kF) {
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < 5; ++j) sum += (lane + 32 * j) / 25 == warp - kBiasWarp ? (double)taps[j] : 0.0;
#pragma unroll 1
    for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
    const float bias = __shfl_sync(0xffffffffu, taps[4], kOffBc - 128 + warp - kBiasWarp);
    if (lane == 0) sm.bc[warp - kBiasWarp] = (float)(-1.4426950408889634 * ((double)bias + (double)level * ((1.0 + kByteExcess) / 255.0) * sum));
  }
  tc::fence_async_smem();      // the operands were written through the generic proxy
  tc::fence_before_sync();
  const bool all_sane = __syncthreads_and(sane);
  if (tid == 0) {
    sm.stop = all_sane ? n_tiles : 0;
    sm.skips = 0;
    sm.most = 60000.f / fmaxf(1.f, __int_as_float((127 + wexp - 3) << 23)) - 255.f;
  }
  __syncthreads();
  tc::fence_after_sync();
  const unsigned tmem_base = sm.tmem_base;
  const volatile int& stop = sm.stop;

  bool gave_up = false;
  CNN_PHASE_BEGIN(blockIdx.x == 0, sm.clock_base)
  GtEnd& end = *reinterpret_cast<GtEnd*>(sm.raw);
  float* row = rows + (size_t)blockIdx.x * kRowStride;

  if (warp < kGtFcThreads / 32) {
    // ================= FC gradient ==================================================================
    const int t = tid;                       // inputs t, t + 64, t + 128 and, the first 24 threads, t + 192
    int u[kGtFcRounds];
    bool live[kGtFcRounds];
    f32x2 gw[kGtFcRounds][kOut / 2];
#pragma unroll
    for (int r = 0; r < kGtFcRounds; ++r) {
      live[r] = t + kGtFcThreads * r < kS;
      u[r] = live[r] ? t + kGtFcThreads * r : kS - 1;
#pragma unroll
      for (int kk = 0; kk < kOut / 2; ++kk) gw[r][kk] = pack2(0.f, 0.f);
    }
    float g_bf = 0.f, err = 0.f;
    for (int k = 0; k < n_tiles; ++k) {
      const int g = k % kGtSets;
      CNN_PHASE(0);
      mbar_wait_bounded(&sm.df_ready[g], (unsigned)(k / kGtSets) & 1u, status, gave_up);
      CNN_PHASE(1);
      if (k >= stop) break;
      f32x2 tile[kGtFcRounds][kOut / 2];      // (added per tile: a sum over all images in one chain would be less exact)
#pragma unroll
      for (int jj = 0; jj < kGtImgs; ++jj) {
        const ulonglong2 e0 = *reinterpret_cast<const ulonglong2*>(&sm.df[g][jj][0]), e1 = *reinterpret_cast<const ulonglong2*>(&sm.df[g][jj][4]);
        const f32x2 d[5] = {e0.x, e0.y, e1.x, e1.y, ld2(&sm.df[g][jj][8])};
#pragma unroll
        for (int r = 0; r < kGtFcRounds; ++r) {
          const float a = sm.as[g][jj][u[r]];
          const f32x2 a2 = pack2(a, a);
#pragma unroll
          for (int kk = 0; kk < kOut / 2; ++kk) tile[r][kk] = jj == 0 ? mul2(d[kk], a2) : fma2(d[kk], a2, tile[r][kk]);
        }
      }
#pragma unroll
      for (int r = 0; r < kGtFcRounds; ++r)
#pragma unroll
        for (int kk = 0; kk < kOut / 2; ++kk) gw[r][kk] = add2(gw[r][kk], tile[r][kk]);
      if (warp == 0 && lane < kOut) {
        float five = 0.f;
#pragma unroll
        for (int jj = 0; jj < kGtImgs; ++jj) five += sm.df[g][jj][lane];
        g_bf += five;
      }
      if (warp == 1 && lane < kGtImgs) {
        float sq = 0.f;
#pragma unroll
        for (int oo = 0; oo < kOut; ++oo) sq = fmaf(sm.df[g][lane][oo], sm.df[g][lane][oo], sq);
        err += sqrtf(sq);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.df_free[g]);
      CNN_PHASE(2);
    }
    // ---- what these warps have gathered ----
#pragma unroll
    for (int r = 0; r < kGtFcRounds; ++r)
      if (live[r]) {
        float* dst = row + kOffWf + (u[r] % 6) * 36 + u[r] / 6;
#pragma unroll
        for (int kk = 0; kk < kOut / 2; ++kk) unpack2(gw[r][kk], dst[2 * kk * kS], dst[(2 * kk + 1) * kS]);
      }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) err += __shfl_xor_sync(0xffffffffu, err, m);
    __syncthreads();      // (the raw images' memory is free)
    if (warp == 0 && lane < kOut) end.bf[lane] = g_bf;
    if (warp == 1 && lane == 0) end.err = err;
  } else if (warp == kGtConvWarp) {
    // ================= MMA issue, convolution: the whole warp runs the loop, one elected lane issues ===========
    const unsigned idesc = tc::idesc_f16(128, kGtBN);
    int known = stop;      // tiles that take part, as far as this warp has heard
    // Where the loaders have stopped, the groups that wait for the next tiles are told by an arrival alone.
    for (int j = 0; j < n_tiles && j < known + kGtSets; ++j) {
      const int s = j % kGtSlabs, set = j % kGtSets;
      CNN_PHASE(0);
      if (j < known) {
        mbar_wait_bounded(&sm.a_full[s], (unsigned)(j / kGtSlabs) & 1u, status, gave_up);
        known = min(known, (int)stop);
      }
      CNN_PHASE(1);
#pragma unroll 1
      for (int xb = 0; xb < 3; ++xb) {
        mbar_wait_bounded(&sm.d_free[3 * set + xb], ((unsigned)(j / kGtSets) & 1u) ^ 1u, status, gave_up);
        __syncwarp();
        if (j >= known) {
          if (lane == 0) mbar_arrive(&sm.d_full[3 * set]);
          __syncwarp();
          break;
        }
        CNN_PHASE(2);
        tc::fence_after_sync();
        // K chunks: input columns 8 xb and 8 xb + 8; the last block's second chunk starts at column 20
        const unsigned long long ad = tc::smem_desc(smem_u32(sm.slab[s]) + (unsigned)(2 * xb) * kGtChunk, xb < 2 ? 2 * kGtChunk : kGtChunk, kGtGroupStride);
        const unsigned d = tmem_base + (unsigned)(set * 3 * kGtBN + xb * kGtBN);
#pragma unroll
        for (int pass = 1; pass >= 0; --pass) {      // the low parts first: the tensor core truncates its sums, which costs little while they are small
          const unsigned long long bd = tc::smem_desc(smem_u32(sm.b[pass]), xb < 2 ? kGtBChunk : 2 * kGtBChunk, 128);
          tc::mma_f16_run_elect<5, 1, kGtBN>(d, ad, bd, idesc, pass ? 0u : 1u);
        }
        tc::mma_commit_elect(&sm.d_full[3 * set + xb]);
        CNN_PHASE(3);
      }
    }
    __syncwarp();
    __syncthreads();
  } else if (warp == kGtGradWarp) {
    // ================= MMA issue, gradient ==========================================================
    const unsigned idesc = tc::idesc_f16(64, kGtGradN) | (1u << 15) | (1u << 16);      // both operands MN-major
    for (int k = 0; k < n_tiles; ++k) {
      const int s = k % kGtSlabs;
      CNN_PHASE(0);
      mbar_wait_bounded(&sm.g_free[k & 1], ((unsigned)(k >> 1) & 1u) ^ 1u, status, gave_up);
      CNN_PHASE(1);
      const unsigned d = tmem_base + (unsigned)(kGtGradCol + (k & 1) * kGtGradN);
      bool halt = false;
#pragma unroll 1
      for (int w = 0; w < 6; ++w) {
        const int at = 6 * k + w, slot = at % kGtWindows;
        CNN_PHASE(2);
        mbar_wait_bounded(&sm.dl_full[slot], (unsigned)(at / kGtWindows) & 1u, status, gave_up);
        CNN_PHASE(3);
        __syncwarp();
        if (w == 0) halt = __any_sync(0xffffffffu, k >= stop);
        if (halt) break;
        tc::fence_after_sync();
        const unsigned long long ad = tc::smem_desc(smem_u32(sm.delta[slot]), 128, kGtDeltaBlock);
        const unsigned long long bd = tc::smem_desc(smem_u32(sm.slab[s]) + (unsigned)w * kGtChunk, kGtGroupStride, 16);
        tc::mma_f16_run_elect<8, 256 / 16, 2 * kGtGroupStride / 16>(d, ad, bd, idesc, w ? 1u : 0u);
        tc::mma_commit_elect(&sm.dl_free[slot]);
        if (w == 5) tc::mma_commit_elect(&sm.a_free[s]);      // D is complete, the slab may be overwritten
        CNN_PHASE(4);
      }
      if (halt) break;
    }
    __syncwarp();
    __syncthreads();
  } else if (warp < kGtEpiWarp0) {
    load_tiles(sm, images + img0 * kImg, imgs_here, n_tiles, wexp, level, tmem_base, status);
  } else {
    run_group(sm, labels + img0, imgs_here, n_tiles, wsmax, tmem_base, status);
  }
  if (warp < kGtLoadWarp0) { CNN_PHASE_END(g_phase_clocks_gt); }

  tc::fence_before_sync();
  __syncthreads();
  if (warp == kGtGradWarp) tc::tmem_dealloc(tmem_base, 512);
  // ---- the block's row ----------------------------------------------------------------------------
  if (tid < kOffBc) {
    const int f = tid / 25, i = tid % 25 / 5, j = tid % 5;
    float s[2] = {0.f, 0.f};
#pragma unroll
    for (int part = 0; part < 2; ++part)
#pragma unroll
      for (int x = 0; x < 4; ++x) s[part] += end.d[24 * part + 8 * (f >> 1) + 2 * x + (f & 1)][8 * i + x + j];
    float b = 0.f;
#pragma unroll
    for (int w = 0; w < 12; ++w) b += end.bc[w][f];
    // (not a division: 1 / (255 * 576) in fp32 is 2.9e-8 of itself too large, as the pixels are by 2.4e-8)
    row[kOffWc + tid] = fmaf((float)level, b, (s[1] - s[0]) * __int_as_float((127 + 3 - wexp) << 23)) * (1.f / (255.f * kC * kC));
  } else if (tid < kOffWs) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 12; ++w) s += end.bc[w][tid - kOffBc];
    row[tid] = s / (float)(kC * kC);
  } else if (tid < kOffBs) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 12; ++w) s += end.ws[w][tid - kOffWs];
    row[tid] = s;
  } else if (tid == kOffBs) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 12; ++w) s += end.bs[w];
    row[tid] = s / (float)kS;
  } else if (tid < kOffBs + 1 + kOut) {
    const int o = tid - kOffBs - 1;
    row[kOffBf + o] = end.bf[o];
  } else if (tid >= 192 && tid < 192 + kRowStride - kNParams) {
    const int i = kNParams + tid - 192;
    row[i] = i == kRowErr ? end.err : 0.f;
  } else if (tid >= 256 && tid < 256 + 3 + kGradSkips) {
    const int i = tid - 256;
    reinterpret_cast<int*>(left + blockIdx.x)[i] = i == 0 ? min(imgs_here, (int)stop * kGtImgs) : (i == 1 ? 1 : (i == 2 ? sm.skips : sm.skipped[i - 3]));
  }
  if (sm.skips > 0 || stop < n_tiles) {
    __syncthreads();
    if (tid == 0) push_left(left, pushed);
  }
}

int launch_grad_tc(cnn_net* net, const float* d_images, const unsigned* d_labels, GradShares shares, GradLeft* left, int* pushed, cudaStream_t st) {
  const size_t smem = sizeof(GtSmem) + 128;
  CNN_CUDA(cudaFuncSetAttribute(k_grad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaError_t e = launch_pdl(k_grad_tc, dim3(shares.blocks), dim3(kGtThreads), smem, st, d_images, d_labels, shares, (const float*)net->d_params,
                             net->d_partials, left, pushed, net->d_status);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "k_grad_tc launch");
  return CNN_OK;
}

}  // namespace cnn

#ifdef CNN_PHASE_CLOCKS
// Sums of the SM clock at each stamp for the 20 warps of CTA 0 of the last launch (tuning builds only).
extern "C" int cnn_debug_phase_clocks_gt(long long* out /* [20][16] */) {
  return cudaMemcpyFromSymbol(out, cnn::g_phase_clocks_gt, sizeof(cnn::g_phase_clocks_gt)) == cudaSuccess ? 0 : 2;
}
#endif
