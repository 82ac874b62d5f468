// Shared definitions of the widened configuration (wide.cu: fp32 SIMT kernels and the C ABI;
// wide_tc.cu: the tensor-core kernels).
#pragma once

#include "net.cuh"

namespace cnn {

struct WideDims {
  int H, F, C, P, S;        // C = H-4, P = C/4, S = F*P*P
  int o_wc, o_bc, o_ws, o_bs, o_wf, o_bf, n_params, n_padded;
};

__host__ __device__ inline WideDims make_wide_dims(int H, int F) {
  WideDims d;
  d.H = H; d.F = F; d.C = H - 4; d.P = d.C / 4; d.S = F * d.P * d.P;
  d.o_wc = 0; d.o_bc = d.o_wc + F * 25; d.o_ws = d.o_bc + F; d.o_bs = d.o_ws + 16;
  d.o_wf = d.o_bs + 1; d.o_bf = d.o_wf + kOut * d.S; d.n_params = d.o_bf + kOut;
  d.n_padded = ((d.n_params + 2 + 31) / 32) * 32;
  return d;
}

}  // namespace cnn

struct cnn_wide {
  cnn::WideDims d;
  float* d_params = nullptr;
  // Workspace: one allocation, laid out anew by each call for its images and kernels; it only grows.
  float* arena = nullptr;
  size_t arena_floats = 0;
  int flavour = 1;              // sigmoid flavour (cnn_common.cuh): 1 = the short form (default, as cnn_net), 2 = refined, 0 = reference expression
  int conv_mode = 0;            // 0 fp32 SIMT, 1 fp16 tensor-core operands (one pass), 2 two fp16 parts each (three passes)
  int* d_status = nullptr;      // bounded-wait status word
};

namespace cnn {
// What a call's kernels keep between them.  SIMT path: as, ds [image][map][window]; tensor-core path: [image][window][map].
struct WideWork {
  float *ac = nullptr;          // SIMT training: conv activations [image][map][C][C]
  float *as = nullptr, *ds = nullptr, *delta_f = nullptr, *err = nullptr;
  float *part_c = nullptr, *part_s = nullptr;            // SIMT training: rows of [F][26] and of [17]
  float *part_f = nullptr;      // FC weight-gradient partials of the batch slices
  float *ds_max = nullptr;      // tensor-core training: largest |ds| per block of the kernel that writes it
  float *img_max = nullptr, *scale_of = nullptr;         // tensor-core path: largest pixel of each image; what the scales follow (k_wide_tc)
  float *wf_t = nullptr;                                 // tensor-core path: FC weights [output][window][map]
  float *part_g = nullptr, *part_b = nullptr;            // tensor-core training: see k_wide_tc
  size_t floats = 0;
};

constexpr int kTwPrepBlocks = 592;             // four per SM: the pixels of a large batch are read with enough loads under way
constexpr int kTwF = 64;                       // maps of a tensor-core CTA (more maps: more CTAs)
constexpr int kTwGradN = 48;                   // (i, c): six kernel rows of eight columns
constexpr int kTwGradCols = 4 * kTwF;          // (x, f)
constexpr int kTwPartB = 4 * kTwF + 20;        // floats of a CTA's bias and subsample-filter sums

// Tensor-core path (wide_tc.cu).  Forward: w.img_max, w.scale_of, w.wf_t, w.as from the images.  Backward: from these, w.ds and w.ds_max
// to w.part_g and w.part_b, of *ctas CTAs for each kTwF maps.
bool wide_tc_supported(const WideDims& d);
int wide_tc_max_ctas();
int wide_tc_forward(cnn_wide* w, const WideWork& k, const float* d_images, long n, cudaStream_t st);
int wide_tc_backward(cnn_wide* w, const WideWork& k, const float* d_images, long n, int ds_blocks, int* ctas, cudaStream_t st);
}  // namespace cnn
