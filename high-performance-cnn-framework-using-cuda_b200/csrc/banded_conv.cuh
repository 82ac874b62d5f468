// The banded (Toeplitz) weight operand of the 28x28 net's convolution on the tensor cores, as forward_tc.cu and grad_tc.cu build it.
#pragma once

#include <cuda_fp16.h>

#include "cnn_common.cuh"

namespace cnn {

// A factor on weights in two fp32 parts, so that it costs them no bit.
struct TwoPart {
  float hi, lo;
};
constexpr TwoPart two_part(double v) { return {(float)v, (float)(v - (double)(float)v)}; }

// Eight input columns of one accumulator column, 16 bytes of either part: weight `first` + j of kernel row w (none if that is not 0 to 4) for the j-th of
// them, times the factor, as fp16 high part and remainder.
__device__ __forceinline__ void band_row(const float (&w)[5], int first, TwoPart factor, __half2 (&hi)[4], __half2 (&lo)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float t[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int tap = first + 2 * c + h;
      t[h] = 0.f;
#pragma unroll
      for (int d = 0; d < 5; ++d) t[h] = (tap == d) ? w[d] : t[h];
    }
    hi[c] = __floats2half2_rn(t[0] * factor.hi, t[1] * factor.hi);
    const float2 b = __half22float2(hi[c]);
    lo[c] = __floats2half2_rn(fmaf(t[0], factor.lo, fmaf(t[0], factor.hi, -b.x)), fmaf(t[1], factor.lo, fmaf(t[1], factor.hi, -b.y)));
  }
}

// Accumulator column nn = 24 * (window column in the block) + 8 * (map / 2) + 2 * (column in the window) + map % 2: its map and output column.
__device__ __forceinline__ int band_map(int nn) { return 2 * (nn % 24 / 8) + (nn % 24 & 1); }
__device__ __forceinline__ int band_column(int nn) { return 4 * (nn / 24) + ((nn % 24 & 7) >> 1); }

}  // namespace cnn
