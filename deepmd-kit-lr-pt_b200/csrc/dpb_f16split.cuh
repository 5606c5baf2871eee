// FP32 values as two FP16 terms for the tensor cores: x s = hi + lo with a
// power-of-two scale s that brings the largest of a row (or matrix) to 2^13 ..
// 2^14. hi + lo then holds 22-23 significant bits of every value within 2^-28
// of the largest, and the rest to 2^-39 of it, as two TF32 terms do at half the
// tensor-core rate. Products are lo hi + hi lo + hi hi (the lo lo term, 2^-22 of
// a product, is left out, as with TF32).
#pragma once

#include <cuda_fp16.h>

#include "dpb_common.cuh"

namespace dpb {

// (x, y) as two FP16 pairs, hi + lo
__device__ __forceinline__ void split_f16(float x, float y, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const unsigned*>(&h);
  lo = *reinterpret_cast<const unsigned*>(&l);
}

// power of two s with bound * s < 2^14 (exponent field clamped so that 1 / s
// is normal too), and its reciprocal
__device__ __forceinline__ float f16_scale(float bound, float& inv) {
  const int e = (__float_as_int(bound) >> 23) & 255;  // bound < 2^(e - 126)
  const int se = min(253, max(1, 267 - e));
  inv = __int_as_float((254 - se) << 23);
  return __int_as_float(se << 23);
}

}  // namespace dpb
