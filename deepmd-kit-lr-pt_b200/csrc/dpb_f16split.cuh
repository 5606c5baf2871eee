// FP32 values as two FP16 terms for the tensor cores: x s = hi + lo with a
// power-of-two scale s that brings the largest of a row (or matrix) to 2^13 ..
// 2^14. FP16 ends at 2^-24, so hi + lo is within max(2^-23 |x s|, 2^-25) of x s: 23
// bits of every value down to 2^-16 of the largest, and below that an absolute
// 2^-38 .. 2^-39 of it (18 bits at 2^-20, 10 at 2^-28), where two TF32 terms, at
// half the tensor-core rate, keep 23 bits at any size. A scale therefore spans
// only values that are summed together: a row of a GEMM's operand, an atom and
// type. Where a bound of the activations takes the place of a row's largest (the
// fitting layers), the bits lost are below the roundings of the activations
// themselves: an adjoint g (1 - y^2) is rounded to 2^-24 |g|. Products are
// lo hi + hi lo + hi hi (the lo lo term, 2^-22 of a product, is left out, as with
// TF32).
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
