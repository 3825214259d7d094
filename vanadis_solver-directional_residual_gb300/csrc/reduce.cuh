// reduce.cuh -- FP64 sums over a warp, counted in FP64 warp instructions (16
// cycles each on GB300's FP64 pipe).
#pragma once
#include <cuda_runtime.h>

#include "dfloat.cuh"

namespace vdr {

constexpr unsigned FULLR = 0xffffffffu;

// Folds over the 8 lanes of each quarter of the warp.
__device__ __forceinline__ double fold8(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(FULLR, v, o);
  return v;
}
// Sums of Q <= 4 values over a warp; lane 8 q holds quantity q.
template <int Q>
__device__ __forceinline__ double warp_sums(const double (&v)[Q], int lane) {
  const bool up = lane & 16, uq = lane & 8;
  if (Q == 1) {
    double d = v[0] + __shfl_xor_sync(FULLR, v[0], 16);
    return fold8(d + __shfl_xor_sync(FULLR, d, 8));
  }
  if (Q == 2) {  // quantities on the lanes with bit 3 clear and set
    double d = (uq ? v[1 % Q] : v[0]) + __shfl_xor_sync(FULLR, uq ? v[0] : v[1 % Q], 8);
    return fold8(d + __shfl_xor_sync(FULLR, d, 16));
  }
  const double v2 = v[2 % Q], v3 = Q > 3 ? v[3 % Q] : 0.0;
  const double d0 = (up ? v2 : v[0]) + __shfl_xor_sync(FULLR, up ? v[0] : v2, 16);
  const double d1 = (up ? v3 : v[1 % Q]) + __shfl_xor_sync(FULLR, up ? v[1 % Q] : v3, 16);
  return fold8((uq ? d1 : d0) + __shfl_xor_sync(FULLR, uq ? d0 : d1, 8));
}

// a += x * y, the product exact, and the sum's value.
__device__ __forceinline__ void dot_acc(DfAcc &a, float x, float y) {
  const float p = __fmul_rn(x, y);
  const float e = __fmaf_rn(x, y, -p);
  const float t = __fadd_rn(a.s, p);
  const float bp = __fsub_rn(t, a.s);
  const float err = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
  a.s = t;
  a.c = __fadd_rn(a.c, __fadd_rn(err, e));
}
__device__ __forceinline__ double dot_val(const DfAcc &a) {
  return df_to_double(a.s, a.c);
}

}  // namespace vdr
