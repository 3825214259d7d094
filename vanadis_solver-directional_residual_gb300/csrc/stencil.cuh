// stencil.cuh -- the assembled operator on the canonical structured
// numbering, and the row product every kernel that applies it shares.
//
// On that numbering a node couples with its 26 neighbours and itself, so
// P A P has at most 27 entries per row: 27 pairs (216 bytes) per node where
// the element matrices hold 64 pairs (512 bytes) per element and there are
// about as many nodes as elements.  A Krylov apply is bound by HBM, so the
// rows are summed once per operator (stencil_assemble) and every apply
// gathers: node n's output is one thread's sum, with no atomics, no cleared
// output vector, and inner products with it can be formed where it is.
// Measured at 8.5M nodes (2.05 GB with the two vectors of the fused inner
// product): 0.34 ms, 6.0 TB/s, against 0.77 ms for the 4.77 GB element-wise
// apply; at 1.08M nodes 41 us against 105 us.
//
// Layout: S[k N + n] = (hi, lo) of the coupling of node n with node n +
// off(k), k = 9 (dz + 1) + 3 (dy + 1) + (dx + 1), off = dx + nax dy + nax
// nay dz; a warp reads 256 contiguous bytes per k for A and for A^T.
// nm[n]: bit k set where some element couples the two nodes and neither is
// a Dirichlet node (rows and columns of Dirichlet nodes are zero); x is read
// through set bits only, so what lies beyond the mesh's faces, at the other
// end of a row or on a Dirichlet node never enters the sum or its scale.
#pragma once
#include <cuda_runtime.h>

#include "dfloat.cuh"
#include "vdr_internal.h"

namespace vdr {

struct StencilView {
  const float2 *S = nullptr;
  const unsigned *nm = nullptr;  // and before it what pair_head reads
  int N = 0, nax = 0, pl = 0;
};

constexpr int NM_LEAD = 32;  // words before nm; the last: the biased FP32
                             // exponent of the largest entry
// A vector whose largest biased exponent is e becomes pairs by 2^-(e + head -
// 1023): largest magnitude in [2^h, 2^(h + 1)), h = -head = 200 - top, at most
// 72.  (The exponents that the iterations keep have head added already.)  A
// row's 27 products then stay below 2^128 for a vector 2^48 times larger than
// the one that gave e: the iterations scale a direction and its s^ by the
// direction before.  (2^53 times larger, FP64 would have nothing left of the
// smaller one; what does not fit reads as a breakdown.)  At the other end,
// with entries around 1, values down to 2^-198 of the largest are held and
// down to 2^-174 in full; with the largest entries that the store allows
// (2^123 once summed) it is 2^-76 and 2^-52.
__device__ __forceinline__ int pair_head(const unsigned *nm) {
  return max((int)nm[-1] - 200, -72);
}

__device__ __forceinline__ int stencil_off(int k, int nax, int pl) {
  return (k / 9 - 1) * pl + (k / 3 % 3 - 1) * nax + (k % 3 - 1);
}

// One row in FP64 from the merged pairs: where a gathered value is inf/NaN.
template <bool TRANS>
__device__ __noinline__ double stencil_row_fp64(const StencilView v, long n,
                                                const double *x) {
  double out = 0.0;
  const unsigned m = v.nm[n];
  for (int k = 0; k < 27; k++) {
    if (!((m >> k) & 1u)) continue;
    const long q = n + stencil_off(k, v.nax, v.pl);
    const float2 a = TRANS ? v.S[(size_t)(26 - k) * v.N + q] : v.S[(size_t)k * v.N + n];
    out += df_to_double(a.x, a.y) * x[q];
  }
  return out;
}

// (A x)_n, or (A^T x)_n: double-float products on the FP32 pipe, plane by
// plane, each of the three 9-node planes scaled by its own power of two (its
// largest gathered value in [1/8, 1/4)) as the element apply scales its 8
// nodes; entries stay below 2^123 (eight element entries below the store's
// 2^120), so a plane's sum stays finite.
// Nine matrix pairs and nine x are in flight per thread at a time.
// KEEP: the rows are read again soon and fit in L2 (plain loads); otherwise
// they stream through it (evict first), leaving it to the vectors.
template <bool TRANS, bool KEEP>
__device__ __forceinline__ double stencil_row(const StencilView &v, long n,
                                              const double *x) {
  const unsigned m = __ldg(v.nm + n);
  double out = 0.0;
  bool bad = false;
#pragma unroll
  for (int z = 0; z < 3; z++) {
    if (!((m >> (9 * z)) & 511u)) continue;
    double xv[9];
    float2 a[9];
    int emax = 0;
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const int k = 9 * z + c;
      const bool on = (m >> k) & 1u;
      const long q = n + ((z - 1) * v.pl + (c / 3 - 1) * v.nax + (c % 3 - 1));
      const float2 *s = TRANS ? v.S + (size_t)(26 - k) * v.N + q : v.S + (size_t)k * v.N + n;
      a[c] = on ? (KEEP ? __ldcg(s) : __ldcs(s)) : make_float2(0.f, 0.f);
      xv[c] = on ? x[q] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < 9; c++) emax = max(emax, df_exp(xv[c]));
    const int shift = emax - 1020;
    DfAcc acc{0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 9; c++) {
      float xh, xl;
      df_split(xv[c], xh, xl, bad, shift);
      df_fma_acc(acc, a[c].x, a[c].y, xh, xl);
    }
    double o = df_to_double(acc.s, acc.c);
    if (!df_scale(o, shift)) o = ldexp(o, shift);
    out += o;
  }
  return bad ? stencil_row_fp64<TRANS>(v, n, x) : out;
}

// The Krylov iteration's form: the input already split into pairs, scaled by
// one power of two per vector (pair_head), with zeros for a plane and a row
// beyond both ends (stencil_pad), so that the 27 products need no mask, no
// index clamp and no split: the rows hold zeros wherever no coupling exists.
// A^T reads its neighbours' rows at shifted places, which stay inside S.
template <bool TRANS, bool KEEP>
__device__ __forceinline__ double stencil_row_pairs(const StencilView &v, long n,
                                                    const float2 *xp, int shift) {
  DfAcc acc{0.f, 0.f};
#pragma unroll
  for (int z = 0; z < 3; z++) {
    float2 a[9], xv[9];
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const int k = 9 * z + c;
      const long q = n + ((z - 1) * v.pl + (c / 3 - 1) * v.nax + (c % 3 - 1));
      const float2 *s = TRANS ? v.S + (size_t)(26 - k) * v.N + q : v.S + (size_t)k * v.N + n;
      a[c] = KEEP ? __ldcg(s) : __ldcs(s);
      xv[c] = xp[q];
    }
#pragma unroll
    for (int c = 0; c < 9; c++) df_fma_acc(acc, a[c].x, a[c].y, xv[c].x, xv[c].y);
  }
  double o = df_to_double(acc.s, acc.c);
  if (!df_scale(o, shift)) o = ldexp(o, shift);
  return o;
}

// d * 2^-shift as a pair; what does not fit (inf, NaN, 2^128 and above)
// becomes inf, which the next inner product finds.
__device__ __forceinline__ float2 stencil_pair(double d, int shift) {
  float2 r;
  bool bad = false;
  df_split(d, r.x, r.y, bad, shift);
  if (bad) r.x = INFINITY;
  return r;
}

// zeros before and after a pair vector
inline size_t stencil_pad(const Handle &h) {
  return ((size_t)h.nax * h.nay + h.nax + 1 + 31) & ~(size_t)31;
}

StencilView stencil_view(const Handle &h);
bool stencil_keep(const Handle &h);  // the rows fit in L2 beside the vectors

}  // namespace vdr
