// block_cols.cuh -- state of the block solve (block.cu, block_rows.cu): K
// independent iterations over block vectors X[n K + k], K = 16, 32 or 64.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "dfloat.cuh"
#include "reduce.cuh"
#include "vdr_internal.h"

namespace vdr {

constexpr int BT = 512;  // threads per block of the block-vector kernels

// device workspace of the block solve, carved from h.bk_f / h.bk_d
constexpr int BK_COLS = 20 * 64;            // per-column doubles and ints
constexpr int BK_PARTIALS = 2 * 64 * 2048;  // NQ x K x blocks
constexpr int BK_MAX_GRID = 2048;

// ------------------------------------------------------ block Krylov state
struct BState {
  unsigned ticket;
  int done, iter, itmax;
  double tol;
};
// per-column arrays, each of length K (kept in one device buffer)
struct BCols {
  double *bnrm2, *err, *rho, *rho_old, *alpha, *omega, *snrm;
  double *rho_next;
  double *tol;  // the column's inner tolerance
  int *active, *sconv, *status;
};

struct BVec {
  long n;  // N*K
  int K;
  BState *st;
  BCols c;
  double *partials;  // [q][k][block]
  const float *b, *dinv;  // dinv per node
  const unsigned char *m; // per node
  float *x, *r, *rh, *p, *v, *s, *t;
  int kshift;               // K = 1 << kshift
  const double *outer_err;  // per column FP64 residual of the refinement
  double outer_tol;         // columns already at outer_tol stay inactive
};

// Grid-stride loops.  BLOOP: over the N*K block entries, one per thread per
// trip (the FP64 glue kernels below).  ULOOP: over units of four
// consecutive columns 4g .. 4g+3 of one node row (unit j = node * K/4 + g,
// float4 loads and stores); the stride is a multiple of K/4, so a thread's
// column group g = threadIdx.x % (K/4) never changes.
#define BSTRIDE ((long)gridDim.x * blockDim.x)
#define BLOOP(i)                                                      \
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; \
       i += BSTRIDE)
#define ULOOP(j)                                                           \
  for (long j = (long)blockIdx.x * blockDim.x + threadIdx.x; j < (a.n >> 2); \
       j += BSTRIDE)

__device__ __forceinline__ float4 ld4(const float *p, long j) {
  return reinterpret_cast<const float4 *>(p)[j];
}
__device__ __forceinline__ void st4(float *p, long j, float4 v) {
  reinterpret_cast<float4 *>(p)[j] = v;
}
__device__ __forceinline__ float f4(const float4 &v, int c) {
  return c == 0 ? v.x : (c == 1 ? v.y : (c == 2 ? v.z : v.w));
}

// ---- the solve on assembled rows (block_rows.cu) ----
struct BlockRows {
  const float4 *rows;  // [N][7]: 27 scaled entries and a zero
  const float2 *S;     // the FP64-accurate pairs [27][N]
  const unsigned *nm;
  int N, nax, nay, naz;
  int nxt, nyt, grid;  // tiles along x and y, blocks
  int *err;            // set where a bounded wait ran out
};
struct BlockOuter {
  double *err, *scale, *bb;          // per column
  unsigned long long *rmax, *bmax;   // bits of max |R|, max |B|
  int *xexp;                         // largest exponent of X
};
// The map of a node-major array of `words` floats a node on the structured
// grid: dimensions (words, nax, nay, naz), box (words, bx, by, 1); nodes
// outside the grid read as zero.
bool make_node_map(CUtensorMap *m, const float *base, int words, int nax, int nay, int naz,
                   int bx, int by);
bool block_rows_usable(Handle &h, int K, BlockRows *g);
// One warp waits for a copy that is never issued, gives up after `limit`
// clocks, drains the ring and sets `bit` of *err.
cudaError_t launch_ring_timeout(int *err, int bit, long long limit, cudaStream_t s);
cudaError_t block_rows_mask(const BVec &a, const BlockOuter &o, double *X, int *nonzero, int grid,
                            cudaStream_t s);
cudaError_t block_rows_residual(const BVec &a, const BlockRows &g, const BlockOuter &o,
                                const double *B, const double *X, double *R, bool zero_x,
                                bool first, int grid, cudaStream_t s);
cudaError_t block_rows_iterations(const BVec &a, const BlockRows &g, int count, int grid,
                                  cudaStream_t s);
cudaError_t block_rows_begin(const BVec &a, cudaStream_t s);
cudaError_t block_rows_update(const BVec &a, const BlockOuter &o, double *X, int grid,
                              cudaStream_t s);

}  // namespace vdr
