// batch.cu -- many independent meshes solved together.
//
// The meshes are concatenated into one block-diagonal system (node and
// element ranges per mesh; no element couples two meshes), so the element
// build and the operator apply of the handle process every mesh in single
// launches.  The Krylov method is Jacobi-BiCGStab with one set of scalars
// per mesh ("segment"):
//
//  * the node range is cut into tiles that never straddle a segment; a
//    block processes one tile, so its partial sums belong to one segment;
//  * each tile writes its partials and takes a ticket on its segment; the
//    last tile of a segment adds the segment's partials in tile order
//    (deterministic) and updates the segment's scalars -- no grid-wide
//    wait and no spin anywhere;
//  * a segment that converges (or breaks down) freezes: its vectors stop
//    changing, and when the last active segment finishes the global `done`
//    flag is raised, which every kernel checks at entry, so K iterations of
//    all meshes are captured once as a CUDA graph and replayed;
//  * the tile size and block size are chosen by measurement at the first
//    solve (autotuner over a representative segmented reduction pass on the
//    actual segment layout), on assembled rows by the number of rows.
//
// Where every mesh is numbered canonically (its elements in the order of its
// grid) and the handle applies by assembled rows, the iteration is the
// three-kernel form on the 27-point rows: every mesh's pair vectors have
// their own zero pads, and a row's products run over its own mesh's axes.
// 216 bytes of rows and 12 of vectors per node and product instead of 512
// per element, a scatter and three more kernels: 96 cubes of 8 to 32
// elements an edge, 1.18 M nodes, 19.9 -> 9.9 ms per solve with its
// operator and right-hand side.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "reduce.cuh"
#include "stencil.cuh"
#include "vdr_internal.h"

namespace vdr {
namespace {

struct SegTile {
  int seg, start, end;
};

// Per-segment state, structure of arrays in one device buffer.
struct SegState {
  double *bnrm2, *err, *rho, *rho_old, *alpha, *omega, *snrm, *rhs, *rho_next, *beta, *partials;
  int *pexp, *pmax, *pmax_next, *rmax;  // exponents of the assembled form
  int *active, *sconv, *status, *iter, *tile_begin, *tile_count;
  unsigned *ticket;
  int *nactive;  // active segments left
  int *done;     // 1 when no segment is active (gates every kernel)
  int itmax;
  double tol;
};

struct SegVec {
  const SegTile *tiles;
  SegState s;
  const double *b, *dinv;
  const unsigned char *m;
  double *x, *r, *rh, *p, *v, *ph, *sv, *sh, *t;
  // the assembled form: rows, grids, pair vectors, w = A^T rh (in ph's place)
  StencilView rows;
  const SegMesh *mesh;
  float2 *php, *shp;
  double *w;
};

// Writes this tile's partials; true in thread 0 of the segment's last tile
// with the segment totals in out (its first warp adds the tiles' partials in
// a fixed order).
template <int NQ>
__device__ __forceinline__ bool seg_sum(double (&v)[NQ], const SegVec &a, int tile,
                                        int seg, double (&out)[NQ]) {
  __shared__ double sm[32][4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  const double f = warp_sums<NQ>(v, lane);
  __syncthreads();
  if ((lane & 7) == 0 && (lane >> 3) < NQ) sm[w][lane >> 3] = f;
  __syncthreads();
  if (w != 0) return false;
  const int tb = a.s.tile_begin[seg], tc = a.s.tile_count[seg];
  const int q = lane >> 3;
  double c = 0.0;
  for (int k = lane & 7; k < nw; k += 8) c += sm[k][q < NQ ? q : 0];
  c = fold8(c);
  if ((lane & 7) == 0 && q < NQ) a.s.partials[(size_t)q * gridDim.x + tile] = c;
  __threadfence();
  __syncwarp();
  unsigned last = 0u;
  if (lane == 0) last = atomicAdd(a.s.ticket + seg, 1u) == (unsigned)(tc - 1);
  if (!__shfl_sync(FULLR, last, 0)) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NQ; k++) {
    v[k] = 0.0;
    for (int t = lane; t < tc; t += 32)
      v[k] += __ldcg(a.s.partials + (size_t)k * gridDim.x + tb + t);
  }
  const double g = warp_sums<NQ>(v, lane);
#pragma unroll
  for (int k = 0; k < NQ; k++) out[k] = __shfl_sync(FULLR, g, 8 * k);
  if (lane == 0) a.s.ticket[seg] = 0u;
  return lane == 0;
}

__device__ __forceinline__ void seg_finish(const SegVec &a, int seg, int status) {
  a.s.active[seg] = 0;
  a.s.status[seg] = status;
  if (atomicSub(a.s.nactive, 1) == 1) *a.s.done = 1;
}

#define TLOOP(i) for (int i = tl.start + threadIdx.x; i < tl.end; i += blockDim.x)

// r = b - r (r holds A x); rh = r; per-segment ||b||, ||r||.
__global__ void sg_start(SegVec a) {
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  double v[2] = {0.0, 0.0};
  TLOOP(i) {
    const double bi = a.b[i];
    const double ri = bi - a.r[i];
    a.r[i] = ri;
    a.rh[i] = ri;
    v[0] += bi * bi;
    v[1] += ri * ri;
  }
  double o[2];
  if (seg_sum<2>(v, a, tile, tl.seg, o)) {
    const int s = tl.seg;
    a.s.bnrm2[s] = o[0];
    a.s.rho[s] = o[1];
    a.s.rho_old[s] = 1.0;
    a.s.alpha[s] = 1.0;
    a.s.omega[s] = 1.0;
    a.s.sconv[s] = 0;
    a.s.iter[s] = 0;
    const double err = o[0] > 0.0 ? sqrt(o[1] / o[0]) : 0.0;
    a.s.err[s] = err;
    if (o[0] == 0.0 || err <= a.s.tol) {
      seg_finish(a, s, VDR_OK);
    } else if (!(err == err)) {
      seg_finish(a, s, VDR_BREAKDOWN);
    } else {
      a.s.status[s] = VDR_NOT_CONVERGED;
    }
  }
}

// x = 0 on segments whose b is zero (their solution).
__global__ void sg_zero(SegVec a) {
  const SegTile tl = a.tiles[blockIdx.x];
  if (a.s.bnrm2[tl.seg] != 0.0) return;
  TLOOP(i) a.x[i] = 0.0;
}

__global__ void sg_p(SegVec a) {
  if (*a.s.done) return;
  const SegTile tl = a.tiles[blockIdx.x];
  const int s = tl.seg;
  const bool act = a.s.active[s];
  if (!act) return;  // frozen: its elements are skipped by the apply too
  const bool first = a.s.iter[s] == 0;
  const double beta = first ? 0.0
      : (a.s.rho[s] / a.s.rho_old[s]) * (a.s.alpha[s] / a.s.omega[s]);
  const double om = a.s.omega[s];
  TLOOP(i) {
    double pi = 0.0;
    if (act) pi = first ? a.r[i] : a.r[i] + beta * (a.p[i] - om * a.v[i]);
    a.p[i] = pi;
    a.ph[i] = a.m[i] ? 0.0 : pi * a.dinv[i];
    a.v[i] = 0.0;
  }
}

__global__ void sg_alpha(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  if (!a.s.active[tl.seg]) return;
  double v[1] = {0.0};
  TLOOP(i) v[0] += a.rh[i] * a.v[i];
  double o[1];
  if (seg_sum<1>(v, a, tile, tl.seg, o)) {
    const int s = tl.seg;
    if (a.s.active[s]) {
      if (o[0] == 0.0 || !isfinite(o[0])) {
        a.s.alpha[s] = 0.0;
        seg_finish(a, s, VDR_BREAKDOWN);
      } else {
        a.s.alpha[s] = a.s.rho[s] / o[0];
      }
    }
  }
}

__global__ void sg_s(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  if (!a.s.active[s]) return;
  const double al = a.s.active[s] ? a.s.alpha[s] : 0.0;
  double v[1] = {0.0};
  TLOOP(i) {
    const double si = a.r[i] - al * a.v[i];
    a.sv[i] = si;
    a.sh[i] = a.m[i] ? 0.0 : si * a.dinv[i];
    a.t[i] = 0.0;
    v[0] += si * si;
  }
  double o[1];
  if (seg_sum<1>(v, a, tile, s, o)) {
    const double sn = a.s.bnrm2[s] > 0.0 ? sqrt(o[0] / a.s.bnrm2[s]) : 0.0;
    a.s.snrm[s] = sn;
    a.s.sconv[s] = (a.s.active[s] && sn <= a.s.tol) ? 1 : 0;
  }
}

__global__ void sg_omega(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  if (!a.s.active[tl.seg]) return;
  double v[2] = {0.0, 0.0};
  TLOOP(i) {
    v[0] += a.t[i] * a.sv[i];
    v[1] += a.t[i] * a.t[i];
  }
  double o[2];
  if (seg_sum<2>(v, a, tile, tl.seg, o)) {
    const int s = tl.seg;
    if (a.s.active[s] && !a.s.sconv[s]) {
      if (o[1] == 0.0 || !isfinite(o[1]) || !isfinite(o[0])) {
        a.s.omega[s] = 0.0;
        seg_finish(a, s, VDR_BREAKDOWN);
      } else {
        a.s.omega[s] = o[0] / o[1];
      }
    }
  }
}

__global__ void sg_xr(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  const bool act = a.s.active[s];
  if (!act) return;
  const bool sc = a.s.sconv[s];
  const double al = a.s.alpha[s];
  const double om = sc ? 0.0 : a.s.omega[s];
  double v[2] = {0.0, 0.0};
  TLOOP(i) {
    double ri = a.r[i];
    if (act) {
      a.x[i] += al * a.ph[i] + om * a.sh[i];
      ri = sc ? a.sv[i] : a.sv[i] - om * a.t[i];
      a.r[i] = ri;
    }
    v[0] += ri * ri;
    v[1] += a.rh[i] * ri;
  }
  double o[2];
  if (seg_sum<2>(v, a, tile, s, o)) {
    if (act) {
      a.s.iter[s] += 1;
      a.s.rho_old[s] = a.s.rho[s];
      a.s.rho[s] = o[1];
      const double err = sqrt(o[0] / a.s.bnrm2[s]);
      a.s.err[s] = err;
      if (!(err == err)) {
        seg_finish(a, s, VDR_BREAKDOWN);
      } else if (err <= a.s.tol || sc) {
        if (sc) a.s.err[s] = a.s.snrm[s];
        seg_finish(a, s, VDR_OK);
      } else if (o[1] == 0.0 || om == 0.0) {
        seg_finish(a, s, VDR_BREAKDOWN);
      } else if (a.s.iter[s] >= a.s.itmax) {
        seg_finish(a, s, VDR_NOT_CONVERGED);
      }
    }
  }
}

// ---- the iteration on assembled rows (krylov.cu's three-kernel form, one
// set of scalars per mesh) ----
__device__ __forceinline__ StencilView mesh_rows(const SegVec &a, const SegMesh &g) {
  StencilView v = a.rows;
  v.nax = g.nax;
  v.pl = g.nax * g.nay;
  return v;
}

// Largest exponents of r and D^-1 r of every mesh.
__global__ void __launch_bounds__(512, 2) sgr_exponents(SegVec a) {
  const SegTile tl = a.tiles[blockIdx.x];
  if (!a.s.active[tl.seg]) return;
  int e = 0, er = 0;
  TLOOP(i) {
    const double ri = a.r[i];
    er = max(er, df_exp(ri));
    if (!a.m[i]) e = max(e, df_exp(ri * a.dinv[i]));
  }
  e = __reduce_max_sync(FULLR, e);
  er = __reduce_max_sync(FULLR, er);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(a.s.pmax + tl.seg, e);
    atomicMax(a.s.rmax + tl.seg, er);
  }
}

// p = r, p^ and rh (in s^'s place, for w) as pairs.
__global__ void __launch_bounds__(512, 2) sgr_first(SegVec a) {
  const SegTile tl = a.tiles[blockIdx.x];
  const int s = tl.seg;
  if (!a.s.active[s]) return;
  const long at = a.mesh[s].shift;
  const int e = a.s.pmax[s], er = a.s.rmax[s], base = 1023 - pair_head(a.rows.nm);
  TLOOP(i) {
    const double ri = a.r[i];
    const bool m = a.m[i] != 0;
    a.p[i] = ri;
    a.php[i + at] = m ? make_float2(0.f, 0.f) : stencil_pair(ri * a.dinv[i], e - base);
    a.shp[i + at] = m ? make_float2(0.f, 0.f) : stencil_pair(ri, er - base);
  }
  if (tl.start == a.mesh[s].n0 && threadIdx.x == 0) a.s.pexp[s] = e + 1023 - base;
}

__device__ __forceinline__ void seg_alpha(const SegVec &a, int s, double wp) {
  if (wp == 0.0 || !isfinite(wp)) {
    a.s.alpha[s] = 0.0;
    seg_finish(a, s, VDR_BREAKDOWN);
  } else {
    a.s.alpha[s] = a.s.rho[s] / wp;
  }
}

// w = A^T rh (through set bits only: a neighbour's row may be another mesh's)
__global__ void __launch_bounds__(512, 2) sgr_w(SegVec a) {
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  if (!a.s.active[s]) return;
  const SegMesh g = a.mesh[s];
  const StencilView v = mesh_rows(a, g);
  const float2 *xp = a.shp + g.shift;
  const int shift = a.s.rmax[s] + pair_head(v.nm) - 1023;
  double q[1] = {0.0};
  TLOOP(i) {
    const unsigned m = v.nm[i];
    DfAcc acc{0.f, 0.f};
#pragma unroll 9
    for (int k = 0; k < 27; k++) {
      const long n = (long)i + stencil_off(k, v.nax, v.pl);
      const bool on = (m >> k) & 1u;
      const float2 e = on ? v.S[(size_t)(26 - k) * v.N + n] : make_float2(0.f, 0.f);
      const float2 x = xp[n];
      df_fma_acc(acc, e.x, e.y, x.x, x.y);
    }
    double o = df_to_double(acc.s, acc.c);
    if (!df_scale(o, shift)) o = ldexp(o, shift);
    a.w[i] = o;
    if (!a.m[i]) q[0] += o * (a.p[i] * a.dinv[i]);
  }
  double o[1];
  if (seg_sum<1>(q, a, tile, s, o)) {
    a.s.pmax[s] += pair_head(v.nm);
    seg_alpha(a, s, o[0]);
  }
}

template <bool KEEP>
__global__ void __launch_bounds__(512, 2) sgr_v(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  if (!a.s.active[s]) return;
  const SegMesh g = a.mesh[s];
  const StencilView v = mesh_rows(a, g);
  const int shift = a.s.pexp[s] - 1023;
  const double al = a.s.alpha[s];
  double q[2] = {0.0, 0.0};
  TLOOP(i) {
    const double ri = a.r[i], di = a.dinv[i], hi = a.rh[i];
    const bool m = a.m[i] != 0;
    const double o = stencil_row_pairs<false, KEEP>(v, i, a.php + g.shift, shift);
    const double si = ri - al * o;
    a.v[i] = o;
    a.sv[i] = si;
    a.shp[i + g.shift] = m ? make_float2(0.f, 0.f) : stencil_pair(si * di, shift);
    q[0] += si * si;
    q[1] += hi * si;
  }
  double o[2];
  if (seg_sum<2>(q, a, tile, s, o)) {
    const double sn = a.s.bnrm2[s] > 0.0 ? sqrt(o[0] / a.s.bnrm2[s]) : 0.0;
    a.s.snrm[s] = sn;
    a.s.rhs[s] = o[1];
    a.s.sconv[s] = sn <= a.s.tol ? 1 : 0;
  }
}

template <bool KEEP>
__global__ void __launch_bounds__(512, 2) sgr_t(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  if (!a.s.active[s] || a.s.sconv[s]) return;
  const SegMesh g = a.mesh[s];
  const StencilView v = mesh_rows(a, g);
  const int shift = a.s.pexp[s] - 1023;
  double q[3] = {0.0, 0.0, 0.0};
  TLOOP(i) {
    const double si = a.sv[i], hi = a.rh[i];
    const double o = stencil_row_pairs<false, KEEP>(v, i, a.shp + g.shift, shift);
    a.t[i] = o;
    q[0] += o * si;
    q[1] += o * o;
    q[2] += hi * o;
  }
  double o[3];
  if (seg_sum<3>(q, a, tile, s, o)) {
    if (o[1] == 0.0 || !isfinite(o[1]) || !isfinite(o[0])) {
      a.s.omega[s] = 0.0;
      seg_finish(a, s, VDR_BREAKDOWN);
    } else {
      a.s.omega[s] = o[0] / o[1];
      a.s.rho_next[s] = a.s.rhs[s] - a.s.omega[s] * o[2];
      a.s.beta[s] = (a.s.rho_next[s] / a.s.rho[s]) * (a.s.alpha[s] / a.s.omega[s]);
    }
  }
}

__global__ void __launch_bounds__(512, 2) sgr_p(SegVec a) {
  if (*a.s.done) return;
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  const int s = tl.seg;
  if (!a.s.active[s]) return;
  const double al = a.s.alpha[s];
  double q[2] = {0.0, 0.0}, o[2];
  if (a.s.sconv[s]) {  // s met the tolerance: x += alpha p^
    TLOOP(i) if (!a.m[i]) a.x[i] += a.dinv[i] * (al * a.p[i]);
    if (seg_sum<2>(q, a, tile, s, o)) {
      a.s.iter[s] += 1;
      a.s.err[s] = a.s.snrm[s];
      seg_finish(a, s, VDR_OK);
    }
    return;
  }
  const double om = a.s.omega[s], rho1 = a.s.rho_next[s];
  const double beta = a.s.beta[s];
  const int e = a.s.pmax[s], shift = e - 1023;
  const long at = a.mesh[s].shift;
  int em = 0;
  TLOOP(i) {
    const double si = a.sv[i], pi0 = a.p[i], di = a.dinv[i];
    const bool m = a.m[i] != 0;
    const double ri = si - om * a.t[i];
    const double pi = ri + beta * (pi0 - om * a.v[i]);
    if (!m) a.x[i] += di * (al * pi0 + om * si);
    a.r[i] = ri;
    a.p[i] = pi;
    const double hi = m ? 0.0 : pi * di;
    a.php[i + at] = stencil_pair(hi, shift);
    em = max(em, df_exp(hi));
    q[0] += ri * ri;
    q[1] += a.w[i] * hi;
  }
  em = __reduce_max_sync(FULLR, em);
  if ((threadIdx.x & 31) == 0) atomicMax(a.s.pmax_next + s, em);
  __threadfence();
  if (seg_sum<2>(q, a, tile, s, o)) {
    a.s.iter[s] += 1;
    a.s.pexp[s] = e;
    a.s.pmax[s] = atomicExch(a.s.pmax_next + s, 0) + pair_head(a.rows.nm);
    a.s.rho[s] = rho1;
    const double err = sqrt(o[0] / a.s.bnrm2[s]);
    a.s.err[s] = err;
    if (!(err == err) || !isfinite(rho1)) {
      seg_finish(a, s, VDR_BREAKDOWN);
    } else if (err <= a.s.tol) {
      seg_finish(a, s, VDR_OK);
    } else if (rho1 == 0.0 || om == 0.0) {
      seg_finish(a, s, VDR_BREAKDOWN);
    } else if (a.s.iter[s] >= a.s.itmax) {
      seg_finish(a, s, VDR_NOT_CONVERGED);
    } else {
      seg_alpha(a, s, o[1]);
    }
  }
}

// Autotuning probe: a two-vector segmented dot product (the shape of the
// reduction passes); results go to scratch.
__global__ void sg_probe(SegVec a) {
  const int tile = blockIdx.x;
  const SegTile tl = a.tiles[tile];
  double v[2] = {0.0, 0.0};
  TLOOP(i) {
    v[0] += a.b[i] * a.r[i];
    v[1] += a.r[i] * a.r[i];
  }
  double o[2];
  if (seg_sum<2>(v, a, tile, tl.seg, o)) a.s.snrm[tl.seg] = o[0] + o[1];
}

}  // namespace

// Builds the tile list for a tile size (nodes) from the segment offsets.
static void make_tiles(const std::vector<int> &off, int tile, std::vector<SegTile> &tiles,
                       std::vector<int> &begin, std::vector<int> &count) {
  tiles.clear();
  begin.assign(off.size() - 1, 0);
  count.assign(off.size() - 1, 0);
  for (size_t s = 0; s + 1 < off.size(); s++) {
    begin[s] = (int)tiles.size();
    for (int i = off[s]; i < off[s + 1]; i += tile)
      tiles.push_back(SegTile{(int)s, i, std::min(off[s + 1], i + tile)});
    count[s] = (int)tiles.size() - begin[s];
  }
}

int set_segments(Handle &h, int nseg, const int *node_off) {
  if (nseg < 1 || !node_off || node_off[0] != 0 || node_off[nseg] != h.N) {
    set_error("segments: need node_off[0] = 0, node_off[nseg] = N");
    return VDR_BAD_ARGUMENT;
  }
  for (int s = 0; s < nseg; s++)
    if (node_off[s + 1] <= node_off[s]) {
      set_error("segments: node offsets must increase");
      return VDR_BAD_ARGUMENT;
    }
  // every element's nodes must lie in one segment
  std::vector<int> conn((size_t)h.E * 8);
  cudaError_t e = cudaMemcpy(conn.data(), h.conn, sizeof(int) * conn.size(),
                             cudaMemcpyDeviceToHost);
  if (e) return cuda_fail(e, "segments: connectivity");
  std::vector<int> off(node_off, node_off + nseg + 1);
  std::vector<int> eseg(h.E);
  for (long p = 0; p < h.E; p++) {
    const int n0 = conn[p] & NODE_BITS;
    const int s0 = (int)(std::upper_bound(off.begin(), off.end(), n0) - off.begin()) - 1;
    eseg[p] = s0;
    for (int k = 1; k < 8; k++) {
      const int n = conn[(size_t)k * h.E + p] & NODE_BITS;
      if (n < off[s0] || n >= off[s0 + 1]) {
        set_error("segments: an element couples two segments");
        return VDR_BAD_ARGUMENT;
      }
    }
  }
  if (!h.seg_of_elem && (e = cudaMalloc(&h.seg_of_elem, sizeof(int) * (size_t)h.E)))
    return cuda_fail(e, "segments: alloc");
  if ((e = cudaMemcpy(h.seg_of_elem, eseg.data(), sizeof(int) * (size_t)h.E,
                      cudaMemcpyHostToDevice)))
    return cuda_fail(e, "segments: upload");
  h.seg_off = off;
  h.seg_rows = false;
  if (h.seg_mesh) cudaFree(h.seg_mesh);
  if (h.seg_x) cudaFree(h.seg_x);
  h.seg_mesh = nullptr;
  h.seg_x = nullptr;
  h.seg_pairs = 0;
  h.seg_largest = 0;
  // every mesh in the canonical numbering, elements in its order: the solve
  // can run on assembled rows
  std::vector<SegMesh> meshes(nseg);
  bool canonical = !h.perm_d;
  long e0 = 0;
  for (int s = 0; s < nseg && canonical; s++) {
    SegMesh &g = meshes[s];
    const long nodes = off[s + 1] - off[s], E = h.E;
    const auto node = [&](int k, long p) { return (long)(conn[k * E + p] & NODE_BITS); };
    if (e0 >= E || eseg[e0] != s) {
      canonical = false;
      break;
    }
    const long nax = node(3, e0) - node(0, e0), pl = node(4, e0) - node(0, e0);
    if (nax < 2 || pl < 2 * nax || pl % nax || nodes % pl || nodes / pl < 2) {
      canonical = false;
      break;
    }
    const long nay = pl / nax, naz = nodes / pl, count = (nax - 1) * (nay - 1) * (naz - 1);
    if (e0 + count > E) {
      canonical = false;
      break;
    }
    const long at[8] = {0, 1, 1 + nax, nax, pl, 1 + pl, 1 + pl + nax, pl + nax};
    for (long q = 0; q < count && canonical; q++) {
      const long i = q % (nax - 1), r = q / (nax - 1), j = r % (nay - 1), k = r / (nay - 1);
      const long base = off[s] + i + nax * j + pl * k;
      for (int c = 0; c < 8; c++) canonical = canonical && node(c, e0 + q) == base + at[c];
    }
    g.n0 = off[s];
    g.nax = (int)nax;
    g.nay = (int)nay;
    g.naz = (int)naz;
    g.e0 = e0;
    const long pad = pl + nax + 1;
    g.shift = (long)h.seg_pairs + pad - off[s];
    h.seg_pairs += (size_t)(nodes + 2 * pad);
    h.seg_largest = std::max(h.seg_largest, nodes);
    e0 += count;
  }
  canonical = canonical && e0 == h.E;
  h.seg_canonical = canonical;
  if (canonical) {
    if ((e = cudaMalloc(&h.seg_mesh, sizeof(SegMesh) * nseg)) ||
        (e = cudaMemcpy(h.seg_mesh, meshes.data(), sizeof(SegMesh) * nseg,
                        cudaMemcpyHostToDevice)))
      return cuda_fail(e, "segments: grids");
  }
  h.seg_tile = 0;  // re-tune at the next solve
  if (h.seg_graph) cudaGraphExecDestroy(h.seg_graph);
  h.seg_graph = nullptr;
  return VDR_OK;
}

namespace {
struct SegLayout {
  SegVec a;
  int ntiles, threads;
};

// Device layout for a tile size: tiles, per-segment arrays, vectors.
cudaError_t seg_layout(Handle &h, int tile, int threads, const double *b, double *x,
                       SegLayout &L) {
  const int nseg = (int)h.seg_off.size() - 1;
  std::vector<SegTile> tiles;
  std::vector<int> begin, count;
  make_tiles(h.seg_off, tile, tiles, begin, count);
  const int nt = (int)tiles.size();
  // doubles: 10 per segment + partials 3 per tile; ints: 10 per segment + 2
  const size_t dwords = (size_t)10 * nseg + 3 * (size_t)nt;
  const size_t iwords = (size_t)10 * nseg + 2 + 3 * (size_t)nt;
  cudaError_t e;
  if (h.seg_dwords < dwords) {
    if (h.seg_d) cudaFree(h.seg_d);
    h.seg_d = nullptr;
    h.seg_dwords = 0;
    if ((e = cudaMalloc(&h.seg_d, sizeof(double) * dwords))) return e;
    h.seg_dwords = dwords;
  }
  if (h.seg_iwords < iwords) {
    if (h.seg_i) cudaFree(h.seg_i);
    h.seg_i = nullptr;
    h.seg_iwords = 0;
    if ((e = cudaMalloc(&h.seg_i, sizeof(int) * iwords))) return e;
    h.seg_iwords = iwords;
  }
  int *ip = h.seg_i;
  SegTile *dt = reinterpret_cast<SegTile *>(ip + 10 * (size_t)nseg + 2);
  if ((e = cudaMemcpyAsync(dt, tiles.data(), sizeof(SegTile) * nt, cudaMemcpyHostToDevice,
                           h.stream)) ||
      (e = cudaMemcpyAsync(ip + 4 * (size_t)nseg, begin.data(), sizeof(int) * nseg,
                           cudaMemcpyHostToDevice, h.stream)) ||
      (e = cudaMemcpyAsync(ip + 5 * (size_t)nseg, count.data(), sizeof(int) * nseg,
                           cudaMemcpyHostToDevice, h.stream)))
    return e;
  SegVec &a = L.a;
  a = SegVec{};
  a.tiles = dt;
  double *dp = h.seg_d;
  a.s.bnrm2 = dp;
  a.s.err = dp + nseg;
  a.s.rho = dp + 2 * (size_t)nseg;
  a.s.rho_old = dp + 3 * (size_t)nseg;
  a.s.alpha = dp + 4 * (size_t)nseg;
  a.s.omega = dp + 5 * (size_t)nseg;
  a.s.snrm = dp + 6 * (size_t)nseg;
  a.s.rhs = dp + 7 * (size_t)nseg;
  a.s.rho_next = dp + 8 * (size_t)nseg;
  a.s.beta = dp + 9 * (size_t)nseg;
  a.s.partials = dp + 10 * (size_t)nseg;
  a.s.active = ip;
  a.s.sconv = ip + nseg;
  a.s.status = ip + 2 * (size_t)nseg;
  a.s.iter = ip + 3 * (size_t)nseg;
  a.s.tile_begin = ip + 4 * (size_t)nseg;
  a.s.tile_count = ip + 5 * (size_t)nseg;
  a.s.ticket = reinterpret_cast<unsigned *>(h.seg_ticket);
  a.s.nactive = ip + 6 * (size_t)nseg;
  a.s.done = ip + 6 * (size_t)nseg + 1;
  a.s.pexp = ip + 6 * (size_t)nseg + 2;
  a.s.pmax = a.s.pexp + nseg;
  a.s.pmax_next = a.s.pmax + nseg;
  a.s.rmax = a.s.pmax_next + nseg;
  a.b = b;
  a.x = x;
  a.dinv = h.dinv;
  a.m = h.mask;
  double *w = h.work;
  const size_t N = h.N;
  a.r = w;
  a.rh = w + N;
  a.p = w + 2 * N;
  a.v = w + 3 * N;
  a.ph = w + 4 * N;
  a.sv = w + 5 * N;
  a.sh = w + 6 * N;
  a.t = w + 7 * N;
  if (h.seg_rows) {
    a.rows.S = h.st_S;
    a.rows.nm = h.st_nm + NM_LEAD;
    a.rows.N = h.N;
    a.mesh = h.seg_mesh;
    a.php = h.seg_x;
    a.shp = h.seg_x + h.seg_pairs;
    a.w = a.ph;
  }
  L.ntiles = nt;
  L.threads = threads;
  return cudaSuccess;
}
}  // namespace

int solve_segmented_device(Handle &h, const double *b, double *x, double tol, int itmax,
                           int *iters, double *errs, int *statuses) {
  const int nseg = (int)h.seg_off.size() - 1;
  if (nseg < 1) {
    set_error("segmented solve: no segments (vdr_set_segments)");
    return VDR_BAD_ARGUMENT;
  }
  cudaError_t e = ensure_solver_workspace(h, 8);
  if (!e) e = ensure_segment_rows(h);
  if (e) return cuda_fail(e, "solver workspace");
  const bool rows = h.seg_rows;
  cudaStream_t s = h.stream;
  if (!h.seg_ticket || h.seg_ticket_n < nseg) {
    if (h.seg_ticket) cudaFree(h.seg_ticket);
    h.seg_ticket = nullptr;
    if ((e = cudaMalloc(&h.seg_ticket, sizeof(unsigned) * nseg))) return cuda_fail(e, "alloc");
    if ((e = cudaMemset(h.seg_ticket, 0, sizeof(unsigned) * nseg))) return cuda_fail(e, "memset");
    h.seg_ticket_n = nseg;
  }
  SegLayout L;
  // ---- autotune the tile shape once per segment layout ----
  if (h.seg_tile == 0 && rows) {
    // Four rows a thread while that leaves four blocks per SM, else two: the
    // block's sum and its ticket cost as much as a row (96 cubes, 1.18 M
    // nodes: tiles of 256 / 512 / 1024 / 4096 rows 189 / 149 / 130 / 145 us
    // per iteration; what the two-vector probe below takes, 2048 rows on 128
    // threads, 170 us).
    h.seg_tile = (h.N >> 10) >= 4 * device_sm_count() ? 1024 : 512;
    h.seg_threads = 256;
  }
  if (h.seg_tile == 0) {
    const int tiles_c[] = {512, 1024, 2048, 4096};
    const int threads_c[] = {128, 256, 512};
    float best = 1e30f;
    int bt = 1024, bth = 256;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int tile : tiles_c)
      for (int th : threads_c) {
        if (th > tile) continue;
        if ((e = seg_layout(h, tile, th, b, h.work, L))) return cuda_fail(e, "layout");
        for (int rep = 0; rep < 2; rep++) sg_probe<<<L.ntiles, th, 0, s>>>(L.a);
        cudaEventRecord(e0, s);
        for (int rep = 0; rep < 5; rep++) sg_probe<<<L.ntiles, th, 0, s>>>(L.a);
        cudaEventRecord(e1, s);
        count_launches(7);
        if ((e = cudaEventSynchronize(e1))) return cuda_fail(e, "autotune");
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best) {
          best = ms;
          bt = tile;
          bth = th;
        }
      }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    h.seg_tile = bt;
    h.seg_threads = bth;
    if (h.seg_graph) cudaGraphExecDestroy(h.seg_graph);
    h.seg_graph = nullptr;
  }
  if ((e = seg_layout(h, h.seg_tile, h.seg_threads, b, x, L))) return cuda_fail(e, "layout");
  const int nt = L.ntiles, th = L.threads;
  SegVec &a = L.a;
  a.s.tol = tol;
  a.s.itmax = itmax;
  const long long launches0 = launches_so_far();
  // initial state: all segments active, done = 0
  std::vector<int> ones(nseg, 1);
  int ctl[2] = {nseg, 0};
  if ((e = cudaMemcpyAsync(a.s.active, ones.data(), sizeof(int) * nseg,
                           cudaMemcpyHostToDevice, s)) ||
      (e = cudaMemcpyAsync(a.s.nactive, ctl, sizeof(int) * 2, cudaMemcpyHostToDevice, s)) ||
      (e = launch_mask_vec(x, h.mask, h.N, s)) ||
      (e = cudaMemsetAsync(a.r, 0, sizeof(double) * h.N, s)) ||
      (e = launch_apply(h, false, x, a.r, nullptr, nullptr, s)))
    return cuda_fail(e, "segmented start");
  sg_start<<<nt, th, 0, s>>>(a);
  sg_zero<<<nt, th, 0, s>>>(a);
  count_launches(2);
  const bool keep = stencil_keep(h);
  if (rows) {
    if ((e = cudaMemsetAsync(a.s.pexp, 0, sizeof(int) * 4 * nseg, s)))
      return cuda_fail(e, "segmented start");
    sgr_exponents<<<nt, th, 0, s>>>(a);
    sgr_first<<<nt, th, 0, s>>>(a);
    sgr_w<<<nt, th, 0, s>>>(a);
    count_launches(3);
  }
  if ((e = cudaGetLastError())) return cuda_fail(e, "segmented start");

  // the applies skip the elements of frozen meshes
  struct GateScope {
    Handle &h;
    GateScope(Handle &hh, const int *active) : h(hh) {
      h.gate_eseg = h.seg_of_elem;
      h.gate_active = active;
    }
    ~GateScope() {
      h.gate_eseg = nullptr;
      h.gate_active = nullptr;
    }
  } gate(h, a.s.active);
  const int K = h.opt.iters_per_graph > 0 ? h.opt.iters_per_graph : 8;
  uintptr_t tol_bits;  // the captured kernels carry the tolerance and itmax
  std::memcpy(&tol_bits, &tol, sizeof tol_bits);
  const GraphKey key{key_of(b), key_of(x), key_of(h.work), (uintptr_t)K, (uintptr_t)h.seg_tile,
                     (uintptr_t)th, (uintptr_t)rows, tol_bits, (uintptr_t)itmax};
  if (!h.seg_graph || h.seg_key != key) {
    if (h.seg_graph) cudaGraphExecDestroy(h.seg_graph);
    h.seg_graph = nullptr;
    cudaGraph_t graph;
    if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)))
      return cuda_fail(e, "begin capture");
    const OwnCapture own(h);
    const long long before = launches_so_far();
    for (int k = 0; k < K && !e; k++) {
      if (rows) {
        if (keep) sgr_v<true><<<nt, th, 0, s>>>(a);
        else sgr_v<false><<<nt, th, 0, s>>>(a);
        if (keep) sgr_t<true><<<nt, th, 0, s>>>(a);
        else sgr_t<false><<<nt, th, 0, s>>>(a);
        sgr_p<<<nt, th, 0, s>>>(a);
        count_launches(3);
        e = cudaGetLastError();
        continue;
      }
      sg_p<<<nt, th, 0, s>>>(a);
      e = launch_apply(h, false, a.ph, a.v, a.s.done, nullptr, s);
      if (e) break;
      sg_alpha<<<nt, th, 0, s>>>(a);
      sg_s<<<nt, th, 0, s>>>(a);
      e = launch_apply(h, false, a.sh, a.t, a.s.done, nullptr, s);
      if (e) break;
      sg_omega<<<nt, th, 0, s>>>(a);
      sg_xr<<<nt, th, 0, s>>>(a);
      count_launches(5);
      e = cudaGetLastError();
    }
    h.seg_graph_launches = (long)(launches_so_far() - before);
    count_launches(before - launches_so_far());
    const cudaError_t e2 = cudaStreamEndCapture(s, &graph);
    if (e) return cuda_fail(e, "segmented capture");
    if (e2) return cuda_fail(e2, "end capture");
    e = cudaGraphInstantiate(&h.seg_graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e) return cuda_fail(e, "graph instantiate");
    h.seg_key = key;
  }
  const int max_launches = (itmax + K - 1) / K + 1;
  int *h_done = reinterpret_cast<int *>(h.h_st);  // pinned scratch
  int launched = 0;
  for (int c = 0; c < max_launches; c++) {
    if ((e = cudaGraphLaunch(h.seg_graph, s))) return cuda_fail(e, "graph launch");
    count_launches(h.seg_graph_launches);
    launched++;
    if ((e = cudaMemcpyAsync(h_done, a.s.done, sizeof(int), cudaMemcpyDeviceToHost, s)) ||
        (e = cudaStreamSynchronize(s)))
      return cuda_fail(e, "state readback");
    if (*h_done) break;
  }
  if ((e = cudaStreamSynchronize(s))) return cuda_fail(e, "segmented solve");
  std::vector<int> st(nseg), it(nseg);
  std::vector<double> er(nseg);
  if ((e = cudaMemcpy(st.data(), a.s.status, sizeof(int) * nseg, cudaMemcpyDeviceToHost)) ||
      (e = cudaMemcpy(it.data(), a.s.iter, sizeof(int) * nseg, cudaMemcpyDeviceToHost)) ||
      (e = cudaMemcpy(er.data(), a.s.err, sizeof(double) * nseg, cudaMemcpyDeviceToHost)))
    return cuda_fail(e, "segment results");
  int status = VDR_OK, maxit = 0;
  for (int k = 0; k < nseg; k++) {
    if (st[k] == VDR_BREAKDOWN) status = VDR_BREAKDOWN;
    else if (st[k] != VDR_OK && status == VDR_OK) status = VDR_NOT_CONVERGED;
    maxit = std::max(maxit, it[k]);
  }
  if (iters) std::copy(it.begin(), it.end(), iters);
  if (errs) std::copy(er.begin(), er.end(), errs);
  if (statuses) std::copy(st.begin(), st.end(), statuses);
  h.last = vdr_solve_stats{};
  h.last.iterations = maxit;
  h.last.status = status;
  h.last.graph_launches = launched;
  h.last.kernel_launches = (int)(launches_so_far() - launches0);
  return status;
}

}  // namespace vdr
