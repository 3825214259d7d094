// resident.cu -- a whole BiCGStab solve in one launch, for meshes whose rows
// and vectors fit on the chip (one node per thread, at most 1024 per SM).
//
// At these sizes an iteration moves little data: what it costs is launches,
// FP64 sums on a pipe that takes 16 cycles per warp instruction, and waits
// (31 us per iteration at 2,800 nodes with four launches, of which the
// products are 2 us).  Here a node's vector entries stay in its thread's
// registers for the whole solve and only p^ and s^ (a pair each) are handed
// to the neighbours.  The CTAs meet three times per iteration:
//
//   v = A p^, s = r - alpha v, s^ out             | (s,s), (rh,s)
//   t = A s^                                       | (t,s), (t,t), (rh,t)
//   x, r, p, p^ out                                | (r,r), (w,p^)
//
// with w = A^T rh formed once, so that alpha = rho / (w, p^) is known before
// the product that it scales, and the next rho is (rh,s) - omega (rh,t).
// Sums: per warp by a transposing butterfly (5-6 FP64 adds for up to four
// quantities), then one warp per CTA adds all partials in the same order, so
// all CTAs hold bit-identical scalars and take the same exit.  Divisions run
// on that warp only (on every warp they took longer than the products).
//
// CLUSTER: up to 16 CTAs of at most 192 nodes in one cluster; p^, s^ and the
// partials lie in shared memory and are read across the cluster, the
// meetings are cluster barriers.  IN_REGS, IN_SMEM: a cooperative grid, one
// CTA per SM, p^ and s^ through L2, meetings at a counter (bounded waits:
// VDR_TIMEOUT); a node's 27 pairs stay in registers up to 512
// threads, in shared memory (216 bytes a thread) above.  Per iteration,
// cluster / grid: 8.1 us at 448 nodes, 9.6 / 12 at 1,170, 11 / 12.5 at 2,800,
// 19.5 / 12.8 at 7,000 (reads across a cluster are slow in number), then 14.1
// at 18,500, 20 at 75,000, 24 at 100,000, 29 at 148,000; four kernels per
// iteration: 31 at 2,800, 53 at 100,000.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "meet.cuh"
#include "stencil.cuh"

namespace vdr {
namespace {

// (Not above 128 bytes: the compiler leaves a larger argument in constant
// memory and resident_bicgstab forms its neighbours' addresses anew in every
// product, 5 per cent of an iteration.  resident_bicg has no registers to hold
// them in, and is asked to leave them there: 48 to 104 bytes of spills less
// and 2 to 5 per cent of a solve.)
struct ResArgs {
  StencilView w;
  const double *b, *dinv;
  const unsigned char *m;
  double *x;
  float2 *php, *shp;  // the grid's p^ and s^
  KState *st;
  MeetArgs mt;
  double tol;
  int itmax, window;
};
static_assert(sizeof(ResArgs) <= 128, "in registers");

__device__ __forceinline__ double row_value(const DfAcc &acc, int shift) {
  double o = df_to_double(acc.s, acc.c);
  if (!df_scale(o, shift)) o = ldexp(o, shift);
  return o;
}

__device__ __forceinline__ float2 masked_pair(bool msk, double d, int shift) {
  return msk ? make_float2(0.f, 0.f) : stencil_pair(d, shift);
}

template <int MODE, int T>
__global__ void __launch_bounds__(T, 1) resident_bicgstab(ResArgs a) {
  extern __shared__ float2 dyn[];  // CLUSTER: p^ and s^, [2][T]; IN_SMEM: rows, [27][T]
  __shared__ ResShared sh;
  const int N = a.w.N, n = (int)(blockIdx.x * T + threadIdx.x);
  const bool on = n < N;
  unsigned target = 0;
  const int base = 1023 - pair_head(a.w.nm);
  const int none[1] = {0};
  const auto nothing = [](int) {};
  double x = 0.0, r = 0.0, p = 0.0, v = 0.0, s = 0.0, t = 0.0, rh = 0.0, wn = 0.0;
  const double di = on ? a.dinv[n] : 0.0;
  const bool msk = on ? a.m[n] != 0 : true;

  // the node's row, and in a cluster where its neighbours' entries lie (its
  // own where there is none: the row holds a zero)
  float2 A[MODE == IN_SMEM ? 1 : 27];
  unsigned nb[MODE == CLUSTER ? 27 : 1];
#pragma unroll
  for (int k = 0; k < 27; k++) {
    const float2 e = on ? __ldcg(a.w.S + (size_t)k * N + n) : make_float2(0.f, 0.f);
    if (MODE == IN_SMEM) dyn[k * T + threadIdx.x] = e;
    else A[MODE == IN_SMEM ? 0 : k] = e;
    if (MODE == CLUSTER) {
      const int q = n + stencil_off(k, a.w.nax, a.w.pl);
      const int u = q >= 0 && q < (int)gridDim.x * T ? q : n;
      nb[MODE == CLUSTER ? k : 0] = cluster_addr(dyn + u % T, u / T);
    }
  }
  if (MODE == CLUSTER) {
    dyn[threadIdx.x] = dyn[T + threadIdx.x] = make_float2(0.f, 0.f);
    cluster_meet();  // every CTA runs before its memory is read
  }
  // the entries handed out: which = 0 p^, 1 s^
  const auto put = [&](int which, float2 e) {
    if (MODE == CLUSTER) dyn[which * T + threadIdx.x] = e;
    else if (on) (which ? a.shp : a.php)[n] = e;
  };
  const auto get = [&](int which, int k) {
    if (MODE == CLUSTER)
      return cluster_pair(nb[MODE == CLUSTER ? k : 0] + (unsigned)(which * T * sizeof(float2)));
    return (which ? a.shp : a.php)[(on ? n : 0) + stencil_off(k, a.w.nax, a.w.pl)];
  };
  const auto row = [&](int which, int shift) {
    DfAcc acc{0.f, 0.f};
    constexpr int G = MODE == IN_SMEM ? 9 : 27;  // entries in flight
#pragma unroll
    for (int z = 0; z < 27; z += G) {
      float2 xv[G];
#pragma unroll
      for (int c = 0; c < G; c++) xv[c] = get(which, z + c);
#pragma unroll
      for (int c = 0; c < G; c++) {
        const float2 e = MODE == IN_SMEM ? dyn[(z + c) * T + threadIdx.x]
                                         : A[MODE == IN_SMEM ? 0 : z + c];
        df_fma_acc(acc, e.x, e.y, xv[c].x, xv[c].y);
      }
    }
    return row_value(acc, shift);
  };

  // x masked in place; r = b - A x (A x skipped when x is zero)
  {
    x = msk ? 0.0 : a.x[n];
    const double z[1] = {0.0};
    const int e1[1] = {df_exp(x)};
    if (!meet<MODE, T, 1, 1, 0, AT_C, AT_C, 2>(sh, a.mt, z, e1, target, nothing))
      return;
  }
  const int ex = sh.etot[0];
  if (ex) {
    put(0, masked_pair(msk, x, ex - base));
    const double z[1] = {0.0};
    if (!meet<MODE, T, 1, 0, 0, AT_D, AT_D, 0>(sh, a.mt, z, none, target, nothing))
      return;
    v = row(0, ex - base);
  }
  {
    const double bi = msk ? 0.0 : a.b[n];
    r = bi - (msk ? 0.0 : v);
    rh = p = r;
    const double q[2] = {bi * bi, r * r};
    const int em[2] = {df_exp(r), df_exp(msk ? 0.0 : r * di)};
    if (!meet<MODE, T, 2, 2, 2, AT_A, AT_A, 0>(sh, a.mt, q, em, target, nothing))
      return;
  }
  const double bnrm2 = sh.tot[0];
  double rho = sh.tot[1], rr2 = rho;
  // ||r|| <= tol ||b|| as squares; a NaN or overflowed sum is told apart first
  const double thr = a.tol * a.tol * bnrm2;
  const int er = sh.etot[0];
  int pexp = sh.etot[1];
  int iter = 0, status = VDR_NOT_CONVERGED, reason = 0, since = 0;
  double best2 = INFINITY;
  bool done = false;
  if (bnrm2 == 0.0) {  // b = 0: the solution is x = 0
    x = 0.0;
    status = VDR_OK;
    rr2 = 0.0;
    done = true;
  } else if (!isfinite(bnrm2) || !isfinite(rr2)) {
    status = VDR_BREAKDOWN;
    reason = 5;
    done = true;
  } else if (rr2 <= thr) {
    status = VDR_OK;
    done = true;
  } else if (a.itmax <= 0) {
    done = true;
  }
  double al = 0.0, iwp = 0.0;
  // alpha = rho / (w, p^) and 1 / (w, p^), on two lanes of one division
  const auto alpha_of = [&](int lane, double wp) {
    const double d = (lane ? 1.0 : rho) / wp;
    if (lane < 2) sh.tot[2 + lane] = d;
  };
  if (!done) {
    // p^ = D^-1 r, and w = A^T rh (the neighbours' rows, from L2)
    put(0, masked_pair(msk, p * di, pexp - base));
    put(1, masked_pair(msk, rh, er - base));
    double q[1] = {0.0};
    if (!meet<MODE, T, 1, 0, 0, AT_C, AT_C, 0>(sh, a.mt, q, none, target, nothing))
      return;
    DfAcc acc{0.f, 0.f};
    for (int z = 0; z < 27; z += 9)
#pragma unroll
      for (int c = 0; c < 9; c++) {
        const int k = z + c, o = n + stencil_off(k, a.w.nax, a.w.pl);
        if (!on || o < 0 || o >= N) continue;
        const float2 e = __ldcg(a.w.S + (size_t)(26 - k) * N + o);
        float2 xv;
        if (MODE == CLUSTER)
          xv = cluster_pair(cluster_addr(dyn + T + o % T, o / T));
        else
          xv = __ldcg(a.shp + o);
        df_fma_acc(acc, e.x, e.y, xv.x, xv.y);
      }
    wn = row_value(acc, er - base);
    if (!msk) q[0] = wn * (p * di);
    if (!meet<MODE, T, 1, 0, 1, AT_D, AT_D, 0>(sh, a.mt, q, none, target,
                                            [&](int lane) { alpha_of(lane, sh.tot[0]); }))
      return;
    if (sh.tot[0] == 0.0 || !isfinite(sh.tot[0])) {
      status = VDR_BREAKDOWN;
      reason = 2;
      done = true;
    }
    al = sh.tot[2];
    iwp = sh.tot[3];
  }
  int pmax = pexp;
  while (!done) {
    const int shift = pexp - base;
    v = row(0, shift);
    s = r - al * v;
    put(1, masked_pair(msk, s * di, shift));
    {
      const double q[2] = {s * s, rh * s};
      if (!meet<MODE, T, 2, 0, 0, AT_C, AT_C, 0>(sh, a.mt, q, none, target, nothing))
        return;
    }
    t = row(1, shift);
    // omega = ts / tt and beta = (rho' / rho) (alpha / omega) = (rhs tt / ts -
    // rht) / (w, p^), rho' = rhs - omega rht: ts / tt and tt / ts on two
    // lanes of one division.
    {
      const double q[3] = {t * s, t * t, rh * t};
      if (!meet<MODE, T, 3, 0, 5, AT_D, AT_C, 0>(sh, a.mt, q, none, target, [&](int lane) {
            const double ts = sh.tot[2], tt = sh.tot[3], rhs = sh.tot[1], rht = sh.tot[4];
            const double num = lane ? tt : ts, den = lane ? ts : tt, d = num / den;
            const double e = lane ? (rhs * d - rht) * iwp : rhs - d * rht;
            __syncwarp();
            if (lane == 0) {
              sh.tot[1] = d;
              sh.tot[4] = e;
            } else if (lane == 1) {
              sh.tot[5] = e;
            }
          }))
        return;
    }
    const double ss = sh.tot[0], om = sh.tot[1], ts = sh.tot[2], tt = sh.tot[3],
                 rho1 = sh.tot[4], beta = sh.tot[5];
    if (ss <= thr) {  // s met the tolerance: x += alpha p^
      if (!msk) x += di * (al * p);
      iter++;
      rr2 = ss;
      status = VDR_OK;
      break;
    }
    if (tt == 0.0 || !isfinite(tt) || !isfinite(ts)) {
      status = VDR_BREAKDOWN;
      reason = 3;
      break;
    }
    if (!msk) x += di * (al * p + om * s);
    r = s - om * t;
    p = r + beta * (p - om * v);
    const double ph = msk ? 0.0 : p * di;
    put(0, stencil_pair(ph, pmax - base));
    rho = rho1;
    {
      const double q[2] = {r * r, wn * ph};
      const int em[1] = {df_exp(ph)};
      if (!meet<MODE, T, 2, 1, 2, AT_A, AT_A, 0>(sh, a.mt, q, em, target,
                                              [&](int lane) { alpha_of(lane, sh.tot[1]); }))
        return;
    }
    pexp = pmax;
    pmax = sh.etot[0];
    rr2 = sh.tot[0];
    const double wp = sh.tot[1];
    al = sh.tot[2];
    iwp = sh.tot[3];
    iter++;
    if (!(rr2 == rr2) || !isfinite(rho1)) {
      status = VDR_BREAKDOWN;
      reason = 5;
      done = true;
    } else if (rr2 <= thr) {
      status = VDR_OK;
      done = true;
    } else if (rho1 == 0.0 || om == 0.0) {
      status = VDR_BREAKDOWN;
      reason = rho1 == 0.0 ? 1 : 4;
      done = true;
    } else if (iter >= a.itmax) {
      done = true;
    } else if (a.window > 0) {
      if (rr2 < 0.9801 * best2) {  // a 1 % drop of the norm
        best2 = rr2;
        since = 0;
      } else if (++since >= a.window) {
        reason = 6;  // stalled
        done = true;
      }
    }
    if (!done && (wp == 0.0 || !isfinite(wp))) {
      status = VDR_BREAKDOWN;
      reason = 2;
      done = true;
    }
  }
  if (on) a.x[n] = x;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    KState *st = a.st;
    st->iter = iter;
    st->err = bnrm2 > 0.0 ? sqrt(rr2) / sqrt(bnrm2) : 0.0;
    st->status = status;
    st->reason = reason;
    st->done = 1;
  }
  if (MODE == CLUSTER) cluster_meet();  // no CTA leaves while its memory is read
}

// Jacobi BiCG in the same form (a cooperative grid): p and p~ handed out, A p
// from the node's row and A^T p~ from its column (in shared memory up to 512
// threads, from L2 above), then (A p, p~), then (r,r) and (D^-1 r, r~).  b is
// taken as it is (the drop-in's may be nonzero on Dirichlet rows, where x
// stays zero).
template <int MODE, int T>
__global__ void __launch_bounds__(T, 1) resident_bicg(const __grid_constant__ ResArgs a) {
  extern __shared__ float2 dyn[];  // [27][T]: columns, or rows (IN_SMEM)
  __shared__ ResShared sh;
  const int N = a.w.N, n = (int)(blockIdx.x * T + threadIdx.x);
  const bool on = n < N;
  unsigned target = 0;
  const int base = 1023 - pair_head(a.w.nm);
  const int none[1] = {0};
  const auto nothing = [](int) {};
  const auto column = [&](int k) {  // A's entry of neighbour k with this node
    const int q = n + stencil_off(k, a.w.nax, a.w.pl);
    return on && q >= 0 && q < N ? __ldcg(a.w.S + (size_t)(26 - k) * N + q)
                                 : make_float2(0.f, 0.f);
  };
  float2 A[MODE == IN_REGS ? 27 : 1];
#pragma unroll
  for (int k = 0; k < 27; k++) {
    const float2 e = on ? __ldcg(a.w.S + (size_t)k * N + n) : make_float2(0.f, 0.f);
    if (MODE == IN_REGS) A[MODE == IN_REGS ? k : 0] = e;
    dyn[k * T + threadIdx.x] = MODE == IN_REGS ? column(k) : e;
  }
  const double di = on ? a.dinv[n] : 0.0;
  const bool msk = on ? a.m[n] != 0 : true;
  double x = 0.0, r, rr, p = 0.0, pp = 0.0, z = 0.0, zz = 0.0;
  const float2 *gp = a.php + (on ? n : 0), *gs = a.shp + (on ? n : 0);
  const auto row = [&](int shift) {
    DfAcc acc{0.f, 0.f};
#pragma unroll
    for (int g = 0; g < 27; g += 9) {
      float2 xv[9];
#pragma unroll
      for (int c = 0; c < 9; c++) xv[c] = gp[stencil_off(g + c, a.w.nax, a.w.pl)];
#pragma unroll
      for (int c = 0; c < 9; c++) {
        const float2 e = MODE == IN_REGS ? A[MODE == IN_REGS ? g + c : 0]
                                         : dyn[(g + c) * T + threadIdx.x];
        df_fma_acc(acc, e.x, e.y, xv[c].x, xv[c].y);
      }
    }
    return row_value(acc, shift);
  };
  const auto trans = [&](int shift) {
    DfAcc acc{0.f, 0.f};
#pragma unroll
    for (int g = 0; g < 27; g += 9) {
      float2 xv[9], e[9];
#pragma unroll
      for (int c = 0; c < 9; c++) {
        xv[c] = gs[stencil_off(g + c, a.w.nax, a.w.pl)];
        e[c] = MODE == IN_REGS ? dyn[(g + c) * T + threadIdx.x] : column(g + c);
      }
#pragma unroll
      for (int c = 0; c < 9; c++) df_fma_acc(acc, e[c].x, e[c].y, xv[c].x, xv[c].y);
    }
    return row_value(acc, shift);
  };

  {
    x = msk ? 0.0 : a.x[n];
    const double q[1] = {0.0};
    const int e1[1] = {df_exp(x)};
    if (!meet<MODE, T, 1, 1, 0, AT_C, AT_C, 2>(sh, a.mt, q, e1, target, nothing))
      return;
  }
  const int ex = sh.etot[0];
  if (ex) {
    if (on) a.php[n] = masked_pair(msk, x, ex - base);
    const double q[1] = {0.0};
    if (!meet<MODE, T, 1, 0, 0, AT_D, AT_D, 0>(sh, a.mt, q, none, target, nothing))
      return;
    z = row(ex - base);
  }
  {
    const double bi = on ? a.b[n] : 0.0;
    r = bi - (msk ? 0.0 : z);
    rr = r;
    const double q[3] = {bi * bi, r * r, (r * di) * rr};
    const int e1[1] = {df_exp(msk ? 0.0 : r * di)};
    if (!meet<MODE, T, 3, 1, 3, AT_A - 1, AT_A - 1, 0>(sh, a.mt, q, e1, target, nothing))
      return;
  }
  const double bnrm2 = sh.tot[0], thr = a.tol * a.tol * bnrm2;
  double rr2 = sh.tot[1], bknum = sh.tot[2], bk = 0.0;
  int pexp = sh.etot[0], qexp = pexp;
  int iter = 0, status = VDR_NOT_CONVERGED, reason = 0;
  bool done = false;
  if (bnrm2 == 0.0) {  // b = 0: the solution is x = 0
    x = 0.0;
    rr2 = 0.0;
    status = VDR_OK;
    done = true;
  } else if (!isfinite(bnrm2) || !isfinite(rr2)) {
    status = VDR_BREAKDOWN;
    reason = 5;
    done = true;
  } else if (rr2 <= thr) {
    status = VDR_OK;
    done = true;
  } else if (a.itmax <= 0) {
    done = true;
  }
  while (!done) {
    p = msk ? 0.0 : r * di + bk * p;
    pp = msk ? 0.0 : rr * di + bk * pp;
    if (on) {
      a.php[n] = stencil_pair(p, pexp - base);
      a.shp[n] = stencil_pair(pp, qexp - base);
    }
    {
      const double q[1] = {0.0};
      if (!meet<MODE, T, 1, 0, 0, AT_C, AT_C, 0>(sh, a.mt, q, none, target, nothing))
        return;
    }
    z = row(pexp - base);
    zz = trans(qexp - base);
    {
      const double q[1] = {z * pp};
      const int em[2] = {df_exp(p), df_exp(pp)};
      if (!meet<MODE, T, 1, 2, 1, AT_C, AT_C, 0>(sh, a.mt, q, em, target, [&](int lane) {
            const double d = bknum / sh.tot[0];
            if (lane == 0) sh.tot[1] = d;
          }))
        return;
    }
    const double ak = sh.tot[1];
    pexp = sh.etot[0];
    qexp = sh.etot[1];
    if (!isfinite(ak)) {
      status = VDR_BREAKDOWN;
      reason = 2;
      break;
    }
    x += ak * p;
    r -= ak * z;
    rr -= ak * zz;
    {
      const double q[2] = {r * r, (r * di) * rr};
      if (!meet<MODE, T, 2, 0, 2, AT_D, AT_D, 0>(sh, a.mt, q, none, target, [&](int lane) {
            const double d = sh.tot[1] / bknum;
            if (lane == 0) sh.tot[2] = d;
          }))
        return;
    }
    rr2 = sh.tot[0];
    bknum = sh.tot[1];
    bk = sh.tot[2];
    iter++;
    if (!(rr2 == rr2)) {
      status = VDR_BREAKDOWN;
      reason = 5;
      done = true;
    } else if (rr2 <= thr) {
      status = VDR_OK;
      done = true;
    } else if (iter >= a.itmax) {
      done = true;
    }
  }
  if (on) a.x[n] = x;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    KState *st = a.st;
    st->iter = iter;
    st->err = bnrm2 > 0.0 ? sqrt(rr2) / sqrt(bnrm2) : 0.0;
    st->status = status;
    st->reason = reason;
    st->done = 1;
  }
}

// A meeting that one CTA of three never comes to, with a short limit; CTA 2
// stores a solve's end all the same.
__global__ void __launch_bounds__(32, 1) absent_kernel(MeetArgs mt, KState *st) {
  __shared__ ResShared sh;
  if (blockIdx.x == 1) return;
  unsigned target = 0;
  const double q[1] = {0.0};
  const int none[1] = {0};
  const bool met =
      meet<IN_REGS, 32, 1, 0, 0, AT_C, AT_C, 0>(sh, mt, q, none, target, [](int) {});
  if (blockIdx.x == 2 && threadIdx.x == 0) {
    st->status = met ? VDR_BREAKDOWN : VDR_OK;
    st->done = 1;
  }
}

// One launch of `grid` CTAs: one cluster, or a cooperative grid.
template <int MODE, int T, bool BICG = false>
cudaError_t launch_one(int grid, const ResArgs &a, cudaStream_t s) {
  void (*kern)(ResArgs);
  if constexpr (BICG) kern = resident_bicg<MODE, T>;
  else kern = resident_bicgstab<MODE, T>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(T);
  cfg.stream = s;
  cudaError_t e;
  cudaLaunchAttribute attr[1];
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (MODE == CLUSTER) {
    cfg.dynamicSmemBytes = sizeof(float2) * 2 * T;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)grid;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    if (grid > 8 &&
        (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
      return e;
  } else {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    if (MODE == IN_SMEM || BICG) {
      cfg.dynamicSmemBytes = sizeof(float2) * 27 * T;
      if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)cfg.dynamicSmemBytes)))
        return e;
    }
  }
  return cudaLaunchKernelEx(&cfg, kern, a);
}

// The smallest power of two of CTAs of T threads that holds N nodes.
int cluster_ctas(int N, int T) {
  int c = 1;
  while ((long)c * T < N) c *= 2;
  return c;
}

}  // namespace

// VDR_TIMEOUT when the meeting's waits ran out of their (about 1 ms) limit and
// that, not the status stored after them, is what a solve would return.
int diag_meeting_timeout(Handle &h) {
  cudaError_t e = ensure_solver_workspace(h, 8);
  cudaStream_t s = h.stream;
  if (e || (e = cudaMemsetAsync(h.st, 0, sizeof(KState), s))) return cuda_fail(e, "diag");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(3);
  cfg.blockDim = dim3(32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MeetArgs mt = meet_args(h);
  mt.limit = 2000000LL;
  if ((e = cudaLaunchKernelEx(&cfg, absent_kernel, mt, h.st))) return cuda_fail(e, "diag launch");
  count_launches(1);
  KState fin;
  if ((e = cudaMemcpyAsync(&fin, h.st, sizeof(KState), cudaMemcpyDeviceToHost, s)) ||
      (e = cudaStreamSynchronize(s)))
    return cuda_fail(e, "diag");
  if (fin.done && fin.status == VDR_OK && outcome(fin) == VDR_TIMEOUT) {
    set_error("diag: the meeting's wait ran out (as intended)");
    return VDR_TIMEOUT;
  }
  set_error("diag: the meeting did not report its timeout");
  return VDR_CUDA_ERROR;
}

long whole_solve_nodes() { return 1024L * std::min(device_sm_count(), 32 * RES_NB); }

bool resident_size(const Handle &h) { return h.resident && h.N <= whole_solve_nodes(); }

cudaError_t launch_resident(Handle &h, int method, const double *b, double *x, double tol,
                            int itmax, int stall_window) {
  cudaError_t e;
  if ((e = meet_reset(h, h.stream))) return e;
  ResArgs a{};
  a.w = stencil_view(h);
  a.b = b;
  a.dinv = h.dinv;
  a.m = h.mask;
  a.x = x;
  a.php = h.st_x + stencil_pad(h);
  a.shp = a.php + h.N + 2 * stencil_pad(h);
  a.st = h.st;
  a.mt = meet_args(h);
  a.tol = tol;
  a.itmax = itmax;
  a.window = stall_window;
  const int N = h.N, sms = std::min(device_sm_count(), 32 * RES_NB);
  const auto blocks = [&](int T) { return (N + T - 1) / T; };
  // the fewest threads per CTA that hold a node each: with few warps per SM
  // the FP64 pipe and the sums are the shortest
  cudaStream_t s = h.stream;
  e = cudaErrorNotSupported;
  if (method == VDR_SOLVER_BICG) {
    if (blocks(128) <= sms) e = launch_one<IN_REGS, 128, true>(blocks(128), a, s);
    else if (blocks(256) <= sms) e = launch_one<IN_REGS, 256, true>(blocks(256), a, s);
    else if (blocks(512) <= sms) e = launch_one<IN_REGS, 512, true>(blocks(512), a, s);
    else e = launch_one<IN_SMEM, 1024, true>(blocks(1024), a, s);
    if (!e) count_launches(1);
    return e;
  }
  if (h.resident_cluster && N <= 192 * CLUSTER_MAX) {
    if (N <= 64 * CLUSTER_MAX) e = launch_one<CLUSTER, 64>(cluster_ctas(N, 64), a, s);
    else if (N <= 128 * CLUSTER_MAX) e = launch_one<CLUSTER, 128>(CLUSTER_MAX, a, s);
    else e = launch_one<CLUSTER, 192>(CLUSTER_MAX, a, s);
    if (e) {  // no cluster of this size here: the grid
      cudaGetLastError();
      h.resident_cluster = false;
    }
  }
  if (e) {
    if (blocks(128) <= sms) e = launch_one<IN_REGS, 128>(blocks(128), a, s);
    else if (blocks(256) <= sms) e = launch_one<IN_REGS, 256>(blocks(256), a, s);
    else if (blocks(512) <= sms) e = launch_one<IN_REGS, 512>(blocks(512), a, s);
    else if (blocks(768) <= sms) e = launch_one<IN_SMEM, 768>(blocks(768), a, s);
    else e = launch_one<IN_SMEM, 1024>(blocks(1024), a, s);
  }
  if (!e) count_launches(1);
  return e;
}

}  // namespace vdr
