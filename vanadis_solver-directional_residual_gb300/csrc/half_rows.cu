// half_rows.cu -- the mixed solve's inner operator on assembled rows.
//
// A^ = P A P D^-1 (as in half.cu) with the 27-point rows of stencil.cuh in
// binary16, one power-of-two scale per row (largest entry in [2^14, 2^15)):
// 55 bytes a node where the element-wise store reads 129 an element, and the
// product is a gather, so the inner BiCGStab takes the FP64 one's form
// (krylov.cu, resident.cu) on FP32 vectors: three meetings per iteration, no
// cleared vectors, no atomics.  Inner products are exact FP32 products
// summed in double-float per thread and in FP64 across threads.
//
// Layout: H[k Np + n] (half planes, Np = N rounded up to 8), e16[n].  A
// thread takes a pair of neighbouring nodes, so one 4-byte load brings both
// rows' entry k and the pair's rows share 18 of their 27 inputs; A^T reads the
// same planes shifted.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "meet.cuh"
#include "stencil.cuh"

namespace vdr {
namespace {

constexpr int HT = 256;  // threads of the kernels of the large form

struct HalfRows {
  const __half *H = nullptr;
  const signed char *e = nullptr;
  int N = 0, Np = 0, nax = 0, pl = 0;
};

__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((127 + e) << 23); }

// Rows from the FP32 heads of the assembled pairs, columns scaled by D^-1;
// bit 0 of *bad when a row's scale leaves [2^-126, 2^113].
__global__ void __launch_bounds__(256) half_rows_kernel(const StencilView v,
                                                        const double *__restrict__ dinv,
                                                        __half *H, signed char *e16, int Np,
                                                        int *bad) {
  for (long n = (long)blockIdx.x * blockDim.x + threadIdx.x; n < Np;
       n += (long)gridDim.x * blockDim.x) {
    const unsigned m = n < v.N ? v.nm[n] : 0u;
    float a[27], mx = 0.f;
#pragma unroll
    for (int k = 0; k < 27; k++) {
      const bool on = (m >> k) & 1u;
      a[k] = on ? __ldcs(v.S + (size_t)k * v.N + n).x *
                      (float)__ldg(dinv + n + stencil_off(k, v.nax, v.pl))
                : 0.f;
      mx = fmaxf(mx, fabsf(a[k]));
    }
    int e = 0;
    if (mx > 0.f) {
      if (!(mx < INFINITY)) {
        atomicOr(bad, 1);
      } else {
        e = ilogbf(mx) - 14;
        if (e < -126 || e > 113) atomicOr(bad, 1);
        e = max(-126, min(113, e));
      }
    }
    const float sc = exp2_int(-e);
#pragma unroll
    for (int k = 0; k < 27; k++) H[(size_t)k * Np + n] = __float2half_rn(a[k] * sc);
    e16[n] = (signed char)e;
  }
}

// Rows n0 and n0 + 1 (n0 even) times x; row(k) gives both rows' entry k.
template <typename F>
__device__ __forceinline__ void pair_rows(F row, long n0, const HalfRows &h, const float *xp,
                                          float &y0, float &y1) {
  y0 = y1 = 0.f;
#pragma unroll
  for (int z = 0; z < 3; z++) {
    float x[3][4];
#pragma unroll
    for (int y = 0; y < 3; y++) {
      const float *q = xp + (n0 + (z - 1) * (long)h.pl + (y - 1) * h.nax);
#pragma unroll
      for (int d = 0; d < 4; d++) x[y][d] = q[d - 1];
    }
#pragma unroll
    for (int y = 0; y < 3; y++)
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const float2 f = __half22float2(row(9 * z + 3 * y + d));
        y0 = fmaf(f.x, x[y][d], y0);
        y1 = fmaf(f.y, x[y][d + 1], y1);
      }
  }
}

// (A^T x)_n0 and (A^T x)_n0+1 (n0 even); xs holds x times its row's scale.
__device__ __forceinline__ void trans_pair(const HalfRows &h, long n0, const float *xs,
                                           float &y0, float &y1) {
  y0 = y1 = 0.f;
#pragma unroll
  for (int z = 0; z < 3; z++) {
    float x[3][4];
    __half a0[9], a1[9];
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const int k = 9 * z + c;
      // a place beyond the plane's ends lies in the next one (26 - k > 13 where
      // the offset is negative) and meets a zero of xs
      const __half *p =
          h.H + ((26 - k) * (long)h.Np + n0 + stencil_off(k, h.nax, h.pl));
      a0[c] = p[0];
      a1[c] = p[1];
    }
#pragma unroll
    for (int y = 0; y < 3; y++)
#pragma unroll
      for (int d = 0; d < 4; d++)
        x[y][d] = xs[n0 + (z - 1) * (long)h.pl + (y - 1) * h.nax + d - 1];
#pragma unroll
    for (int c = 0; c < 9; c++) {
      y0 = fmaf(__half2float(a0[c]), x[c / 3][c % 3], y0);
      y1 = fmaf(__half2float(a1[c]), x[c / 3][c % 3 + 1], y1);
    }
  }
}

struct VecH {
  HalfRows h;
  KState *st;
  double *partials;
  float *x, *r, *rh, *v, *t, *w;  // [Np]
  float *p, *s;                   // padded
};

// ---- the large form: three kernels per iteration ----
// Sums of Q values over the grid; true in thread 0 of the last block.
template <int Q>
__device__ __forceinline__ bool sums(const DfAcc (&d)[Q], const VecH &a, double (&out)[Q]) {
  __shared__ double sm[HT / 32][4];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int G = (int)gridDim.x;
  double v[Q];
#pragma unroll
  for (int q = 0; q < Q; q++) v[q] = dot_val(d[q]);
  const auto block = [&]() {  // totals in lanes 8 q of warp 0
    const double f = warp_sums<Q>(v, l);
    __syncthreads();
    if ((l & 7) == 0 && (l >> 3) < Q) sm[w][l >> 3] = f;
    __syncthreads();
    return w == 0 ? fold8((l >> 3) < Q ? sm[l & 7][l >> 3] : 0.0) : 0.0;
  };
  double c = block();
  if (w == 0) {
    if ((l & 7) == 0 && (l >> 3) < Q) a.partials[(l >> 3) * G + blockIdx.x] = c;
    __threadfence();
    __syncwarp();
    if (l == 0) last = atomicAdd(&a.st->ticket, 1u) == (unsigned)G - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < Q; q++) {
    v[q] = 0.0;
    for (int b = threadIdx.x; b < G; b += HT) v[q] += __ldcg(a.partials + q * G + b);
  }
  c = block();
  if (w == 0)
#pragma unroll
    for (int q = 0; q < Q; q++) out[q] = __shfl_sync(FULLR, c, 8 * q);
  if (threadIdx.x == 0) a.st->ticket = 0u;
  return threadIdx.x == 0;
}

__device__ __forceinline__ void set_alpha(KState *st, double wp) {
  if (wp == 0.0 || !isfinite(wp)) {
    st->status = VDR_BREAKDOWN;
    st->reason = 2;
    st->done = 1;
  } else {
    st->alpha = st->rho / wp;
  }
}

#define PAIRS_OF(a)                                                             \
  for (long n = 2 * ((long)blockIdx.x * blockDim.x + threadIdx.x); n < (a).h.N; \
       n += 2 * (long)gridDim.x * blockDim.x)
__device__ __forceinline__ float2 ld2(const float *p, long n) {
  return *reinterpret_cast<const float2 *>(p + n);
}
__device__ __forceinline__ void st2(float *p, long n, float x, float y) {
  *reinterpret_cast<float2 *>(p + n) = make_float2(x, y);
}

// r = rh = p = scale res, x = 0; s = rh times its row's scale, for w.
__global__ void __launch_bounds__(HT) hb_start(VecH a, const double *res, double scale) {
  DfAcc d[1] = {{0.f, 0.f}};
  PAIRS_OF(a) {
    const float b0 = (float)(res[n] * scale);
    const float b1 = n + 1 < a.h.N ? (float)(res[n + 1] * scale) : 0.f;
    st2(a.x, n, 0.f, 0.f);
    st2(a.r, n, b0, b1);
    st2(a.rh, n, b0, b1);
    st2(a.p, n, b0, b1);
    st2(a.s, n, b0 * exp2_int(a.h.e[n]), b1 * exp2_int(a.h.e[n + 1]));
    dot_acc(d[0], b0, b0);
    dot_acc(d[0], b1, b1);
  }
  double o[1];
  if (sums<1>(d, a, o)) {
    KState *st = a.st;
    st->bnrm2 = st->rho = o[0];
    st->err = o[0] == 0.0 ? 0.0 : 1.0;
    if (o[0] == 0.0) {
      st->status = VDR_OK;
      st->done = 1;
    } else if (!isfinite(o[0])) {
      st->status = VDR_BREAKDOWN;
      st->reason = 5;
      st->done = 1;
    } else if (st->err <= st->tol) {
      st->status = VDR_OK;
      st->done = 1;
    } else if (st->itmax <= 0) {
      st->done = 1;
    }
  }
}

__global__ void __launch_bounds__(HT, 4) hb_w(VecH a) {
  if (a.st->done) return;
  DfAcc d[1] = {{0.f, 0.f}};
  PAIRS_OF(a) {
    const float2 p = ld2(a.p, n);
    float w0, w1;
    trans_pair(a.h, n, a.s, w0, w1);
    st2(a.w, n, w0, w1);
    dot_acc(d[0], w0, p.x);
    dot_acc(d[0], w1, p.y);
  }
  double o[1];
  if (sums<1>(d, a, o)) set_alpha(a.st, o[0]);
}

// KEEP: the rows fit in L2 beside the vectors; otherwise they stream through
// it.  All 27 loads are issued before the first use.
template <bool KEEP>
__device__ __forceinline__ void row_pair(const VecH &a, long n, const float *xp, float &y0,
                                         float &y1) {
  const unsigned *h = reinterpret_cast<const unsigned *>(a.h.H + n);
  const long pitch = a.h.Np >> 1;
  unsigned e[27];
#pragma unroll
  for (int k = 0; k < 27; k++) e[k] = KEEP ? __ldcg(h + k * pitch) : __ldcs(h + k * pitch);
  pair_rows([&](int k) { return *reinterpret_cast<const __half2 *>(&e[k]); }, n, a.h, xp, y0,
            y1);
  y0 *= exp2_int(a.h.e[n]);
  y1 *= exp2_int(a.h.e[n + 1]);
}

template <bool KEEP>
__global__ void __launch_bounds__(HT, 4) hb_v(VecH a) {
  if (a.st->done) return;
  const float al = (float)a.st->alpha;
  DfAcc d[2] = {{0.f, 0.f}, {0.f, 0.f}};
  PAIRS_OF(a) {
    const float2 r = ld2(a.r, n), h = ld2(a.rh, n);
    float v0, v1;
    row_pair<KEEP>(a, n, a.p, v0, v1);
    const float s0 = r.x - al * v0, s1 = r.y - al * v1;
    st2(a.v, n, v0, v1);
    st2(a.s, n, s0, s1);
    dot_acc(d[0], s0, s0);
    dot_acc(d[0], s1, s1);
    dot_acc(d[1], h.x, s0);
    dot_acc(d[1], h.y, s1);
  }
  double o[2];
  if (sums<2>(d, a, o)) {
    KState *st = a.st;
    st->snrm = sqrt(o[0]) / sqrt(st->bnrm2);
    st->rhs = o[1];
    if (st->snrm <= st->tol) st->sconv = 1;
  }
}

template <bool KEEP>
__global__ void __launch_bounds__(HT, 4) hb_t(VecH a) {
  if (a.st->done || a.st->sconv) return;
  DfAcc d[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  PAIRS_OF(a) {
    const float2 s = ld2(a.s, n), h = ld2(a.rh, n);
    float t0, t1;
    row_pair<KEEP>(a, n, a.s, t0, t1);
    st2(a.t, n, t0, t1);
    dot_acc(d[0], t0, s.x);
    dot_acc(d[0], t1, s.y);
    dot_acc(d[1], t0, t0);
    dot_acc(d[1], t1, t1);
    dot_acc(d[2], h.x, t0);
    dot_acc(d[2], h.y, t1);
  }
  double o[3];
  if (sums<3>(d, a, o)) {
    KState *st = a.st;
    if (o[1] == 0.0 || !isfinite(o[1]) || !isfinite(o[0])) {
      st->status = VDR_BREAKDOWN;
      st->reason = 3;
      st->done = 1;
    } else {
      st->omega = o[0] / o[1];
      st->rho_next = st->rhs - st->omega * o[2];
      st->beta = (st->rho_next / st->rho) * (st->alpha / st->omega);
    }
  }
}

__global__ void __launch_bounds__(HT) hb_p(VecH a) {
  KState *st = a.st;
  if (st->done) return;
  const float al = (float)st->alpha;
  DfAcc d[2] = {{0.f, 0.f}, {0.f, 0.f}};
  double o[2];
  if (st->sconv) {  // s met the tolerance: x += alpha p
    PAIRS_OF(a) {
      const float2 x = ld2(a.x, n), p = ld2(a.p, n);
      st2(a.x, n, x.x + al * p.x, x.y + al * p.y);
    }
    if (sums<2>(d, a, o)) {
      st->iter += 1;
      st->err = st->snrm;
      st->status = VDR_OK;
      st->done = 1;
    }
    return;
  }
  const double omega = st->omega, rho1 = st->rho_next;
  const float om = (float)omega, beta = (float)st->beta;
  PAIRS_OF(a) {
    const float2 x = ld2(a.x, n), p = ld2(a.p, n), s = ld2(a.s, n), t = ld2(a.t, n),
                 v = ld2(a.v, n), w = ld2(a.w, n);
    st2(a.x, n, x.x + al * p.x + om * s.x, x.y + al * p.y + om * s.y);
    const float r0 = s.x - om * t.x, r1 = s.y - om * t.y;
    const float p0 = r0 + beta * (p.x - om * v.x), p1 = r1 + beta * (p.y - om * v.y);
    st2(a.r, n, r0, r1);
    st2(a.p, n, p0, p1);
    dot_acc(d[0], r0, r0);
    dot_acc(d[0], r1, r1);
    dot_acc(d[1], w.x, p0);
    dot_acc(d[1], w.y, p1);
  }
  if (sums<2>(d, a, o)) {
    st->iter += 1;
    st->rho = rho1;
    st->err = sqrt(o[0]) / sqrt(st->bnrm2);
    if (!(st->err == st->err) || !isfinite(rho1)) {
      st->status = VDR_BREAKDOWN;
      st->reason = 5;
      st->done = 1;
    } else if (st->err <= st->tol) {
      st->status = VDR_OK;
      st->done = 1;
    } else if (rho1 == 0.0 || omega == 0.0) {
      st->status = VDR_BREAKDOWN;
      st->reason = rho1 == 0.0 ? 1 : 4;
      st->done = 1;
    } else if (st->iter >= st->itmax) {
      st->status = VDR_NOT_CONVERGED;
      st->done = 1;
    } else {
      set_alpha(st, o[1]);
    }
  }
}

// x += scale D^-1 y
__global__ void __launch_bounds__(HT) hb_out(VecH a, double *x, double scale,
                                             const double *dinv) {
  for (long n = (long)blockIdx.x * blockDim.x + threadIdx.x; n < a.h.N;
       n += (long)gridDim.x * blockDim.x)
    x[n] += scale * dinv[n] * (double)a.x[n];
}

// ---- the whole inner solve in one launch (resident.cu's form) ----
// PAIRS pairs of nodes per thread, their rows in shared memory (54 bytes a
// node), their vector entries in registers; p and s through L2.
struct ResHArgs {
  HalfRows h;
  const double *res, *dinv;
  double scale, xscale;
  double *x;
  float *p, *s;
  KState *st;
  MeetArgs mt;
  double tol;
  int itmax;
};

template <int T, int PAIRS>
__global__ void __launch_bounds__(T, 1) resident_half(ResHArgs a) {
  extern __shared__ __half2 rows[];  // [27][PAIRS T]
  __shared__ ResShared sh;
  constexpr int M = PAIRS * T;
  const int N = a.h.N, none[1] = {0};
  unsigned target = 0;
  const auto nothing = [](int) {};
  float x[PAIRS][2], r[PAIRS][2], p[PAIRS][2], v[PAIRS][2], t[PAIRS][2], rh[PAIRS][2],
      w[PAIRS][2], sc[PAIRS][2];  // r holds s between the two products
  const auto node = [&](int i) { return 2L * ((long)blockIdx.x * M + i * T + threadIdx.x); };
  DfAcc d0{0.f, 0.f}, d1{0.f, 0.f}, d2{0.f, 0.f};
  const auto clear = [&]() { d0 = d1 = d2 = DfAcc{0.f, 0.f}; };
#pragma unroll
  for (int i = 0; i < PAIRS; i++) {
    const long n = node(i);
    const bool on = n < N;
    const __half2 *h = reinterpret_cast<const __half2 *>(a.h.H + (on ? n : 0));
#pragma unroll
    for (int k = 0; k < 27; k++)
      rows[k * M + i * T + threadIdx.x] =
          on ? __ldcg(h + k * (long)(a.h.Np >> 1)) : __float2half2_rn(0.f);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const bool is = n + j < N;
      sc[i][j] = is ? exp2_int(a.h.e[n + j]) : 0.f;
      const float b = is ? (float)(a.res[n + j] * a.scale) : 0.f;
      r[i][j] = rh[i][j] = p[i][j] = b;
      x[i][j] = v[i][j] = t[i][j] = w[i][j] = 0.f;
      dot_acc(d0, b, b);
    }
    if (on) {
      st2(a.p, n, p[i][0], p[i][1]);
      st2(a.s, n, rh[i][0] * sc[i][0], rh[i][1] * sc[i][1]);
    }
  }
  const auto product = [&](int i, const float *xp, float &y0, float &y1) {
    const long n = node(i);
    pair_rows([&](int k) { return rows[k * M + i * T + threadIdx.x]; }, n < N ? n : 0, a.h, xp,
              y0, y1);
    y0 *= sc[i][0];
    y1 *= sc[i][1];
  };
  {
    const double q[1] = {dot_val(d0)};
    if (!meet<IN_REGS, T, 1, 0, 1, AT_A, AT_A, 0>(sh, a.mt, q, none, target, nothing))
      return;
  }
  const double bnrm2 = sh.tot[0];
  double rho = bnrm2, rr2 = bnrm2, al64 = 0.0, iwp = 0.0;
  const double thr = a.tol * a.tol * bnrm2;
  int iter = 0, status = VDR_NOT_CONVERGED, reason = 0;
  bool done = false;
  if (bnrm2 == 0.0) {
    status = VDR_OK;
    done = true;
  } else if (!isfinite(bnrm2)) {
    status = VDR_BREAKDOWN;
    reason = 5;
    done = true;
  } else if (rr2 <= thr) {
    status = VDR_OK;
    done = true;
  } else if (a.itmax <= 0) {
    done = true;
  }
  const auto alpha_of = [&](int lane, double wp) {
    const double d = (lane ? 1.0 : rho) / wp;
    if (lane < 2) sh.tot[2 + lane] = d;
  };
  if (!done) {
    clear();
#pragma unroll
    for (int i = 0; i < PAIRS; i++)
      if (node(i) < N) {
        trans_pair(a.h, node(i), a.s, w[i][0], w[i][1]);
#pragma unroll
        for (int j = 0; j < 2; j++) dot_acc(d0, w[i][j], p[i][j]);
      }
    const double q[1] = {dot_val(d0)};
    if (!meet<IN_REGS, T, 1, 0, 1, AT_D, AT_D, 0>(
            sh, a.mt, q, none, target, [&](int lane) { alpha_of(lane, sh.tot[0]); }))
      return;
    if (sh.tot[0] == 0.0 || !isfinite(sh.tot[0])) {
      status = VDR_BREAKDOWN;
      reason = 2;
      done = true;
    }
    al64 = sh.tot[2];
    iwp = sh.tot[3];
  }
  while (!done) {
    const float al = (float)al64;
    clear();
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
      product(i, a.p, v[i][0], v[i][1]);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float s = r[i][j] - al * v[i][j];
        r[i][j] = s;
        dot_acc(d0, s, s);
        dot_acc(d1, rh[i][j], s);
      }
      if (node(i) < N) st2(a.s, node(i), r[i][0], r[i][1]);
    }
    {
      const double q[2] = {dot_val(d0), dot_val(d1)};
      if (!meet<IN_REGS, T, 2, 0, 0, AT_C, AT_C, 0>(sh, a.mt, q, none, target, nothing))
        return;
    }
    clear();
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
      product(i, a.s, t[i][0], t[i][1]);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        dot_acc(d0, t[i][j], r[i][j]);
        dot_acc(d1, t[i][j], t[i][j]);
        dot_acc(d2, t[i][j], rh[i][j]);
      }
    }
    {
      const double q[3] = {dot_val(d0), dot_val(d1), dot_val(d2)};
      if (!meet<IN_REGS, T, 3, 0, 5, AT_D, AT_C, 0>(sh, a.mt, q, none, target, [&](int lane) {
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
    const double ss = sh.tot[0], omega = sh.tot[1], ts = sh.tot[2], tt = sh.tot[3],
                 rho1 = sh.tot[4];
    const float om = (float)omega, beta = (float)sh.tot[5];
    if (ss <= thr) {  // s met the tolerance: x += alpha p
#pragma unroll
      for (int i = 0; i < PAIRS; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) x[i][j] += al * p[i][j];
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
    clear();
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float s = r[i][j];
        x[i][j] += al * p[i][j] + om * s;
        const float rn = s - om * t[i][j];
        p[i][j] = rn + beta * (p[i][j] - om * v[i][j]);
        r[i][j] = rn;
        dot_acc(d0, rn, rn);
        dot_acc(d1, w[i][j], p[i][j]);
      }
      if (node(i) < N) st2(a.p, node(i), p[i][0], p[i][1]);
    }
    rho = rho1;
    {
      const double q[2] = {dot_val(d0), dot_val(d1)};
      if (!meet<IN_REGS, T, 2, 0, 2, AT_A, AT_A, 0>(
              sh, a.mt, q, none, target, [&](int lane) { alpha_of(lane, sh.tot[1]); }))
        return;
    }
    rr2 = sh.tot[0];
    const double wp = sh.tot[1];
    al64 = sh.tot[2];
    iwp = sh.tot[3];
    iter++;
    if (!(rr2 == rr2) || !isfinite(rho1)) {
      status = VDR_BREAKDOWN;
      reason = 5;
      done = true;
    } else if (rr2 <= thr) {
      status = VDR_OK;
      done = true;
    } else if (rho1 == 0.0 || omega == 0.0) {
      status = VDR_BREAKDOWN;
      reason = rho1 == 0.0 ? 1 : 4;
      done = true;
    } else if (iter >= a.itmax) {
      done = true;
    } else if (wp == 0.0 || !isfinite(wp)) {
      status = VDR_BREAKDOWN;
      reason = 2;
      done = true;
    }
  }
#pragma unroll
  for (int i = 0; i < PAIRS; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const long n = node(i) + j;
      if (n < N) a.x[n] += a.xscale * a.dinv[n] * (double)x[i][j];
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    KState *st = a.st;
    st->iter = iter;
    st->err = bnrm2 > 0.0 ? sqrt(rr2) / sqrt(bnrm2) : 0.0;
    st->status = status;
    st->reason = reason;
    st->done = 1;
  }
}

template <int T, int PAIRS>
cudaError_t launch_resident_half(int N, const ResHArgs &a, cudaStream_t s) {
  const auto kern = resident_half<T, PAIRS>;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((N + 2L * T * PAIRS - 1) / (2L * T * PAIRS)));
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = sizeof(__half2) * 27 * T * PAIRS;
  cfg.stream = s;
  const cudaError_t e = cudaFuncSetAttribute(
      kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes);
  if (e) return e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, a);
}

size_t vec_pad(const Handle &h) {  // zeros around p and s; keeps pairs aligned
  return ((size_t)h.nax * h.nay + h.nax + 2 + 31) & ~(size_t)31;
}

HalfRows rows_view(const Handle &h) {
  HalfRows v;
  v.H = reinterpret_cast<const __half *>(h.hr_H);
  v.e = h.hr_e;
  v.N = h.N;
  v.Np = (h.N + 7) & ~7;
  v.nax = h.nax;
  v.pl = h.nax * h.nay;
  return v;
}

}  // namespace

bool half_rows_ready(const Handle &h) {
  return h.hr_state == 1 && h.st_state == 1 && h.mixed_op == VDR_MIXED_HALF;
}

int ensure_half_rows(Handle &h) {
  if (h.hr_state != 0 || h.mixed_op != VDR_MIXED_HALF) return VDR_OK;
  cudaError_t e = ensure_stencil(h);
  if (e) return cuda_fail(e, "assembled rows");
  if (!stencil_ready(h)) return VDR_OK;
  const size_t Np = ((size_t)h.N + 7) & ~(size_t)7, pad = vec_pad(h), V = Np + 2 * pad;
  if (!h.hr_H) {
    const size_t need = 54 * Np + Np + sizeof(float) * (6 * Np + 2 * V);
    size_t free_b = 0, total_b = 0;
    if (!h.rows_room || cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || need > free_b / 2 ||
        cudaMalloc(&h.hr_H, 54 * Np) || cudaMalloc(&h.hr_e, Np) ||
        cudaMalloc(&h.hr_vec, sizeof(float) * (6 * Np + 2 * V)) ||
        cudaMemsetAsync(h.hr_vec, 0, sizeof(float) * (6 * Np + 2 * V), h.stream)) {
      cudaGetLastError();  // no room: the element-wise inner operator
      cudaFree(h.hr_H);
      cudaFree(h.hr_e);
      cudaFree(h.hr_vec);
      h.hr_H = nullptr;
      h.hr_e = nullptr;
      h.hr_vec = nullptr;
      h.hr_state = -1;
      return VDR_OK;
    }
  }
  const int grid =
      (int)std::min<long>((long)(Np + 255) / 256, (long)device_sm_count() * 16);
  int bad = 0;
  if ((e = cudaMemsetAsync(h.flag, 0, sizeof(int), h.stream)))
    return cuda_fail(e, "16-bit rows");
  half_rows_kernel<<<grid, 256, 0, h.stream>>>(stencil_view(h), h.dinv,
                                               reinterpret_cast<__half *>(h.hr_H), h.hr_e,
                                               (int)Np, h.flag);
  count_launches(1);
  if ((e = cudaGetLastError()) ||
      (e = cudaMemcpyAsync(&bad, h.flag, sizeof(int), cudaMemcpyDeviceToHost, h.stream)) ||
      (e = cudaStreamSynchronize(h.stream)))
    return cuda_fail(e, "16-bit rows");
  h.hr_state = bad ? 2 : 1;
  return VDR_OK;
}

// One correction: y from A^ y = res / rnorm to `tol` on FP32 vectors, then x
// += rnorm D^-1 y.
int solve_half_rows(Handle &h, const double *res, double rnorm, double *x, double tol,
                    int itmax, int *iter, double *err) {
  cudaStream_t s = h.stream;
  cudaError_t e = cudaSuccess;
  const size_t Np = ((size_t)h.N + 7) & ~(size_t)7, pad = vec_pad(h), V = Np + 2 * pad;
  VecH a{};
  a.h = rows_view(h);
  a.st = h.st;
  a.partials = h.partials;
  float *f = h.hr_vec;
  a.x = f;
  a.r = f + Np;
  a.rh = f + 2 * Np;
  a.v = f + 3 * Np;
  a.t = f + 4 * Np;
  a.w = f + 5 * Np;
  a.p = f + 6 * Np + pad;
  a.s = a.p + V;
  const long sms = std::min(device_sm_count(), 32 * RES_NB);
  if (h.resident && h.N <= 4096 * sms) {
    ResHArgs ra{a.h, res, h.dinv, 1.0 / rnorm, rnorm, x, a.p, a.s, h.st, meet_args(h),
                tol, itmax};
    if ((e = meet_reset(h, s))) return cuda_fail(e, "inner solve");
    if (h.N <= 256 * sms) e = launch_resident_half<128, 1>(h.N, ra, s);
    else if (h.N <= 512 * sms) e = launch_resident_half<256, 1>(h.N, ra, s);
    else if (h.N <= 1024 * sms) e = launch_resident_half<512, 1>(h.N, ra, s);
    else if (h.N <= 2048 * sms) e = launch_resident_half<1024, 1>(h.N, ra, s);
    else if (h.N <= 3072 * sms) e = launch_resident_half<768, 2>(h.N, ra, s);
    else e = launch_resident_half<1024, 2>(h.N, ra, s);
    if (!e) {
      count_launches(1);
      if ((e = cudaMemcpyAsync(&h.h_st[0], h.st, sizeof(KState), cudaMemcpyDeviceToHost, s)) ||
          (e = cudaStreamSynchronize(s)))
        return cuda_fail(e, "inner solve");
      const KState &fin = h.h_st[0];
      if (iter) *iter = fin.late ? 0 : fin.iter;
      if (err) *err = fin.late ? INFINITY : fin.err;
      return outcome(fin);
    }
    cudaGetLastError();
    h.resident = false;
  }
  KState init{};
  init.tol = tol;
  init.itmax = itmax;
  init.status = VDR_NOT_CONVERGED;
  std::memcpy(&h.h_st[0], &init, sizeof(KState));
  if ((e = cudaMemcpyAsync(h.st, &h.h_st[0], sizeof(KState), cudaMemcpyHostToDevice, s)))
    return cuda_fail(e, "state upload");
  const bool keep = 55.0 * h.N < 80.0e6;
  const long need = (h.N / 2 + HT) / HT;
  const int g = (int)std::max<long>(1, std::min<long>(need, device_sm_count() * 4L));
  hb_start<<<g, HT, 0, s>>>(a, res, 1.0 / rnorm);
  hb_w<<<g, HT, 0, s>>>(a);
  count_launches(2);
  if ((e = cudaGetLastError())) return cuda_fail(e, "start kernel");
  const int K = h.opt.iters_per_graph > 0 ? h.opt.iters_per_graph : 8;
  if (!h.hr_graph || h.hr_graph_iters != K) {  // its arguments are the handle's own
    if (h.hr_graph) cudaGraphExecDestroy(h.hr_graph);
    h.hr_graph = nullptr;
    cudaGraph_t graph;
    if ((e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal)))
      return cuda_fail(e, "begin capture");
    for (int k = 0; k < K; k++) {
      if (keep) {
        hb_v<true><<<g, HT, 0, s>>>(a);
        hb_t<true><<<g, HT, 0, s>>>(a);
      } else {
        hb_v<false><<<g, HT, 0, s>>>(a);
        hb_t<false><<<g, HT, 0, s>>>(a);
      }
      hb_p<<<g, HT, 0, s>>>(a);
    }
    e = cudaGetLastError();
    const cudaError_t e2 = cudaStreamEndCapture(s, &graph);
    if (e || e2) return cuda_fail(e ? e : e2, "capture");
    e = cudaGraphInstantiate(&h.hr_graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e) {
      h.hr_graph = nullptr;
      return cuda_fail(e, "capture");
    }
    h.hr_graph_iters = K;
  }
  const int max_launches = (itmax + K - 1) / K + 1;
  bool finished = false;
  for (int c = 0; c < max_launches && !finished; c++) {
    if ((e = cudaGraphLaunch(h.hr_graph, s))) return cuda_fail(e, "graph launch");
    count_launches(3L * K);
    if ((e = cudaMemcpyAsync(&h.h_st[c & 1], h.st, sizeof(KState), cudaMemcpyDeviceToHost, s)) ||
        (e = cudaEventRecord(h.ev[c & 1], s)))
      return cuda_fail(e, "state readback");
    if (c > 0) {
      if ((e = cudaEventSynchronize(h.ev[(c - 1) & 1]))) return cuda_fail(e, "sync");
      if (h.h_st[(c - 1) & 1].done) finished = true;
    }
  }
  hb_out<<<g, HT, 0, s>>>(a, x, rnorm, h.dinv);
  count_launches(1);
  KState fin;
  if ((e = cudaGetLastError()) || (e = cudaStreamSynchronize(s)) ||
      (e = cudaMemcpy(&fin, h.st, sizeof(KState), cudaMemcpyDeviceToHost)))
    return cuda_fail(e, "inner solve");
  if (iter) *iter = fin.iter;
  if (err) *err = fin.err;
  return fin.done ? fin.status : VDR_NOT_CONVERGED;
}

}  // namespace vdr
