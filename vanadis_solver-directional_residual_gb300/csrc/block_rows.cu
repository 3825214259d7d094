// block_rows.cu -- the block solve on assembled 27-point rows.
//
// On the canonical structured numbering a product with K columns needs 27
// multiply-adds per node and column where the element matrices need 64 per
// element and column, atomics into a cleared result, and passes of their own
// for every inner product.  Here a thread owns four columns of one (x, y)
// and marches along z: it reads the nine neighbours of a plane once and adds
// them to the three output rows they feed, so a result is complete where it
// is formed and the inner products with it cost one more read at most.
// Plain FP32 multiply-adds (24 bits, against 21 of the split TF32 product and
// 11 of plain TF32) are not what bounds it: 27 of them are 27 cycles a warp
// and SM, the 39 bytes that a thread moves for its four outputs 53 at the
// HBM's rate.
//
// An iteration is four kernels and 17 passes over block vectors:
//   product  v = A D^-1 p;  (rh, v)                        p, rh -> v
//   br_s     s = r - alpha v;  (s, s)                      r, v -> s
//   product  t = A D^-1 s;  (t,s) (t,t) (rh,t) (rh,s)      s, rh -> t
//   br_xp    x, r = s - omega t, the next p;  (r, r)       s,t,x,p,v -> x,r,p
// with rho' = (rh, s) - omega (rh, t), where the element-wise form takes
// seven kernels and 26 passes (clearing v and t among them).  The FP64
// residual of the refinement runs the same way on the pair rows.  At 1.08 M
// nodes and 64 columns an iteration takes 905 us instead of 1346, a residual
// 1.8 ms instead of 3.9 + 0.35; a whole solve 128 -> 83 ms, and 4.1 -> 3.5 ms
// at 343 nodes.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "block_cols.cuh"
#include "stencil.cuh"
#include "tc_ptx.cuh"

namespace vdr {
namespace {

// The product's blocks: K / 4 lanes a pair of nodes along x, PT threads a
// tile of TX x TY nodes; the tile and its neighbours of one plane (SX x SY
// nodes) and the tile's rows make a stage.
constexpr int PT = 256, STAGES = 4;
template <int K>
struct Tile {
  static constexpr int L = K / 4, TX = K == 16 ? 16 : 8, TY = PT / L / (TX / 2);
  static constexpr int SX = TX + 2, SY = TY + 2;
  static constexpr int XB = SX * SY * K * 4, RB = TX * TY * 112;  // bytes of a plane
  static constexpr int STAGE = XB + RB, PRODUCT = STAGES * STAGE, RESIDUAL = 4 * XB + 2 * 27 * TX * TY * 8;
};

// Per-column sums of NQ quantities over the grid; true in every thread of
// the last block, with the totals in out[q K + k] (shared).  A warp's lanes
// with the same columns fold first; partials lie [block][q][k], so the last
// block reads whole lines.
constexpr int sum_words(int K, int NQ, int NT) {
  return NT / 32 * NQ * K > NT ? NT / 32 * NQ * K : NT;
}
template <int K, int NQ, int NT, class D>
__device__ __forceinline__ bool col_sums(const D (&d)[NQ][4], const BVec &a, double *sm,
                                         double *out) {
  constexpr int L = K / 4, P = NQ * K, SL = NT / P > 0 ? NT / P : 1;
  __shared__ int last;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
#pragma unroll
  for (int q = 0; q < NQ; q++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      double v = dot_val(d[q][c]);
#pragma unroll
      for (int o = L; o < 32; o <<= 1) v += __shfl_xor_sync(FULLR, v, o);
      if (lane < L) sm[w * P + q * K + 4 * lane + c] = v;
    }
  __syncthreads();
  for (int j = tid; j < P; j += NT) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < NT / 32; i++) s += sm[i * P + j];
    a.partials[(size_t)blockIdx.x * P + j] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&a.st->ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int G = (int)gridDim.x;
  for (int j = tid; j < SL * P; j += NT) {
    const int i = j % P;
    double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int b = j / P; b < G; b += 8 * SL) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; u++)
        v[u] = b + u * SL < G ? __ldcg(a.partials + (size_t)(b + u * SL) * P + i) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; u++) s[u] += v[u];
    }
    sm[j] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
  }
  __syncthreads();
  for (int j = tid; j < P; j += NT) {
    double t = 0.0;
    for (int u = 0; u < SL; u++) t += sm[u * P + j];
    out[j] = t;
  }
  __syncthreads();
  if (tid == 0) a.st->ticket = 0u;
  return true;
}

__device__ __forceinline__ float2 half_of(const float4 &v, int h) {
  return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
}

__device__ __forceinline__ void fma4(float4 &o, float c, const float4 &x) {
  o.x = fmaf(c, x.x, o.x);
  o.y = fmaf(c, x.y, o.y);
  o.z = fmaf(c, x.z, o.z);
  o.w = fmaf(c, x.w, o.w);
}
template <int NQ>
__device__ __forceinline__ void clear(DfAcc (&d)[NQ][4]) {
#pragma unroll
  for (int q = 0; q < NQ; q++)
#pragma unroll
    for (int c = 0; c < 4; c++) d[q][c] = DfAcc{0.f, 0.f};
}
// Whether any of the thread's four columns is still iterating.
template <int K>
__device__ __forceinline__ bool group_active(const BVec &a) {
  const int4 on = reinterpret_cast<const int4 *>(a.c.active)[threadIdx.x % (K / 4)];
  return on.x | on.y | on.z | on.w;
}

// The rows in the order in which the march reads them: node n = (x, y, z)
// holds the entries that multiply plane z around (x, y), for the rows one
// plane down, in the plane and one plane up: rows[28 n + 9 (c / 3) + 3 j +
// c % 3] = entry 9 (2 - j) + c of node n + (j - 1) planes, times D^-1 of the
// neighbour, c = 3 (dy + 1) + dx + 1.
__global__ void br_rows(const float2 *__restrict__ S, const float *__restrict__ dinv, int N, int nax,
                        int pl, float *__restrict__ rows) {
  for (long n = (long)blockIdx.x * blockDim.x + threadIdx.x; n < N;
       n += (long)gridDim.x * blockDim.x) {
    float o[28];
    o[27] = 0.f;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const long row = n + (j - 1) * (long)pl;
      const bool in = row >= 0 && row < N;
#pragma unroll
      for (int c = 0; c < 9; c++) {
        float2 e = make_float2(0.f, 0.f);
        if (in) e = S[(size_t)(9 * (2 - j) + c) * N + row];
        const long q = n + (c / 3 - 1) * nax + (c % 3 - 1);
        const float d = (e.x != 0.f && q >= 0 && q < N) ? dinv[q] : 0.f;
        o[9 * (c / 3) + 3 * j + c % 3] = e.x != 0.f ? fmaf(e.x, d, e.y * d) : 0.f;
      }
    }
    float4 *r = reinterpret_cast<float4 *>(rows + 28 * n);
#pragma unroll
    for (int u = 0; u < 7; u++) r[u] = make_float4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
  }
}

// A block's share of the tiles' planes: whole columns in rounds while there is
// one for every block, so that neighbouring tiles march side by side and find
// their common nodes in L2, then an equal part of the columns left, taken as
// one sequence along z, then over the tiles.  Segments [z0, z1) of a tile,
// read from the plane before to the plane after.
struct Share {
  int round, rounds, first;  // columns taken in rounds, all of them
  long at, end;
  int x0, y0, z0, z1, zb, ze;
  __device__ Share(const BlockRows &g) {
    const int tiles = g.nxt * g.nyt, G = (int)gridDim.x;
    round = 0;
    rounds = tiles / G;
    first = rounds * G;
    const long total = (long)(tiles - first) * g.naz;
    at = total * blockIdx.x / G;
    end = total * (blockIdx.x + 1) / G;
  }
  template <class T>
  __device__ bool next(const BlockRows &g) {
    int t;
    if (round < rounds) {
      t = (round++) * (int)gridDim.x + (int)blockIdx.x;
      z0 = 0;
      z1 = g.naz;
    } else {
      if (at >= end) return false;
      t = (int)(at / g.naz);
      z0 = (int)(at - (long)t * g.naz);
      z1 = (int)min((long)g.naz, z0 + (end - at));
      at += z1 - z0;
      t += first;
    }
    x0 = t % g.nxt * T::TX;
    y0 = t / g.nxt * T::TY;
    zb = max(z0 - 1, 0);
    ze = min(z1, g.naz - 1);
    return true;
  }
};

constexpr long long WAIT_LIMIT = 2000000000LL;  // ~1 s of clocks per wait

// After a wait of a ring of copies ran out: says so and lets the copies on
// their way land (each wait bounded).  One thread.
template <int ST>
__device__ __forceinline__ void ring_gave_up(uint64_t (&full)[ST], int *err, int bit,
                                             long long limit) {
  atomicOr(err, bit);
  for (int i = 0; i < ST; i++) {
    tc::mbar_wait(tc::smem_u32(full + i), 0u, limit);
    tc::mbar_wait(tc::smem_u32(full + i), 1u, limit);
  }
}

// The ring's failure path on its own: a stage announced whose copy is never
// issued, so nothing is in flight.
__global__ void __launch_bounds__(32) ring_timeout_kernel(int *err, int bit, long long limit) {
  __shared__ __align__(8) uint64_t full[STAGES];
  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; i++) tc::mbar_init(tc::smem_u32(full + i), 1);
    tc::mbar_init_fence();
    tc::mbar_arrive_expect_tx(tc::smem_u32(full), 1024);
  }
  __syncthreads();
  const bool ok = __syncthreads_and(tc::mbar_wait(tc::smem_u32(full), 0u, limit));
  if (!ok && threadIdx.x == 0) ring_gave_up(full, err, bit, limit);
}

struct Maps {
  CUtensorMap x, rows;
};

// v = A D^-1 p with (rh, v) and alpha, or (SECOND) t = A D^-1 s with its four
// products, omega and the next rho.  A block marches along z with STAGES
// planes of the input's tile and of the rows in shared memory, three of them
// on their way (tensor copies, which also put the zeros beyond the faces).
// At 1.08 M nodes and 64 columns, the two products: straight from L1, nine
// 16-byte loads a node, 254 and 437 us (latency); tiles fetched by the
// threads' own asynchronous copies 264 and 355 (as many instructions for
// addresses as for products); by tensor copies 212 and 280; with the inner
// products packed and rh prefetched to L2 190 and 272; with
// the columns taken side by side (Share) 167 and 270 (HBM: 140 each; the
// second is bound by issue, 60 % busy with its four products).  Three blocks
// an SM for the first: no change.  Forming s in the second product's tiles
// instead of in br_s (130 us) took 594: the registers do not suffice.
template <int K, bool SECOND>
__global__ void __launch_bounds__(PT, 2) br_apply(const BVec a, const BlockRows g,
                                                  const __grid_constant__ Maps maps) {
  using T = Tile<K>;
  constexpr int NQ = SECOND ? 4 : 1, L = T::L, ST = STAGES;
  extern __shared__ __align__(128) unsigned char stage[];
  __shared__ __align__(8) uint64_t full[ST];
  if (a.st->done) return;
  DfAccx2 d[NQ][2];
#pragma unroll
  for (int q = 0; q < NQ; q++)
    d[q][0] = d[q][1] = DfAccx2{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  const float4 *__restrict__ H = reinterpret_cast<const float4 *>(a.rh);
  float4 *__restrict__ Y = reinterpret_cast<float4 *>(SECOND ? a.t : a.v);
  const int l = threadIdx.x % L, pair = threadIdx.x / L;
  const int px = 2 * (pair % (T::TX / 2)), py = pair / (T::TX / 2);
  const int pl = g.nax * g.nay;
  if (threadIdx.x == 0) {
    for (int i = 0; i < ST; i++) tc::mbar_init(tc::smem_u32(full + i), 1);
    tc::mbar_init_fence();
  }
  __syncthreads();
  const bool on = group_active<K>(a);
  bool ok = true;
  unsigned seen = 0;  // planes of the segments before
  for (Share w(g); ok && w.template next<T>(g);) {
    const int count = w.ze - w.zb + 1;
    const auto fetch = [&](int i) {  // the segment's plane i
      if (i >= count || threadIdx.x != 0) return;
      const unsigned q = seen + (unsigned)i;
      const uint32_t bar = tc::smem_u32(full + q % ST);
      const uint32_t dst = tc::smem_u32(stage + q % ST * T::STAGE);
      tc::mbar_arrive_expect_tx(bar, T::STAGE);
      tc::tma_load_4d(dst, &maps.x, 0, w.x0 - 1, w.y0 - 1, w.zb + i, bar);
      tc::tma_load_4d(dst + T::XB, &maps.rows, 0, w.x0, w.y0, w.zb + i, bar);
    };
#pragma unroll
    for (int u = 0; u < ST - 1; u++) fetch(u);
    const bool in0 = on && w.x0 + px < g.nax && w.y0 + py < g.nay;
    const bool in1 = in0 && w.x0 + px + 1 < g.nax;
    float4 lo[2], mid[2], up[2], last[2];
#pragma unroll
    for (int u = 0; u < 2; u++) lo[u] = mid[u] = last[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    long n = (((long)w.zb * g.nay + w.y0 + py) * g.nax + w.x0 + px) * L + l;
    for (int i = 0; i < count; i++, n += (long)pl * L) {
      const int z = w.zb + i;
      const unsigned q = seen + (unsigned)i;
      ok = __syncthreads_and(ok);
      if (!ok) break;
      fetch(i + ST - 1);
      ok = tc::mbar_wait(tc::smem_u32(full + q % ST), q / ST & 1u, WAIT_LIMIT);
      if (!in0 || !ok) continue;
      const bool out = z > w.z0;
      float4 h[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        h[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (out && (u ? in1 : in0)) h[u] = H[n + (u - (long)pl) * L];
      }
      // the shadow residual of the next plane, on its way to L2
      if (z + 1 < g.naz && l % 8 == 0) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(H + n + (long)pl * L));
        if (in1) asm volatile("prefetch.global.L2 [%0];" ::"l"(H + n + (long)pl * L + L));
      }
      const unsigned char *st = stage + q % ST * T::STAGE;
      const float4 *xs = reinterpret_cast<const float4 *>(st) + (py * T::SX + px) * L + l;
      const float4 *rs = reinterpret_cast<const float4 *>(st + T::XB) + (py * T::TX + px) * 7;
      float e[2][28];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        up[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 7; j++) {
          const float4 r = rs[7 * u + j];
          e[u][4 * j] = r.x;
          e[u][4 * j + 1] = r.y;
          e[u][4 * j + 2] = r.z;
          e[u][4 * j + 3] = r.w;
        }
      }
      float4 mine[2];
#pragma unroll
      for (int dy = 0; dy < 3; dy++) {
        float4 xv[4];
#pragma unroll
        for (int j = 0; j < 4; j++) xv[j] = xs[(dy * T::SX + j) * L];
        if (dy == 1) {
          mine[0] = xv[1];
          mine[1] = xv[2];
        }
#pragma unroll
        for (int dx = 0; dx < 3; dx++)
#pragma unroll
          for (int u = 0; u < 2; u++) {
            fma4(lo[u], e[u][9 * dy + dx], xv[dx + u]);
            fma4(mid[u], e[u][9 * dy + 3 + dx], xv[dx + u]);
            fma4(up[u], e[u][9 * dy + 6 + dx], xv[dx + u]);
          }
      }
      // row z - 1 is complete; on the grid's last plane row z is too
#pragma unroll 1
      for (int fin = 0; fin < 2; fin++) {
        if (fin == 0 ? out : (z == g.naz - 1 && z < w.z1)) {
          const long o = fin == 0 ? n - (long)pl * L : n;
#pragma unroll
          for (int u = 0; u < 2; u++) {
            if (!(u ? in1 : in0)) continue;
            if (fin) h[u] = H[o + u * L];
            Y[o + u * L] = lo[u];
#pragma unroll
            for (int c = 0; c < 2; c++) {
              const float2 y2 = half_of(lo[u], c), h2 = half_of(h[u], c), ny = neg2(y2);
              if (SECOND) {
                const float2 s2 = half_of(last[u], c);
                dot_acc2(d[0][c], y2, ny, s2);
                dot_acc2(d[1 % NQ][c], y2, ny, y2);
                dot_acc2(d[2 % NQ][c], y2, ny, h2);
                dot_acc2(d[3 % NQ][c], s2, neg2(s2), h2);
              } else {
                dot_acc2(d[0][c], y2, ny, h2);
              }
            }
          }
        }
        if (fin == 0)
#pragma unroll
          for (int u = 0; u < 2; u++) {
            lo[u] = mid[u];
            mid[u] = up[u];
            last[u] = mine[u];
          }
      }
    }
    seen += (unsigned)count;
    ok = __syncthreads_and(ok);  // and the segment's stages are read
  }
  if (!ok && threadIdx.x == 0) {  // a copy did not arrive: the iteration stops
    *(volatile int *)&a.st->done = 1;
    ring_gave_up(full, g.err, 1, WAIT_LIMIT);
  }
  __syncthreads();
  DfAcc sums[NQ][4];
#pragma unroll
  for (int q = 0; q < NQ; q++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
      sums[q][2 * c] = DfAcc{d[q][c].s.x, d[q][c].c.x};
      sums[q][2 * c + 1] = DfAcc{d[q][c].s.y, d[q][c].c.y};
    }
  double *sm = reinterpret_cast<double *>(stage), *out = sm + sum_words(K, NQ, PT);
  if (!col_sums<K, NQ, PT>(sums, a, sm, out) || threadIdx.x >= K) return;
  const int k = threadIdx.x;
  if (!a.c.active[k]) return;
  if (!SECOND) {
    const double rv = out[k];
    if (rv == 0.0 || !isfinite(rv)) {
      a.c.active[k] = 0;
      a.c.status[k] = VDR_BREAKDOWN;
      a.c.alpha[k] = 0.0;
    } else {
      a.c.alpha[k] = a.c.rho[k] / rv;
    }
  } else if (!a.c.sconv[k]) {
    const double ts = out[k], tt = out[K + k];
    const double om = (tt == 0.0 || !isfinite(tt) || !isfinite(ts)) ? 0.0 : ts / tt;
    a.c.omega[k] = om;
    a.c.rho_next[k] = out[3 * K + k] - om * out[2 * K + k];
  }
}

// s = r - alpha v, ||s|| per column.
template <int K>
__global__ void __launch_bounds__(BT, 2) br_s(const BVec a) {
  if (a.st->done) return;
  const int k0 = 4 * (threadIdx.x % (K / 4));
  DfAcc d[1][4];
  clear<1>(d);
  if (group_active<K>(a)) {
    float al[4];
#pragma unroll
    for (int c = 0; c < 4; c++) al[c] = a.c.active[k0 + c] ? (float)a.c.alpha[k0 + c] : 0.f;
    ULOOP(j) {
      const float4 rv = ld4(a.r, j), vv = ld4(a.v, j);
      const float4 sv = make_float4(rv.x - al[0] * vv.x, rv.y - al[1] * vv.y,
                                    rv.z - al[2] * vv.z, rv.w - al[3] * vv.w);
#pragma unroll
      for (int c = 0; c < 4; c++) dot_acc(d[0][c], f4(sv, c), f4(sv, c));
      st4(a.s, j, sv);
    }
  }
  __shared__ double sm[sum_words(K, 1, BT)], out[K];
  if (!col_sums<K, 1, BT>(d, a, sm, out) || threadIdx.x >= K) return;
  const int k = threadIdx.x;
  const double sn = a.c.bnrm2[k] > 0.0 ? sqrt(out[k] / a.c.bnrm2[k]) : 0.0;
  a.c.snrm[k] = sn;
  a.c.sconv[k] = (a.c.active[k] && sn <= a.c.tol[k]) ? 1 : 0;
}

// x += D^-1 (alpha p + omega s) (Dirichlet entries stay); r = s - omega t (s
// where it met the tolerance); p = r + beta (p - omega v); the iteration's end.
// Columns that have finished keep x and r.
template <int K>
__global__ void __launch_bounds__(BT, 2) br_xp(const BVec a) {
  if (a.st->done) return;
  const int k0 = 4 * (threadIdx.x % (K / 4));
  DfAcc d[1][4];
  clear<1>(d);
  if (group_active<K>(a)) {
    bool act[4];
    float al[4], om[4], be[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int k = k0 + c;
      act[c] = a.c.active[k] != 0;
      const bool go = act[c] && !a.c.sconv[k] && a.c.omega[k] != 0.0;
      al[c] = act[c] ? (float)a.c.alpha[k] : 0.f;
      om[c] = go ? (float)a.c.omega[k] : 0.f;
      be[c] = go ? (float)((a.c.rho_next[k] / a.c.rho[k]) * (a.c.alpha[k] / a.c.omega[k])) : 0.f;
    }
    ULOOP(j) {
      const long node = j / (K / 4);
      const float4 xv = ld4(a.x, j), sv = ld4(a.s, j), tv = ld4(a.t, j);
      const float4 pv = ld4(a.p, j), vv = ld4(a.v, j);
      float4 rv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!(act[0] && act[1] && act[2] && act[3])) rv = ld4(a.r, j);
      const float dn = a.m[node] ? 0.f : a.dinv[node];
      float xo[4], ro[4], po[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float p = f4(pv, c), s = f4(sv, c);
        const float ri = act[c] ? s - om[c] * f4(tv, c) : f4(rv, c);
        xo[c] = act[c] ? f4(xv, c) + dn * (al[c] * p + om[c] * s) : f4(xv, c);
        ro[c] = ri;
        po[c] = act[c] ? ri + be[c] * (p - om[c] * f4(vv, c)) : 0.f;
        dot_acc(d[0][c], ri, ri);
      }
      st4(a.x, j, make_float4(xo[0], xo[1], xo[2], xo[3]));
      st4(a.r, j, make_float4(ro[0], ro[1], ro[2], ro[3]));
      st4(a.p, j, make_float4(po[0], po[1], po[2], po[3]));
    }
  }
  __shared__ double sm[sum_words(K, 1, BT)], out[K];
  if (!col_sums<K, 1, BT>(d, a, sm, out)) return;
  bool on = false;
  if (threadIdx.x < K) {
    const int k = threadIdx.x;
    if (a.c.active[k]) {
      const bool sc = a.c.sconv[k] != 0;
      const double om = a.c.omega[k], rho = a.c.rho_next[k];
      const double err = sqrt(out[k] / a.c.bnrm2[k]);
      a.c.err[k] = err;
      if (!sc) a.c.rho[k] = rho;
      int st = VDR_NOT_CONVERGED;
      if (!(err == err)) st = VDR_BREAKDOWN;
      else if (err <= a.c.tol[k] || sc) st = VDR_OK;
      else if (rho == 0.0 || (float)om == 0.f) st = VDR_BREAKDOWN;
      on = st == VDR_NOT_CONVERGED;
      if (!on) {
        a.c.active[k] = 0;
        a.c.status[k] = st;
      }
    }
  }
  const int any = __syncthreads_or(on);
  if (threadIdx.x == 0) {
    a.st->iter += 1;
    if (!any || a.st->iter >= a.st->itmax) a.st->done = 1;
  }
}

// ------------------------------------------------------------ refinement
template <int K>
__device__ __forceinline__ void column_max(const int (&e)[4], int *xexp) {
  __shared__ int sm[K];
  if (threadIdx.x < K) sm[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; c++) atomicMax(&sm[4 * (threadIdx.x % (K / 4)) + c], e[c]);
  __syncthreads();
  if (threadIdx.x < K) atomicMax(xexp + threadIdx.x, sm[threadIdx.x]);
}
__device__ __forceinline__ void ld4d(const double *p, long j, double (&v)[4]) {
  const double2 u = reinterpret_cast<const double2 *>(p)[2 * j];
  const double2 w = reinterpret_cast<const double2 *>(p)[2 * j + 1];
  v[0] = u.x;
  v[1] = u.y;
  v[2] = w.x;
  v[3] = w.y;
}
__device__ __forceinline__ void st4d(double *p, long j, const double (&v)[4]) {
  reinterpret_cast<double2 *>(p)[2 * j] = make_double2(v[0], v[1]);
  reinterpret_cast<double2 *>(p)[2 * j + 1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ unsigned long long magnitude(double d) {
  return (unsigned long long)__double_as_longlong(d) & 0x7fffffffffffffffull;
}

// X = 0 on Dirichlet rows; *nonzero set when any entry is left nonzero; the
// columns' largest exponents.
template <int K>
__global__ void __launch_bounds__(BT, 2) br_mask(const BVec a, const BlockOuter o, double *X,
                                                 int *nonzero) {
  int e[4] = {0, 0, 0, 0};
  bool nz = false;
  ULOOP(j) {
    double v[4];
    ld4d(X, j, v);
    if (a.m[j / (K / 4)]) {
      const double z[4] = {0.0, 0.0, 0.0, 0.0};
      st4d(X, j, z);
    } else {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        nz = nz || magnitude(v[c]) != 0;
        e[c] = max(e[c], df_exp(v[c]));
      }
    }
  }
  if (__any_sync(FULLR, nz) && (threadIdx.x & 31) == 0) atomicOr(nonzero, 1);
  column_max<K>(e, o.xexp);
}

// X += D scale, and the columns' largest exponents.
template <int K>
__global__ void __launch_bounds__(BT, 2) br_update(const BVec a, const BlockOuter o, double *X) {
  const int k0 = 4 * (threadIdx.x % (K / 4));
  double sc[4];
#pragma unroll
  for (int c = 0; c < 4; c++) sc[c] = o.scale[k0 + c];
  int e[4] = {0, 0, 0, 0};
  ULOOP(j) {
    double v[4];
    ld4d(X, j, v);
    const float4 dv = ld4(a.x, j);
#pragma unroll
    for (int c = 0; c < 4; c++) {
      v[c] += df_f2d(f4(dv, c)) * sc[c];
      e[c] = max(e[c], df_exp(v[c]));
    }
    st4d(X, j, v);
  }
  column_max<K>(e, o.xexp);
}

// R = B - A X (A X = 0 unless PROD: the largest |B| alone), the columns'
// largest |R| and |B| as bit patterns (ordered as the magnitudes are, NaN
// above infinity).  The march of br_apply with pairs: a plane's tile is split
// as it is put into shared memory, the column scaled by one power of two;
// what does not fit becomes infinite.  Bound by issue: 27 pair products of 12
// instructions an output, two columns at once.  At 1.08 M nodes and 64 columns
// the element matrices took 3.9 ms, every thread splitting what it gathered
// 2.9, the split tiles 2.3 (waiting for the rows), packed products 2.1, and
// with the next plane's rows copied ahead into shared memory 1.8.
template <int K, bool PROD>
__global__ void __launch_bounds__(PT, 2) br_residual(const BVec a, const BlockRows g,
                                                     const BlockOuter o,
                                                     const double *__restrict__ B,
                                                     const double *__restrict__ X,
                                                     double *__restrict__ R) {
  using T = Tile<K>;
  constexpr int L = T::L, CELLS = T::SX * T::SY, NP = (CELLS * L + PT - 1) / PT;
  extern __shared__ __align__(128) unsigned char stage[];
  float4 *sx = reinterpret_cast<float4 *>(stage);  // [2][cell][hi, lo][lane]
  // the entries that multiply a plane, [2][9 j + c][node], j as in br_rows
  constexpr int NODES = T::TX * T::TY;
  float2 *se = reinterpret_cast<float2 *>(stage + 4 * T::XB);
  const int l = threadIdx.x % L, pair = threadIdx.x / L;
  unsigned long long rm[4] = {0, 0, 0, 0}, bm[4] = {0, 0, 0, 0};
  if (!PROD) {
    ULOOP(j) {
      double v[4];
      ld4d(B, j, v);
#pragma unroll
      for (int c = 0; c < 4; c++) bm[c] = max(bm[c], magnitude(v[c]));
    }
#pragma unroll
    for (int c = 0; c < 4; c++) rm[c] = bm[c];
  } else {
    const int base = 1023 - pair_head(g.nm);
    int shift[4];
#pragma unroll
    for (int c = 0; c < 4; c++) shift[c] = o.xexp[4 * l + c] - base;
    const int pl = g.nax * g.nay;
    const int px = 2 * (pair % (T::TX / 2)), py = pair / (T::TX / 2);
    for (Share w(g); w.template next<T>(g);) {
      const int x0 = w.x0, y0 = w.y0, z0 = w.z0, z1 = w.z1, zb = w.zb, ze = w.ze;
      double v[NP][4];
      const auto load = [&](int z) {
#pragma unroll
        for (int u = 0; u < NP; u++) {
          const int i = pair + u * (PT / L);
          const int x = x0 - 1 + i % T::SX, y = y0 - 1 + i / T::SX;
#pragma unroll
          for (int c = 0; c < 4; c++) v[u][c] = 0.0;
          if (i < CELLS && x >= 0 && x < g.nax && y >= 0 && y < g.nay)
            ld4d(X, (((long)z * g.nay + y) * g.nax + x) * L + l, v[u]);
        }
      };
      const auto store = [&](int z) {
        float4 *st = sx + ((z - zb) & 1) * CELLS * 2 * L;
#pragma unroll
        for (int u = 0; u < NP; u++) {
          const int i = pair + u * (PT / L);
          const float2 q0 = stencil_pair(v[u][0], shift[0]), q1 = stencil_pair(v[u][1], shift[1]);
          const float2 q2 = stencil_pair(v[u][2], shift[2]), q3 = stencil_pair(v[u][3], shift[3]);
          if (i < CELLS) {
            st[2 * i * L + l] = make_float4(q0.x, q1.x, q2.x, q3.x);
            st[(2 * i + 1) * L + l] = make_float4(q0.y, q1.y, q2.y, q3.y);
          }
        }
      };
      const auto fetch_rows = [&](int z) {
        float2 *dst = se + ((z - zb) & 1) * 27 * NODES;
        for (int i = threadIdx.x; i < 27 * NODES; i += PT) {
          const int k = i / NODES, j = k / 9, x = x0 + i % T::TX, y = y0 + i % NODES / T::TX;
          const int zr = z + j - 1;
          const bool in = x < g.nax && y < g.nay && zr >= 0 && zr < g.naz;
          const float2 *src =
              g.S + (in ? (size_t)(9 * (2 - j) + k % 9) * g.N + ((long)zr * g.nay + y) * g.nax + x
                        : 0);
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(tc::smem_u32(dst + i)),
                       "l"(src), "r"(in ? 8 : 0)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      const bool in0 = x0 + px < g.nax && y0 + py < g.nay, in1 = in0 && x0 + px + 1 < g.nax;
      DfAccx2 lo[2][2], mid[2][2], up[2][2];
      const DfAccx2 none{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int u = 0; u < 2; u++)
        lo[u][0] = lo[u][1] = mid[u][0] = mid[u][1] = none;
      __syncthreads();  // the stages of the segment before are read
      fetch_rows(zb);
      load(zb);
      store(zb);
      long n = ((long)zb * g.nay + y0 + py) * g.nax + x0 + px;
      for (int z = zb; z <= ze; z++, n += pl) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (z < ze) {
          fetch_rows(z + 1);
          load(z + 1);
          store(z + 1);
        }
        if (in0) {
          up[0][0] = up[0][1] = up[1][0] = up[1][1] = none;
          const float4 *xs = sx + (((z - zb) & 1) * CELLS + py * T::SX + px) * 2 * L + l;
          const float2 *es = se + ((z - zb) & 1) * 27 * NODES + py * T::TX + px;
#pragma unroll 1
          for (int dy = 0; dy < 3; dy++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const float4 xh = xs[(dy * T::SX + i) * 2 * L];
              const float4 xl = xs[((dy * T::SX + i) * 2 + 1) * L];
#pragma unroll
              for (int u = 0; u < 2; u++) {
                const int dx = i - u;
                if (dx < 0 || dx > 2) continue;
                DfDup e[3];
#pragma unroll
                for (int j = 0; j < 3; j++) {
                  const float2 v = es[(9 * j + 3 * dy + dx) * NODES + u];
                  e[j] = df_dup(Df2{v.x, v.y});
                }
#pragma unroll
                for (int c = 0; c < 2; c++) {
                  const Df2x2 xp{half_of(xh, c), half_of(xl, c)};
                  df_acc2(lo[u][c], e[0], xp);
                  df_acc2(mid[u][c], e[1], xp);
                  df_acc2(up[u][c], e[2], xp);
                }
              }
            }
          }
#pragma unroll 1
          for (int fin = 0; fin < 2; fin++) {
            if (fin == 0 ? z > z0 : (z == g.naz - 1 && z < z1)) {
#pragma unroll
              for (int u = 0; u < 2; u++) {
                if (!(u ? in1 : in0)) continue;
                const long at = ((fin == 0 ? n - pl : n) + u) * L + l;
                double b[4], r[4];
                ld4d(B, at, b);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                  const DfAccx2 &t = lo[u][c / 2];
                  double ax = c & 1 ? df_to_double(t.s.y, t.c.y) : df_to_double(t.s.x, t.c.x);
                  if (!df_scale(ax, shift[c])) ax = ldexp(ax, shift[c]);
                  r[c] = b[c] - ax;
                  bm[c] = max(bm[c], magnitude(b[c]));
                  rm[c] = max(rm[c], magnitude(r[c]));
                }
                st4d(R, at, r);
              }
            }
            if (fin == 0)
#pragma unroll
              for (int u = 0; u < 2; u++)
#pragma unroll
                for (int c = 0; c < 2; c++) {
                  lo[u][c] = mid[u][c];
                  mid[u][c] = up[u][c];
                }
          }
        }
      }
    }
  }
  __shared__ unsigned long long sr[K], sb[K];
  if (threadIdx.x < K) sr[threadIdx.x] = sb[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 4; c++) {
    atomicMax(&sr[4 * l + c], rm[c]);
    atomicMax(&sb[4 * l + c], bm[c]);
  }
  __syncthreads();
  if (threadIdx.x < K) {
    atomicMax(o.rmax + threadIdx.x, sr[threadIdx.x]);
    atomicMax(o.bmax + threadIdx.x, sb[threadIdx.x]);
  }
}

// Biased exponent that scales |d| into [1/2, 1), as frexp gives it.
__device__ __forceinline__ int unit_exp(double d) {
  int e = 0;
  if (d > 0.0 && isfinite(d)) frexp(d, &e);
  return e;
}

// The inner solve's start from the residual R: its FP32 copy scaled by the
// power of two above its largest magnitude, as r, p and rh, with x = 0; the
// column's ||R|| / ||B|| (||B||^2 from the FIRST pass) and ||rh||^2.
template <int K, bool FIRST>
__global__ void __launch_bounds__(BT, 2) br_scale(const BVec a, const BlockOuter o,
                                                  const double *__restrict__ B,
                                                  const double *__restrict__ R) {
  constexpr int NQ = FIRST ? 4 : 2;  // the fourth stays zero
  const int k0 = 4 * (threadIdx.x % (K / 4));
  int er[4], eb[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    er[c] = unit_exp(__longlong_as_double((long long)o.rmax[k0 + c]));
    eb[c] = unit_exp(__longlong_as_double((long long)o.bmax[k0 + c]));
  }
  DfAcc d[NQ][4];
  clear<NQ>(d);
  float4 *rh = reinterpret_cast<float4 *>(a.rh);
  ULOOP(j) {
    double v[4];
    ld4d(R, j, v);
    float f[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const float2 q = stencil_pair(v[c], er[c]);
      f[c] = __fadd_rn(q.x, q.y);
      df_fma_acc(d[0][c], q.x, q.y, q.x, q.y);
      dot_acc(d[1][c], f[c], f[c]);
    }
    const float4 fv = make_float4(f[0], f[1], f[2], f[3]);
    rh[j] = fv;
    st4(a.r, j, fv);
    st4(a.p, j, fv);
    st4(a.x, j, make_float4(0.f, 0.f, 0.f, 0.f));
    if (FIRST) {
      ld4d(B, j, v);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float2 q = stencil_pair(v[c], eb[c]);
        df_fma_acc(d[2 % NQ][c], q.x, q.y, q.x, q.y);
      }
    }
  }
  __shared__ double sm[sum_words(K, NQ, BT)], out[NQ * K];
  if (!col_sums<K, NQ, BT>(d, a, sm, out) || threadIdx.x >= K) return;
  const int k = threadIdx.x;
  const double rmax = __longlong_as_double((long long)o.rmax[k]);
  const double bmax = __longlong_as_double((long long)o.bmax[k]);
  const int e_r = unit_exp(rmax), e_b = unit_exp(bmax);
  if (FIRST) o.bb[k] = out[(2 * K) % (NQ * K) + k];
  o.scale[k] = ldexp(1.0, e_r);
  double err;
  if (!(rmax == rmax) || isinf(rmax)) err = rmax + rmax;  // NaN / inf propagate
  else if (rmax == 0.0) err = 0.0;
  else if (!(bmax > 0.0)) err = INFINITY;  // zero column, nonzero R
  else err = ldexp(sqrt(out[k] / o.bb[k]), e_r - e_b);
  o.err[k] = err;
  a.c.bnrm2[k] = a.c.rho[k] = out[K + k];
}

// Which columns iterate: those whose inner tolerance and outer residual are
// not met yet (x = 0, so the inner residual is the right-hand side).
__global__ void br_begin(const BVec a) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  const int k = threadIdx.x;
  if (k < a.K) {
    const double bb = a.c.bnrm2[k], err = bb > 0.0 ? 1.0 : 0.0;
    a.c.alpha[k] = 1.0;
    a.c.omega[k] = 1.0;
    a.c.sconv[k] = 0;
    a.c.err[k] = err;
    const int on = (bb > 0.0 && err > a.c.tol[k] && !(a.outer_err[k] <= a.outer_tol)) ? 1 : 0;
    a.c.active[k] = on;
    a.c.status[k] = on ? VDR_NOT_CONVERGED : VDR_OK;
    if (on) any = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    a.st->iter = 0;
    a.st->done = any ? 0 : 1;
  }
}

// Tiles and shared memory of the products with K columns; two blocks an SM.
template <int K>
cudaError_t plan(const Handle &h, BlockRows *g) {
  using T = Tile<K>;
  const cudaFuncAttribute smem = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(br_apply<K, false>, smem, T::PRODUCT)) ||
      (e = cudaFuncSetAttribute(br_apply<K, true>, smem, T::PRODUCT)) ||
      (e = cudaFuncSetAttribute(br_residual<K, true>, smem, T::RESIDUAL)))
    return e;
  g->nxt = (h.nax + T::TX - 1) / T::TX;
  g->nyt = (h.nay + T::TY - 1) / T::TY;
  const long planes = (long)g->nxt * g->nyt * h.naz;
  g->grid = (int)std::min<long>((planes + 3) / 4, 2L * device_sm_count());
  return cudaGetLastError();
}

template <int K>
bool make_maps(const BlockRows &g, const float *x, Maps *m) {
  using T = Tile<K>;
  return make_node_map(&m->x, x, K, g.nax, g.nay, g.naz, T::SX, T::SY) &&
         make_node_map(&m->rows, reinterpret_cast<const float *>(g.rows), 28, g.nax, g.nay, g.naz,
                       T::TX, T::TY);
}

}  // namespace

cudaError_t launch_ring_timeout(int *err, int bit, long long limit, cudaStream_t s) {
  ring_timeout_kernel<<<1, 32, 0, s>>>(err, bit, limit);
  count_launches(1);
  return cudaGetLastError();
}

// The rows of the current operator and the inverse diagonal in h.dinv32;
// false where the element-wise form stays: another numbering, store or
// scatter, a variant asked for by name, no room for the rows.
bool block_rows_usable(Handle &h, int K, BlockRows *g) {
  if (h.block_tma || !h.block_tile || h.blk_tc_mode >= 0) return false;
  if (ensure_stencil(h) || h.st_state != 1) return false;
  if (!h.block_err) {
    if (cudaMalloc(&h.block_err, sizeof(int))) return false;
    cudaMemsetAsync(h.block_err, 0, sizeof(int), h.stream);
  }
  if ((long)h.N * K >= (1l << 31) || !block_tc_supported(h)) return false;
  const size_t words = 28 * (size_t)h.N;
  if (h.br_words < words) {
    cudaFree(h.br_rows);
    h.br_rows = nullptr;
    h.br_words = 0;
    if (!h.rows_room || cudaMalloc(&h.br_rows, sizeof(float) * words)) {
      cudaGetLastError();
      return false;
    }
    h.br_words = words;
  }
  const int grid = (int)std::min<long>((h.N + 255L) / 256, (long)device_sm_count() * 16);
  br_rows<<<grid, 256, 0, h.stream>>>(h.st_S, h.dinv32, h.N, h.nax, h.nax * h.nay, h.br_rows);
  count_launches(1);
  g->rows = reinterpret_cast<const float4 *>(h.br_rows);
  g->S = h.st_S;
  g->nm = h.st_nm + NM_LEAD;
  g->N = h.N;
  g->nax = h.nax;
  g->nay = h.nay;
  g->naz = h.naz;
  g->err = h.block_err;
  return !(K == 16 ? plan<16>(h, g) : K == 32 ? plan<32>(h, g) : plan<64>(h, g));
}

#define VDR_BY_K(CALL)      \
  do {                      \
    if (a.K == 16) {        \
      constexpr int K = 16; \
      CALL;                 \
    } else if (a.K == 32) { \
      constexpr int K = 32; \
      CALL;                 \
    } else {                \
      constexpr int K = 64; \
      CALL;                 \
    }                       \
  } while (0)

cudaError_t block_rows_mask(const BVec &a, const BlockOuter &o, double *X, int *nonzero, int grid,
                            cudaStream_t s) {
  VDR_BY_K((br_mask<K><<<grid, BT, 0, s>>>(a, o, X, nonzero)));
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t block_rows_residual(const BVec &a, const BlockRows &g, const BlockOuter &o,
                                const double *B, const double *X, double *R, bool zero_x,
                                bool first, int grid, cudaStream_t s) {
  if (zero_x) VDR_BY_K((br_residual<K, false><<<g.grid, PT, 0, s>>>(a, g, o, B, X, R)));
  else
    VDR_BY_K((br_residual<K, true>
              <<<g.grid, PT, Tile<K>::RESIDUAL, s>>>(a, g, o, B, X, R)));
  const double *src = zero_x ? B : R;
  if (first) VDR_BY_K((br_scale<K, true><<<grid, BT, 0, s>>>(a, o, B, src)));
  else VDR_BY_K((br_scale<K, false><<<grid, BT, 0, s>>>(a, o, B, src)));
  count_launches(2);
  return cudaGetLastError();
}

cudaError_t block_rows_begin(const BVec &a, cudaStream_t s) {
  br_begin<<<1, 64, 0, s>>>(a);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t block_rows_iterations(const BVec &a, const BlockRows &g, int count, int grid,
                                  cudaStream_t s) {
  Maps mp, ms;
  bool made = false;
  VDR_BY_K((made = make_maps<K>(g, a.p, &mp) && make_maps<K>(g, a.s, &ms)));
  if (!made) return cudaErrorInvalidValue;
  for (int it = 0; it < count; it++) {
    VDR_BY_K((br_apply<K, false><<<g.grid, PT, Tile<K>::PRODUCT, s>>>(a, g, mp)));
    VDR_BY_K((br_s<K><<<grid, BT, 0, s>>>(a)));
    VDR_BY_K((br_apply<K, true><<<g.grid, PT, Tile<K>::PRODUCT, s>>>(a, g, ms)));
    VDR_BY_K((br_xp<K><<<grid, BT, 0, s>>>(a)));
  }
  return cudaGetLastError();
}

cudaError_t block_rows_update(const BVec &a, const BlockOuter &o, double *X, int grid,
                              cudaStream_t s) {
  VDR_BY_K((br_update<K><<<grid, BT, 0, s>>>(a, o, X)));
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace vdr
