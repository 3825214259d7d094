// meet.cuh -- meetings of all CTAs of a resident launch (one cluster, or a
// cooperative grid) that leave grid-wide sums behind.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "reduce.cuh"
#include "vdr_internal.h"

namespace vdr {

constexpr long long RES_LIMIT = 2000000000LL;  // ~1 s of clocks
constexpr int RES_NB = 5;                      // at most 32 RES_NB CTAs in a grid
constexpr int CLUSTER_MAX = 16;

enum { CLUSTER, IN_REGS, IN_SMEM };
// BiCGStab's partial sums and their places:
// (s,s) (rh,s) | (t,s) (t,t) (rh,t) | (r,r) (w,p)
enum { AT_C = 0, AT_D = 2, AT_A = 5, SLOTS = 7 };

struct MeetArgs {
  double *part;     // [SLOTS][gridDim]; behind them [3][gridDim] largest exponents
  unsigned *bar;    // arrivals, zero at launch; the next word: where a wait ran out
  long long limit;  // clocks that a wait may take
  __device__ int *ipart() const { return reinterpret_cast<int *>(part + SLOTS * 32 * RES_NB); }
};

struct ResShared {
  double s[SLOTS][32];  // this CTA's sums, per warp
  int e[3][32];
  double tot[6];  // totals, or scalars made of them
  int etot[2];
  int ok;
};

// ---- thread-block clusters
__device__ __forceinline__ void cluster_meet() {
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
          : "memory");
}
__device__ __forceinline__ unsigned cluster_addr(const void *p, int cta) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(cta));
  return a;
}
__device__ __forceinline__ double cluster_f64(unsigned a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int cluster_s32(unsigned a) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 cluster_pair(unsigned a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a)
               : "memory");
  return v;
}

// A meeting of all CTAs.  Each leaves its sums of Q quantities at place SLOT
// (and NE largest exponents at place ES); what any thread wrote before is
// visible to all after.  Then the totals of the R quantities from place READ
// on (R = 0: none) are in sh.tot and the largest exponents in sh.etot, and
// `scalars` runs on warp 0 with them there, its results in sh for all
// threads.  No place is written again before a meeting that follows its
// reads.
template <int MODE, int T, int Q, int NE, int R, int SLOT, int READ, int ES, typename F>
__device__ __forceinline__ bool meet(ResShared &sh, const MeetArgs &a, const double (&v)[Q],
                                     const int (&em)[NE > 0 ? NE : 1], unsigned &target,
                                     F scalars) {
  constexpr int nw = T / 32;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int B = (int)gridDim.x;
  const double f = warp_sums<Q>(v, lane);
  if ((lane & 7) == 0 && (lane >> 3) < Q) sh.s[SLOT + (lane >> 3)][w] = f;
#pragma unroll
  for (int k = 0; k < NE; k++) {
    const int e = __reduce_max_sync(FULLR, em[k]);
    if (lane == 0) sh.e[ES + k][w] = e;
  }
  constexpr int RP = R > 0 ? R : 1, R4 = RP < 4 ? RP : 4;
  double tot[RP];
  int etot[NE > 0 ? NE : 1] = {0};
  if (MODE == CLUSTER) {
    cluster_meet();
    if (R == 0 && NE == 0) return true;
    if (w == 0) {  // all warps' sums of all CTAs, every load before the adds
      constexpr int NI = (CLUSTER_MAX * nw + 31) / 32;
      double in[NI][RP];
      int ein[NI][NE > 0 ? NE : 1];
#pragma unroll
      for (int i = 0; i < NI; i++) {
        const int j = lane + 32 * i, c = min(j / nw, B - 1), u = j % nw;
        const unsigned at = cluster_addr(&sh.s[READ][u], c);
        if (R > 0)
#pragma unroll
          for (int k = 0; k < RP; k++)
            in[i][k] = cluster_f64(at + (unsigned)(k * sizeof sh.s[0]));
#pragma unroll
        for (int k = 0; k < NE; k++) ein[i][k] = cluster_s32(cluster_addr(&sh.e[ES + k][u], c));
      }
#pragma unroll
      for (int k = 0; k < RP; k++) tot[k] = 0.0;
#pragma unroll
      for (int i = 0; i < NI; i++) {
        const bool mine = lane + 32 * i < B * nw;
        if (R > 0 && (i == 0 || 32 * i < B * nw))
#pragma unroll
          for (int k = 0; k < RP; k++) tot[k] += mine ? in[i][k] : 0.0;
#pragma unroll
        for (int k = 0; k < NE; k++) etot[k] = max(etot[k], ein[i][k]);
      }
    }
  } else {
    target += gridDim.x;
    __syncthreads();
    if (w == 0) {
      const int q = lane >> 3, sub = lane & 7;
      double c = 0.0;
      for (int k = sub; k < nw; k += 8) c += sh.s[SLOT + (q < Q ? q : 0)][k];
      c = fold8(c);
      if (sub == 0 && q < Q) __stcg(a.part + (size_t)(SLOT + q) * B + blockIdx.x, c);
#pragma unroll
      for (int k = 0; k < NE; k++) {
        const int e = __reduce_max_sync(FULLR, lane < nw ? sh.e[ES + k][lane] : 0);
        if (lane == 0) __stcg(a.ipart() + (size_t)(ES + k) * B + blockIdx.x, e);
      }
      __syncwarp();
      if (lane == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
      __syncwarp();
      // the whole warp polls: with one lane polling, what followed ran split
      // (13 us more per iteration at 145 CTAs)
      const long long t0 = clock64();
      bool met, late = false;
      const auto arrived = [&]() {
        unsigned seen;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
        return (int)(seen - target) >= 0;
      };
      do {
        met = arrived();
        late = clock64() - t0 > a.limit;
      } while (!__all_sync(FULLR, met || late));
      if (!met) met = arrived();  // a pause of this CTA is not another's delay
      if (lane == 0) {
        sh.ok = met;
        if (!met) *(volatile unsigned *)(a.bar + 1) = 1u;
      }
      if (R > 0) {
        double in[RES_NB][RP];  // every load before the first add
#pragma unroll
        for (int i = 0; i < RES_NB; i++)
#pragma unroll
          for (int k = 0; k < RP; k++)
            in[i][k] = __ldcg(a.part + (size_t)(READ + k) * B + min(lane + 32 * i, B - 1));
#pragma unroll
        for (int k = 0; k < RP; k++) tot[k] = lane < B ? in[0][k] : 0.0;
#pragma unroll
        for (int i = 1; i < RES_NB; i++)
          if (32 * i < B)
#pragma unroll
            for (int k = 0; k < RP; k++) tot[k] += lane + 32 * i < B ? in[i][k] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < NE; k++)
#pragma unroll
        for (int i = 0; i < RES_NB; i++)
          etot[k] =
              max(etot[k], __ldcg(a.ipart() + (size_t)(ES + k) * B + min(lane + 32 * i, B - 1)));
    }
  }
  if (w == 0) {
    if (R > 0) {
      double u[R4];
#pragma unroll
      for (int k = 0; k < R4; k++) u[k] = tot[k];
      const double g = warp_sums<R4>(u, lane);
      if ((lane & 7) == 0 && (lane >> 3) < R4) sh.tot[lane >> 3] = g;
      if (R > 4) {
        const double u1[1] = {tot[RP - 1]};
        const double g1 = warp_sums<1>(u1, lane);
        if (lane == 0) sh.tot[4] = g1;
      }
    }
#pragma unroll
    for (int k = 0; k < NE; k++) {
      const int e = __reduce_max_sync(FULLR, etot[k]);
      if (lane == 0) sh.etot[k] = e;
    }
    __syncwarp();
    if (R > 0) scalars(lane);
  }
  __syncthreads();
  return MODE == CLUSTER || sh.ok != 0;
}

inline MeetArgs meet_args(const Handle &h) {
  return MeetArgs{h.partials, &h.st->bar_count, RES_LIMIT};
}
// No arrivals and nobody late.
inline cudaError_t meet_reset(Handle &h, cudaStream_t s) {
  static_assert(offsetof(KState, late) == offsetof(KState, bar_count) + sizeof(unsigned), "one fill");
  return cudaMemsetAsync(&h.st->bar_count, 0, 2 * sizeof(unsigned), s);
}

}  // namespace vdr
