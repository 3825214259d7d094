// stencil.cu -- assembly of the 27-point operator (stencil.cuh) from the
// double-float element store, and its plain applies.
#include "stencil.cuh"

#include <algorithm>

namespace vdr {
namespace {

constexpr int slot_of(int a, int b, int c) {
  return 4 * c + (b ? (a ? 2 : 3) : (a ? 1 : 0));
}
constexpr int slot_x(int s) { return ((s + 1) & 2) ? 1 : 0; }
constexpr int slot_y(int s) { return (s & 2) ? 1 : 0; }
constexpr int slot_z(int s) { return (s & 4) ? 1 : 0; }

// acc += (h, l), the error terms gathered in acc.c.
__device__ __forceinline__ void acc_pair(DfAcc &acc, float h, float l) {
  df_acc_add(acc, Df2{h, l});
}

// Row n of P A P: the sum of its row in each of the up to eight elements
// around it, TwoSum per entry (error ~2^-47 of the largest element entry, as
// the sums of an element-wise apply).  One thread per node: an element's
// row i is read by exactly one thread, so the store is read once (512 E
// bytes) and 220 N written: 1.23 ms at 8.4M elements (5.0 TB/s).  The mesh's
// elements lie from e0 on in the store of E, `l` is the node's number in it.
// Returns the largest entry's magnitude bits.
__device__ __forceinline__ unsigned assemble_node(const float4 *__restrict__ Ahi,
                                              const float4 *__restrict__ Alo,
                                              const unsigned char *__restrict__ emask, int E,
                                              long e0, int nax, int nay, int naz, unsigned l,
                                              long n, long N, float2 *S, unsigned *nm) {
  const unsigned r = l / (unsigned)nax;
  const int i = (int)(l - r * (unsigned)nax);
  const int k = (int)(r / (unsigned)nay), j = (int)(r - (unsigned)k * (unsigned)nay);
  DfAcc acc[27];
#pragma unroll
  for (int t = 0; t < 27; t++) acc[t] = DfAcc{0.f, 0.f};
  unsigned m = 0u;
#pragma unroll
  for (int e = 0; e < 8; e++) {
    const int ex = (e & 1) - 1, ey = ((e >> 1) & 1) - 1, ez = (e >> 2) - 1;
    const int ei = i + ex, ej = j + ey, ek = k + ez;
    if (ei < 0 || ei >= nax - 1 || ej < 0 || ej >= nay - 1 || ek < 0 || ek >= naz - 1)
      continue;
    const long p = e0 + ei + (long)(nax - 1) * (ej + (long)(nay - 1) * ek);
    const int own = slot_of(-ex, -ey, -ez);
    const unsigned dm = __ldg(emask + p);
    if ((dm >> own) & 1u) continue;  // a Dirichlet row
    float4 h[2], lo[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      h[q] = __ldcs(Ahi + (size_t)(2 * own + q) * E + p);
      lo[q] = __ldcs(Alo + (size_t)(2 * own + q) * E + p);
    }
#pragma unroll
    for (int s = 0; s < 8; s++) {
      const int t = 9 * (slot_z(s) + ez + 1) + 3 * (slot_y(s) + ey + 1) + slot_x(s) + ex + 1;
      const float4 &hq = h[s >> 2], &lq = lo[s >> 2];
      const int w = s & 3;
      const float hv = w == 0 ? hq.x : w == 1 ? hq.y : w == 2 ? hq.z : hq.w;
      const float lv = w == 0 ? lq.x : w == 1 ? lq.y : w == 2 ? lq.z : lq.w;
      if (!((dm >> s) & 1u)) {
        acc_pair(acc[t], hv, lv);
        m |= 1u << t;
      }
    }
  }
  unsigned big = 0u;
#pragma unroll
  for (int t = 0; t < 27; t++) {
    const Df2 a = df_norm(acc[t]);
    S[(size_t)t * N + n] = make_float2(a.h, a.l);
    big = max(big, __float_as_uint(a.h) & 0x7fffffffu);
  }
  nm[n] = m;
  return big;
}

__device__ __forceinline__ void raise_top(unsigned big, unsigned *top) {
  const unsigned e = __reduce_max_sync(0xffffffffu, big) >> 23;
  if ((threadIdx.x & 31) == 0 && e > *(volatile unsigned *)top) atomicMax(top, e);
}

__global__ void __launch_bounds__(256, 2) stencil_assemble(
    const float4 *__restrict__ Ahi, const float4 *__restrict__ Alo,
    const unsigned char *__restrict__ emask, int nax, int nay, int naz, float2 *S,
    unsigned *nm) {
  unsigned big = 0u;
  const int E = (nax - 1) * (nay - 1) * (naz - 1), N = nax * nay * naz;
  for (long n = (long)blockIdx.x * blockDim.x + threadIdx.x; n < N;
       n += (long)gridDim.x * blockDim.x)
    big = max(big, assemble_node(Ahi, Alo, emask, E, 0, nax, nay, naz, (unsigned)n, n, N, S, nm));
  raise_top(big, nm - 1);
}

// The same for many meshes side by side (one row of blocks per mesh).
__global__ void __launch_bounds__(256, 2) stencil_assemble_meshes(
    const float4 *__restrict__ Ahi, const float4 *__restrict__ Alo,
    const unsigned char *__restrict__ emask, int E, long N,
    const SegMesh *__restrict__ meshes, float2 *S, unsigned *nm) {
  unsigned big = 0u;
  const SegMesh g = meshes[blockIdx.y];
  const int count = g.nax * g.nay * g.naz;
  for (int l = (int)(blockIdx.x * blockDim.x + threadIdx.x); l < count;
       l += (int)(gridDim.x * blockDim.x))
    big = max(big, assemble_node(Ahi, Alo, emask, E, g.e0, g.nax, g.nay, g.naz, (unsigned)l,
                                 g.n0 + (long)l, N, S, nm));
  raise_top(big, nm - 1);
}

// y += A x or A^T x, any FP64 x, for the products of solvers that keep FP64
// vectors (GCR, a preconditioned BiCGStab, first residuals) where another
// solve has formed the rows (products_on_rows).  Here every thread splits its
// 27 gathered values and scales each plane by itself, which makes it bound by
// instruction issue: 95 / 718 us at 1.08 / 8.5 M nodes where the element-wise
// apply takes 105 / 773; the Krylov iterations split once per node.  Rows are
// not formed for it: their sum (160 us, 1.23 ms) costs what 15 products save
// (GCR of one to three iterations on a new operator took up to 10 per cent
// longer).  A caller's own applies stay element-wise also because FP64 sums
// over the elements are closer to the exact product (3.5e-15 against 5.9e-15
// relative, random input).
template <bool TRANS, bool KEEP>
__global__ void __launch_bounds__(256, 4) stencil_apply(const StencilView v,
                                                        const double *__restrict__ x,
                                                        double *__restrict__ y,
                                                        const int *skip, const int *skip2) {
  if (skip && *(volatile const int *)skip) return;
  if (skip2 && *(volatile const int *)skip2) return;
  for (long n = (long)blockIdx.x * blockDim.x + threadIdx.x; n < v.N;
       n += (long)gridDim.x * blockDim.x) {
    y[n] += stencil_row<TRANS, KEEP>(v, n, x);
  }
}

}  // namespace

StencilView stencil_view(const Handle &h) {
  StencilView v;
  v.S = h.st_S;
  v.nm = h.st_nm + NM_LEAD;
  v.N = h.N;
  v.nax = h.nax;
  v.pl = h.nax * h.nay;
  return v;
}

bool stencil_keep(const Handle &h) { return 220.0 * h.N < 80.0e6; }

bool stencil_ready(const Handle &h) {
  return h.st_state == 1 && h.apply_mode == VDR_APPLY_STORED && !h.apply_fp32 &&
         !h.gate_active && h.storage == VDR_STORE_DF;
}

// Current rows, and a mesh on which a product with them is the faster one:
// 18,513 nodes 57.5 us an iteration of GCR by rows, 56.7 by elements; 100,096
// nodes 92.4 and 93.0.
bool products_on_rows(const Handle &h) { return h.N >= 65536 && stencil_ready(h); }

// Whether a caller records on the stream: what it replays later is to follow
// the operator as it is then, and rows are summed anew by solves and applies
// that are called, not replayed.  The element matrices are rebuilt in place.
bool foreign_capture(const Handle &h, cudaStream_t s) {
  if (h.own_capture) return false;
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s, &c) != cudaSuccess || c != cudaStreamCaptureStatusNone;
}

// Room for the rows of the handle's nodes and for `len` pairs in *x (its
// present length in *have; a new one is not zeroed).  False where the device
// has no room for them: the element-wise apply stays.
static bool row_storage(Handle &h, float2 **x, size_t *have, size_t len) {
  const size_t N = (size_t)h.N;
  const bool rows = N > h.st_rows, vec = len > *have;
  if (!rows && !vec) return true;
  if (rows) {
    cudaFree(h.st_S);
    cudaFree(h.st_nm);
    h.st_S = nullptr;
    h.st_nm = nullptr;
    h.st_rows = 0;
  }
  if (vec) {
    cudaFree(*x);
    *x = nullptr;
    *have = 0;
    h.st_nax = 0;  // its pads are to be zeroed
  }
  size_t free_b = 0, total_b = 0;
  if (h.rows_room && cudaMemGetInfo(&free_b, &total_b) == cudaSuccess &&
      (rows ? 220 * N : 0) + (vec ? sizeof(float2) * len : 0) <= free_b / 2 &&
      (!rows || (!cudaMalloc(&h.st_S, sizeof(float2) * 27 * N) &&
                 !cudaMalloc(&h.st_nm, sizeof(unsigned) * (NM_LEAD + N)))) &&
      (!vec || !cudaMalloc(x, sizeof(float2) * len))) {
    if (rows) h.st_rows = N;
    if (vec) *have = len;
    return true;
  }
  cudaGetLastError();
  cudaFree(h.st_S);
  cudaFree(h.st_nm);
  cudaFree(*x);
  h.st_S = nullptr;
  h.st_nm = nullptr;
  *x = nullptr;
  *have = h.st_rows = 0;
  h.st_state = -1;
  h.seg_rows = false;  // they were these rows
  return false;
}

cudaError_t take_memory(Handle &h, void **p, size_t bytes) {
  const bool held = h.st_S || h.hr_H || h.br_rows;
  cudaError_t e = cudaErrorMemoryAllocation;
  if ((h.other_room || !held) && !(e = cudaMalloc(p, bytes))) return cudaSuccess;
  *p = nullptr;
  if (!held) return e;
  cudaGetLastError();
  cudaFree(h.st_S);
  cudaFree(h.st_nm);
  cudaFree(h.st_x);
  cudaFree(h.seg_x);
  h.st_S = h.st_x = h.seg_x = nullptr;
  h.st_nm = nullptr;
  h.st_rows = h.st_len = 0;
  h.st_nax = 0;
  h.st_state = -1;
  h.seg_rows = false;
  cudaFree(h.hr_H);
  cudaFree(h.hr_e);
  cudaFree(h.hr_vec);
  if (h.hr_graph) cudaGraphExecDestroy(h.hr_graph);
  h.hr_H = nullptr;
  h.hr_e = nullptr;
  h.hr_vec = nullptr;
  h.hr_graph = nullptr;
  h.hr_state = -1;
  cudaFree(h.br_rows);
  h.br_rows = nullptr;
  h.br_words = 0;
  if ((e = cudaMalloc(p, bytes))) *p = nullptr;
  return e;
}

cudaError_t ensure_stencil(Handle &h) {
  if (h.st_state != 0 || !h.op64_valid || h.apply_mode != VDR_APPLY_STORED ||
      h.storage != VDR_STORE_DF || h.opt.scatter != VDR_SCATTER_AUTO || h.perm_d || !h.Ahi ||
      !h.emask || h.nax < 2 || h.nay < 2 || h.naz < 2)
    return cudaSuccess;
  const size_t N = (size_t)h.N, len = 2 * (N + 2 * stencil_pad(h));
  if (!row_storage(h, &h.st_x, &h.st_len, len)) return cudaSuccess;
  cudaError_t e;
  // the pads lie before, between and behind the vectors: where they lie
  // depends on the strides and on N, and their zeros meet other planes'
  // entries (A^T) or a stored infinity (0 x inf) when they are not zero
  if (h.st_nax != h.nax || h.st_pl != h.nax * h.nay || h.st_n != h.N) {
    if ((e = cudaMemsetAsync(h.st_x, 0, sizeof(float2) * h.st_len, h.stream))) return e;
    h.st_nax = h.nax;
    h.st_pl = h.nax * h.nay;
    h.st_n = h.N;
  }
  const long need = (h.N + 255L) / 256;
  const int grid = (int)std::min<long>(need, (long)device_sm_count() * 32);
  unsigned *nm = h.st_nm + NM_LEAD;
  if ((e = cudaMemsetAsync(nm - 1, 0, sizeof(unsigned), h.stream))) return e;
  stencil_assemble<<<grid, 256, 0, h.stream>>>(h.Ahi, h.Alo, h.emask, h.nax, h.nay, h.naz,
                                               h.st_S, nm);
  count_launches(1);
  e = cudaGetLastError();
  if (!e) h.st_state = 1;
  return e;
}

cudaError_t ensure_segment_rows(Handle &h) {
  if (h.seg_rows || !h.seg_canonical || !h.op64_valid ||
      h.apply_mode != VDR_APPLY_STORED || h.storage != VDR_STORE_DF ||
      h.opt.scatter != VDR_SCATTER_AUTO || h.perm_d || !h.Ahi || h.st_state < 0)
    return cudaSuccess;
  cudaError_t e;
  if (!h.emask && (e = cudaMalloc(&h.emask, (size_t)h.E))) return e;
  size_t have = h.seg_x ? 2 * h.seg_pairs : 0;
  const bool fresh = have == 0;
  if (!row_storage(h, &h.seg_x, &have, 2 * h.seg_pairs)) return cudaSuccess;
  if (fresh && (e = cudaMemsetAsync(h.seg_x, 0, sizeof(float2) * have, h.stream))) return e;
  if ((e = launch_element_masks(h))) return e;
  const int per = (int)std::max<long>(1, std::min<long>(64, (h.seg_largest + 255) / 256));
  unsigned *nm = h.st_nm + NM_LEAD;
  if ((e = cudaMemsetAsync(nm - 1, 0, sizeof(unsigned), h.stream))) return e;
  stencil_assemble_meshes<<<dim3((unsigned)per, (unsigned)(h.seg_off.size() - 1)), 256, 0,
                            h.stream>>>(h.Ahi, h.Alo, h.emask, h.E, h.N, h.seg_mesh, h.st_S,
                                        nm);
  count_launches(1);
  if (!(e = cudaGetLastError())) h.seg_rows = true;
  return e;
}

cudaError_t launch_stencil_apply(const Handle &h, bool transpose, const double *x, double *y,
                                 const int *skip, const int *skip2, cudaStream_t s) {
  const StencilView v = stencil_view(h);
  const bool keep = stencil_keep(h);
  const auto kern = transpose ? (keep ? stencil_apply<true, true> : stencil_apply<true, false>)
                              : (keep ? stencil_apply<false, true> : stencil_apply<false, false>);
  kern<<<(unsigned)((h.N + 255L) / 256), 256, 0, s>>>(v, x, y, skip, skip2);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace vdr
