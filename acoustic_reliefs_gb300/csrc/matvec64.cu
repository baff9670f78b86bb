// The FP64 H-matrix's matvec: the three passes of matvec.cu (dot, reduce, gather) over the same segments.
//
// Bound by the FP64 pipe, not by memory: GB300 runs two FP64 lanes per clock and SM, so an element (four
// multiply-adds, 16 bytes) takes 3 times as long to compute as to read, a warp instruction holds a
// scheduler's pipe for 64 clocks, and lanes without an element cost as much as those with one. Leaves hold 16 to 32
// elements (or their doubles), so lanes laid along a column's rows were a third empty and added
// up over shuffles. Here the dot pass gives a lane a whole column (up to 32 rows of it), and the gather
// pass gives a thread a row and every G-th column, G = 256 / R groups, which reads a segment as one
// contiguous stream. At 64 clocks an instruction a few warps hide the loads, so these go from global
// memory to registers. 5280-triangle relief, 2 kHz (170 MB): dot 107 -> 36 us, gather 128 ->
// 68 us; 1280-triangle sphere in 16 leaves: gather 92 -> 19 us. The CTAs per leaf (up to 8, where the
// leaves alone are fewer than four per SM) are what the sphere gains from.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "internal.h"
#include "launch.cuh"
#include "segstream.cuh"

namespace ac3d {

namespace cg = cooperative_groups;

namespace {
constexpr int kDotThreads = 128, kGatherThreads = 256;
constexpr int kMaxRows = 256;  // the largest leaf
}  // namespace

__device__ __forceinline__ void mac64(double& re, double& im, const cd& a, const cd& z) {
  re = fma(a.re, z.re, re);
  re = fma(-a.im, z.im, re);
  im = fma(a.re, z.im, im);
  im = fma(a.im, z.re, im);
}

// p[kptr[leaf] + k] = sum over the leaf's rows of S[k][row] x[row]. G lanes per column (1 up to 32
// rows, so that a lane has at most 32), gridDim.y CTAs per leaf, whose warps take 32 / G columns in turn.
template <int G>
__global__ void __launch_bounds__(kDotThreads, 6) dot64_kernel(SegView V, const cd* __restrict__ lrseg,
                                                               const cd* __restrict__ x, cd* __restrict__ p,
                                                               const int* __restrict__ done) {
  __shared__ cd xs[kMaxRows];
  const int leaf = V.order[blockIdx.x];
  const int ls = V.leaf_start[leaf], R = V.leaf_start[leaf + 1] - ls;
  const int k0 = V.b_kptr[leaf], K = V.b_kptr[leaf + 1] - k0;
  grid_dep_wait();
  grid_dep_launch();
  const bool skip = done && *(volatile const int*)done;
  for (int r = threadIdx.x; r < R; r += kDotThreads) xs[r] = x[ls + r];
  if (__syncthreads_or(skip)) return;
  const int lane = threadIdx.x & 31, g = lane % G;
  const cd* seg = lrseg + V.b_seg[leaf];
  constexpr int CW = 32 / G, U = 4;
  const int warp = blockIdx.y * (kDotThreads / 32) + (threadIdx.x >> 5), nw = gridDim.y * (kDotThreads / 32);
  for (int c0 = warp * CW; c0 < K; c0 += nw * CW) {
    const int c = c0 + lane / G;
    const cd* col = seg + (long long)min(c, K - 1) * R;
    double re[2] = {0, 0}, im[2] = {0, 0};
    cd a[U];
#pragma unroll
    for (int u = 0; u < U; u++) a[u] = col[min(g + u * G, R - 1)];
    for (int r0 = g; r0 < R; r0 += U * G) {
      cd b[U];
#pragma unroll
      for (int u = 0; u < U; u++) b[u] = col[min(r0 + (U + u) * G, R - 1)];
#pragma unroll
      for (int u = 0; u < U; u++)
        if (r0 + u * G < R) mac64(re[u & 1], im[u & 1], a[u], xs[r0 + u * G]);
#pragma unroll
      for (int u = 0; u < U; u++) a[u] = b[u];
    }
    double sr = re[0] + re[1], si = im[0] + im[1];
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (g == 0 && c < K) p[k0 + c] = cd(sr, si);
  }
}

// Thread (group g, row r) of a segment's columns g, g + G, ... of steps [s0, s1)
__device__ __forceinline__ void gather_steps(double& re, double& im, const cd* __restrict__ seg, int K,
                                             const int* __restrict__ idx, const cd* __restrict__ z, int R, int G,
                                             int g, int tid, int s0, int s1) {
  constexpr int U = 4;
  for (int s = s0; s < s1; s += U) {
    cd a[U], v[U];
    int j[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int c = min((s + u) * G + g, K - 1);
      j[u] = max(idx[c], 0);  // padding columns are zero and take any multiplier
      a[u] = seg[(long long)c * R + tid];
    }
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = z[j[u]];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (s + u < s1 && (s + u) * G + g < K) mac64(re, im, a[u], v[u]);
  }
}

// y[leaf rows] = -x/2 + S_A x[a_idx] + S_B t[b_idx], or b - that, with the optional dot partials of
// seg_gather_persist_kernel. A cluster of CTAs per leaf shares its columns; the first one adds their row sums in
// order and finishes the leaf. The near part runs before the wait for the reduce pass.
__global__ void __launch_bounds__(kGatherThreads, 3) gather64_kernel(
    SegView V, int nleaf, const cd* __restrict__ near, const cd* __restrict__ lrseg, const cd* __restrict__ t,
    const cd* __restrict__ x, cd* __restrict__ y, const cd* __restrict__ bminus, const cd* __restrict__ dot_a,
    const cd* __restrict__ dot_b, double* partials, double* red5, unsigned* ticket, const int* __restrict__ done) {
  constexpr int W = kGatherThreads / 32;
  __shared__ cd part[kGatherThreads];
  __shared__ cd rows[kMaxRows];
  __shared__ double sdot[W][5];
  __shared__ bool s_last;
  __shared__ int s_skip;
  grid_dep_launch();
  const cg::cluster_group cl = cg::this_cluster();
  const int S = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int leaf = V.order[blockIdx.x / S];
  const int ls = V.leaf_start[leaf], R = V.leaf_start[leaf + 1] - ls;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // the flag may be set while this kernel runs: a thread that sees it skips its sums, but not the barriers,
  // and its cluster writes nothing
  const bool skip = done && *(volatile const int*)done;
  const int G = kGatherThreads / R, g = tid / R, r = tid - g * R;
  double re = 0, im = 0;
  const int ak = V.a_kptr[leaf], ac = V.a_kptr[leaf + 1] - ak, na = (ac + G - 1) / G;
  if (!skip && g < G && ac > 0)
    gather_steps(re, im, near + V.a_seg[leaf], ac, V.a_idx + ak, x, R, G, g, r, na * rank / S,
                 na * (rank + 1) / S);
  const int bk = V.b_kptr[leaf], bc = V.b_kptr[leaf + 1] - bk, nb = (bc + G - 1) / G;
  grid_dep_wait();
  if (!skip && g < G && bc > 0)
    gather_steps(re, im, lrseg + V.b_seg[leaf], bc, V.b_idx + bk, t, R, G, g, r, (int)((long long)nb * rank / S),
                 (int)((long long)nb * (rank + 1) / S));
  part[tid] = cd(re, im);
  bool any = __syncthreads_or(skip);
  if (tid == 0) s_skip = any;
  if (tid < R) {
    double sr = part[tid].re, si = part[tid].im;
    for (int i = 1; i < G; i++) {
      sr += part[i * R + tid].re;
      si += part[i * R + tid].im;
    }
    rows[tid] = cd(sr, si);
  }
  if (S > 1) {
    cl.sync();
    if (rank == 0)
      for (int i = 1; i < S; i++) any |= *cl.map_shared_rank(&s_skip, i) != 0;
  }
  if (rank == 0 && !any) {
    double d[5] = {0, 0, 0, 0, 0};
    if (tid < R) {
      double sr = rows[tid].re, si = rows[tid].im;
      for (int i = 1; i < S; i++) {
        const cd v = cl.map_shared_rank(rows, i)[tid];
        sr += v.re;
        si += v.im;
      }
      const cd xv = x[ls + tid];
      double yr = sr - 0.5 * xv.re, yi = si - 0.5 * xv.im;
      if (bminus) {
        const cd bv = bminus[ls + tid];
        yr = bv.re - yr;
        yi = bv.im - yi;
      }
      y[ls + tid] = cd(yr, yi);
      if (dot_a) {
        const cd a = dot_a[ls + tid];
        d[0] = a.re * yr + a.im * yi;
        d[1] = a.re * yi - a.im * yr;
      }
      if (dot_b) {
        const cd b = dot_b[ls + tid];
        d[2] = yr * b.re + yi * b.im;
        d[3] = yr * b.im - yi * b.re;
      }
      d[4] = yr * yr + yi * yi;
    }
    if (partials) {
      warp_sum5(d, sdot[warp], 32 * warp < R);
      __syncthreads();
      if (tid < 5) {
        double sum = 0;
        for (int w = 0; w < W; w++) sum += sdot[w][tid];
        partials[(size_t)leaf * 5 + tid] = sum;
      }
    }
  }
  if (S > 1) cl.sync();  // the row sums stay until they are read
  if (rank == 0 && !any && partials && red5) {
    // the last leaf to finish reduces all partials in fixed order
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(ticket, 1u) == (unsigned)nleaf - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      double acc[5] = {0, 0, 0, 0, 0};
      for (int l = tid; l < nleaf; l += kGatherThreads)
        for (int i = 0; i < 5; i++) acc[i] += __ldcg(&partials[(size_t)l * 5 + i]);
      warp_sum5(acc, sdot[warp], 32 * warp < nleaf);
      __syncthreads();
      if (tid < 5) {
        double sum = 0;
        for (int w = 0; w < W; w++) sum += sdot[w][tid];
        red5[tid] = sum;
      }
      if (tid == 0) *ticket = 0u;
    }
  }
}

void launch_matvec_f64(const DevPartition& DP, const DevHMat& H, bool tr, const void* x, void* y, const void* bminus,
                       const MatvecEpilogue& ep, const int* done, cudaStream_t s, bool pdl) {
  SegView v = {};
  v.leaf_start = DP.leaf_start.as<int>();
  v.a_seg = (tr ? DP.near_seg_t : DP.near_seg).as<long long>();
  v.a_kptr = (tr ? DP.didx_t_ptr : DP.didx_ptr).as<int>();
  v.a_idx = (tr ? DP.didx_t : DP.didx).as<int>();
  if (tr && DP.nd > 0 && !H.nearT.p) throw Error(3, "internal: transposed near field not built");
  const cd* useg = H.useg.as<cd>();
  const cd* vseg = H.vseg.as<cd>();
  cd* t = H.tvec64.as<cd>();
  cd* p = H.pbuf.as<cd>();
  const int sms = device_sm_count();
  if (DP.na > 0) {
    SegView d = v;
    d.b_seg = (tr ? H.seg_f : H.seg_t).as<long long>();
    d.b_kptr = (tr ? H.kseg_f : H.kseg_t).as<int>();
    d.order = (tr ? H.order_rows : H.order_cols).as<int>();
    auto dot = DP.max_leaf <= 32 ? dot64_kernel<1>
               : DP.max_leaf <= 64 ? dot64_kernel<2>
               : DP.max_leaf <= 128 ? dot64_kernel<4>
                                    : dot64_kernel<8>;
    int parts = 1;  // a warp per 32 columns or so: 222 us a matvec against 229 with half of them (10620 triangles)
    while (parts < 32 && DP.nleaf * parts < 16 * sms) parts *= 2;
    launch_k(pdl, dot, dim3(DP.nleaf, parts), dim3(kDotThreads), 0, s, d, tr ? useg : vseg, (const cd*)x, p, done);
    launch_reduce_f64(DP, H, tr, p, t, done, s, pdl);
  }
  v.b_seg = (tr ? H.seg_t : H.seg_f).as<long long>();
  v.b_kptr = (tr ? H.kseg_t : H.kseg_f).as<int>();
  v.b_idx = (tr ? H.vidx : H.uidx).as<int>();
  v.order = (tr ? H.order_cols : H.order_rows).as<int>();
  // CTAs per leaf: up to two per SM always (128 leaves of 2720 triangles: 72 us a matvec with 1024 CTAs, 62 with
  // 512), up to four while a CTA keeps 160 KB of the leaf (512 leaves of 10620 triangles: 238 us with
  // 512 CTAs, 229 with 1024; 256 leaves of 5280: 109 us with 512, 114 with 1024, 156 with 256)
  const size_t bytes = (tr ? H.nearT : H.near).bytes + (tr ? H.vseg : H.useg).bytes;
  unsigned parts = 1;
  while (parts < 8 && (DP.nleaf * (int)parts < 2 * sms ||
                       (DP.nleaf * (int)parts < 4 * sms && bytes / ((size_t)DP.nleaf * parts) >= 320 * 1024)))
    parts *= 2;
  launch_clusters(pdl && DP.na > 0, parts, gather64_kernel, dim3(DP.nleaf * parts), dim3(kGatherThreads), s, v,
                  DP.nleaf, (tr ? H.nearT : H.near).as<cd>(), tr ? vseg : useg, t, (const cd*)x, (cd*)y,
                  (const cd*)bminus, (const cd*)ep.dot_a, (const cd*)ep.dot_b, ep.partials, ep.red5,
                  H.ticket.as<unsigned>(), done);
}

}  // namespace ac3d
