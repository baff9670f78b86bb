// The FP64 H-matrix's matvec: the three passes of matvec.cu (dot, reduce, gather) over the same segments.
//
// Bound by the FP64 pipe, not by memory: GB300 runs two FP64 lanes per clock and SM, so an element (four
// multiply-adds, 16 bytes) takes 3 times as long to compute as to read, a warp instruction holds a
// scheduler's pipe for 64 clocks, and lanes without an element cost as much as those with one. Leaves hold 16 to
// 32 elements (or their doubles), so lanes laid along a column's rows were a third empty and added
// up over shuffles. Here the dot pass gives a lane a whole column (up to 32 rows of it), several CTAs a
// leaf; the gather pass gives a thread a row of one column class (every 8th to 32nd column) and a leaf to a
// cluster of 4 or 8 CTAs. At 64 clocks an instruction the other warps hide the loads, so these go from
// global memory to registers (five CTAs per SM and two columns in flight: 123 us a matvec on 5280
// triangles; three and four: 141; two and eight: 147). Matvec, against the FP32 layout: 248 -> 123 us on
// 5280 triangles; gather on the sphere of 1280 triangles in 16 leaves: 92 -> 19 us.
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

// Sums have the order of the FP32 kernels' layout (G0 lanes per column in the dot pass; warps and
// column slots in the gather), so that a solve ends on the same iterate whatever the layout.

// p[kptr[leaf] + k] = sum over the leaf's rows of S[k][row] x[row]. G lanes per column (1 up to 32
// rows, so that a lane has at most 32), gridDim.y CTAs per leaf, whose warps take 32 / G columns in turn.
// Rows g, g + G0, ... are summed apart for every g, then pairs G0 / 2 apart, G0 / 4, ...
template <int G, int G0>
__global__ void __launch_bounds__(kDotThreads, 6) dot64_kernel(SegView V, const cd* __restrict__ lrseg,
                                                               const cd* __restrict__ x, cd* __restrict__ p,
                                                               const int* __restrict__ done) {
  __shared__ __align__(16) unsigned char xraw[kMaxRows * sizeof(cd)];
  cd* xs = reinterpret_cast<cd*>(xraw);
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
  constexpr int CW = 32 / G, NA = G0 / G;
  const int warp = blockIdx.y * (kDotThreads / 32) + (threadIdx.x >> 5), nw = gridDim.y * (kDotThreads / 32);
  for (int c0 = warp * CW; c0 < K; c0 += nw * CW) {
    const int c = c0 + lane / G;
    const cd* col = seg + (long long)min(c, K - 1) * R;
    double re[NA], im[NA];
#pragma unroll
    for (int u = 0; u < NA; u++) re[u] = im[u] = 0;
    for (int r0 = g; r0 < R; r0 += G0) {
      cd a[NA];
#pragma unroll
      for (int u = 0; u < NA; u++) a[u] = col[min(r0 + u * G, R - 1)];
#pragma unroll
      for (int u = 0; u < NA; u++)
        if (r0 + u * G < R) mac64(re[u], im[u], a[u], xs[r0 + u * G]);
    }
#pragma unroll
    for (int h = NA / 2; h > 0; h >>= 1)
#pragma unroll
      for (int u = 0; u < h; u++) {
        re[u] += re[u + h];
        im[u] += im[u + h];
      }
    double sr = re[0], si = im[0];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (g == 0 && c < K) p[k0 + c] = cd(sr, si);
  }
}

// Thread (class k of NC, row r): the columns k, k + NC, ... of every chunk of cpc columns
template <int NC>
__device__ __forceinline__ void gather_class(double& re, double& im, const cd* __restrict__ seg, int K,
                                             const int* __restrict__ idx, const cd* __restrict__ z, int R, int cpc,
                                             int k, int r) {
  constexpr int U = 2;
  int c0 = 0, j = k;
  auto next = [&]() {
    while (c0 < K && j >= min(cpc, K - c0)) {
      c0 += cpc;
      j = k;
    }
    const int c = c0 < K ? c0 + j : -1;
    j += NC;
    return c;
  };
  for (int c = next(); c >= 0;) {
    int cc[U], jx[U];
    cd a[U], v[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      cc[u] = c;
      if (c >= 0) c = next();
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      jx[u] = max(idx[max(cc[u], 0)], 0);  // padding columns are zero and take any multiplier
      a[u] = seg[(long long)max(cc[u], 0) * R + r];
    }
#pragma unroll
    for (int u = 0; u < U; u++) v[u] = z[jx[u]];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (cc[u] >= 0) mac64(re, im, a[u], v[u]);
  }
}

// The gather pass's directions: A x, and A^T x with the near field from its transposed copy or, where the
// device has no room for that, in place
enum : int { kForward = 0, kTransposed = 1, kInPlace = 2 };

// A^T: the near part of row r (a column of the near blocks that have the leaf's columns) that warp w of the FP32
// layout's eight adds: of the blocks w, w + 8, ..., their rows in order.
template <int DIR>
__device__ __forceinline__ void near_transposed(double& re, double& im, const SegView& V, int leaf,
                                                const cd* __restrict__ near, const cd* __restrict__ x, int R, int w,
                                                int r) {
  constexpr int U = 4;  // loads in flight
  const int end = V.trn_ptr[leaf + 1];
  for (int it = V.trn_ptr[leaf] + w; it < end; it += 8) {
    const int b = V.trn[it];
    const int4 q = V.blocks_d[b];
    const int m = q.y - q.x, step = DIR == kInPlace ? 1 : R;
    const cd* D = near + V.near_off[b] + (long long)r * (DIR == kInPlace ? m : 1);
    const cd* xs = x + q.x;
    int i = 0;
    for (; i + U <= m; i += U, D += U * step) {
      cd a[U], z[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        a[u] = D[u * step];
        z[u] = xs[i + u];
      }
#pragma unroll
      for (int u = 0; u < U; u++) mac64(re, im, a[u], z[u]);
    }
#pragma unroll 1
    for (; i < m; i++, D += step) mac64(re, im, *D, xs[i]);
  }
}

// y[leaf rows] = -x/2 + S_A x[a_idx] + S_B t[b_idx], or b - that, with the optional dot partials of
// seg_gather_persist_kernel. The NC column classes are that kernel's (warp, slot) pairs: a cluster of S CTAs
// holds them all, NC / S each with a thread per row. Every CTA adds its warps' slots, the first one the warps in
// order, and finishes the leaf. The near part runs before the wait for the reduce pass; in A^T it is summed
// apart, by a thread per row and warp, and added to the warp's low-rank part, as the FP32 layout has it. (With
// the near columns in the classes, as in A x, FP64 adjoint BiCGSTAB solves ended on other iterates. A^T x on
// 5736 triangles in leaves of up to 32, 64, 128 and 256, in the FP32 layout, so, and in the classes: 287, 186,
// 136 us; 450, 212, 177; 970, 255, 280; 1926, 316, 695.)
template <int NC, int S, int DIR>
__global__ void __launch_bounds__(kGatherThreads, 5) gather64_kernel(
    SegView V, int nleaf, const cd* __restrict__ near, const cd* __restrict__ lrseg, const cd* __restrict__ t,
    const cd* __restrict__ x, cd* __restrict__ y, const cd* __restrict__ bminus, const cd* __restrict__ dot_a,
    const cd* __restrict__ dot_b, double* partials, double* red5, unsigned* ticket, const int* __restrict__ done) {
  constexpr int W = 8, GP = NC / S, SL = NC / W, LW = GP / SL;  // slots per warp, warps per CTA
  static_assert(GP % SL == 0 && LW * S == W, "a CTA holds whole warps");
  __shared__ __align__(16) unsigned char praw[kGatherThreads * sizeof(cd)];
  __shared__ __align__(16) unsigned char rraw[LW * kGatherThreads / GP * sizeof(cd)];
  cd* part = reinterpret_cast<cd*>(praw);
  cd* rows = reinterpret_cast<cd*>(rraw);
  __shared__ double sdot[W][5];
  __shared__ bool s_last;
  __shared__ int s_skip;
  grid_dep_launch();
  const cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int leaf = V.order[blockIdx.x / S];
  const int ls = V.leaf_start[leaf], R = V.leaf_start[leaf + 1] - ls;
  const int tid = threadIdx.x, warp = tid >> 5;
  // the flag may be set while this kernel runs: a thread that sees it skips its sums, but not the barriers,
  // and its cluster writes nothing
  const bool skip = done && *(volatile const int*)done;
  // two warps per CTA are one from either end: the first classes of a chunk have a column more
  const int g = tid / R, r = tid - g * R, k = (g < SL ? rank : W - 1 - rank) * SL + g % SL;
  const int cpc = min(128, max(2, (int)(kStageBytes / sizeof(cd)) / R & ~1));  // columns per chunk of its ring
  double re = 0, im = 0, near_re = 0, near_im = 0;
  if constexpr (DIR == kForward) {
    const int ak = V.a_kptr[leaf], ac = V.a_kptr[leaf + 1] - ak;
    if (!skip && g < GP) gather_class<NC>(re, im, near + V.a_seg[leaf], ac, V.a_idx + ak, x, R, cpc, k, r);
  } else {
    if (!skip && g < LW) near_transposed<DIR>(near_re, near_im, V, leaf, near, x, R, g ? W - 1 - rank : rank, r);
  }
  const int bk = V.b_kptr[leaf], bc = V.b_kptr[leaf + 1] - bk;
  grid_dep_wait();
  if (!skip && g < GP) gather_class<NC>(re, im, lrseg + V.b_seg[leaf], bc, V.b_idx + bk, t, R, cpc, k, r);
  if (g < GP) part[tid] = cd(re, im);
  bool any = __syncthreads_or(skip);
  if (tid == 0) s_skip = any;
  if (tid < LW * R) {
    const cd* q = part + (size_t)(tid / R) * SL * R + tid % R;
    cd v = q[0];
    if constexpr (SL == 2) v = cd(v.re + q[R].re, v.im + q[R].im);
    if constexpr (SL == 4)
      v = cd((v.re + q[R].re) + (q[2 * R].re + q[3 * R].re), (v.im + q[R].im) + (q[2 * R].im + q[3 * R].im));
    if constexpr (DIR != kForward) v = cd(v.re + near_re, v.im + near_im);
    rows[tid] = v;
  }
  cl.sync();
  if (rank == 0)
    for (int i = 1; i < S; i++) any |= *cl.map_shared_rank(&s_skip, i) != 0;
  if (rank == 0 && !any) {
    double d[5] = {0, 0, 0, 0, 0};
    if (tid < R) {
      double sr = 0, si = 0;
      for (int i = 0; i < W; i++) {
        const bool own = LW == 1 || i < S;
        const cd v = cl.map_shared_rank(rows, own ? i : W - 1 - i)[(own ? 0 : R) + tid];
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
        d[0] += a.re * yr + a.im * yi;
        d[1] += a.re * yi - a.im * yr;
      }
      if (dot_b) {
        const cd b = dot_b[ls + tid];
        d[2] += yr * b.re + yi * b.im;
        d[3] += yr * b.im - yi * b.re;
      }
      d[4] += yr * yr + yi * yi;
    }
    if (partials) {
      warp_sum5(d, sdot[warp], 32 * warp < R);
      __syncthreads();
      if (tid < 5) {
        double sum = 0;
        for (int w = 0; w < (int)blockDim.x / 32; w++) sum += sdot[w][tid];  // (warps from R / 32 on add 0)
        partials[(size_t)leaf * 5 + tid] = sum;
      }
    }
  }
  cl.sync();  // the row sums stay until they are read
  if (rank == 0 && !any && partials && red5) {
    // the last leaf to finish reduces all partials in fixed order
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(ticket, 1u) == (unsigned)nleaf - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      for (int vt = tid; vt < 256; vt += blockDim.x) {  // in the order of 256 threads
        double acc[5] = {0, 0, 0, 0, 0};
        for (int l = vt; l < nleaf; l += 256)
          for (int i = 0; i < 5; i++) acc[i] += __ldcg(&partials[(size_t)l * 5 + i]);
        warp_sum5(acc, sdot[vt >> 5], (vt & ~31) < nleaf);
      }
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
  v.a_seg = DP.near_seg.as<long long>();
  v.a_kptr = DP.didx_ptr.as<int>();
  v.a_idx = DP.didx.as<int>();
  const int dir = !tr ? kForward : H.nearT.p ? kTransposed : kInPlace;
  v.blocks_d = DP.blocks_d.as<int4>();
  v.near_off = (dir == kTransposed ? DP.near_off_t : DP.near_off).as<long long>();
  v.trn_ptr = DP.tr_near_ptr.as<int>();
  v.trn = DP.tr_near.as<int>();
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
    auto dot = DP.max_leaf <= 32 ? dot64_kernel<1, 8>
               : DP.max_leaf <= 64 ? dot64_kernel<2, 8>
               : DP.max_leaf <= 128 ? dot64_kernel<4, 16>
                                    : dot64_kernel<8, 32>;
    int parts = 1;  // a warp per 32 columns or so: 222 us a matvec against 229 with half of them (10620 triangles)
    while (parts < 32 && DP.nleaf * parts < 16 * sms) parts *= 2;
    launch_k(pdl, dot, dim3(DP.nleaf, parts), dim3(kDotThreads), 0, s, d, tr ? useg : vseg, (const cd*)x, p, done);
    launch_reduce_f64(DP, H, tr, p, t, done, s, pdl);
  }
  v.b_seg = (tr ? H.seg_t : H.seg_f).as<long long>();
  v.b_kptr = (tr ? H.kseg_t : H.kseg_f).as<int>();
  v.b_idx = (tr ? H.vidx : H.uidx).as<int>();
  v.order = (tr ? H.order_cols : H.order_rows).as<int>();
  auto gather = [&](auto kern, int classes, int ctas) {
    const int threads = (classes / ctas * DP.max_leaf + 31) / 32 * 32;
    launch_clusters(pdl && DP.na > 0, (unsigned)ctas, kern, dim3(DP.nleaf * ctas), dim3(threads), s, v, DP.nleaf,
                    (dir == kTransposed ? H.nearT : H.near).as<cd>(), tr ? vseg : useg, t, (const cd*)x, (cd*)y, (const cd*)bminus,
                    (const cd*)ep.dot_a, (const cd*)ep.dot_b, ep.partials, ep.red5, H.ticket.as<unsigned>(), done);
  };
#define AC3D_GATHER64(NC, S)                                              \
  gather(dir == kForward      ? gather64_kernel<NC, S, kForward>          \
         : dir == kTransposed ? gather64_kernel<NC, S, kTransposed>       \
                              : gather64_kernel<NC, S, kInPlace>,         \
         NC, S)
  if (DP.max_leaf <= 32)
    AC3D_GATHER64(32, 4);
  else if (DP.max_leaf <= 64)
    AC3D_GATHER64(32, 8);
  else if (DP.max_leaf <= 128)
    AC3D_GATHER64(16, 8);
  else
    AC3D_GATHER64(8, 8);
#undef AC3D_GATHER64
}

}  // namespace ac3d
