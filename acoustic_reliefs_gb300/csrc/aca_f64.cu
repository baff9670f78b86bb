// ACA of the FP64 path (compute_ACA_block, aca.cpp:38-82, argmax rules aca.cpp:9-36; receivers
// compute_ACA_listener, aca.cpp:84-134): the sequence of assemble.cu's kernels in complex FP64, one CTA
// per block.
//
// Bound by the FP64 pipe: GB300 runs two FP64 lanes per clock and SM, a warp instruction every 64
// clocks and scheduler, which is also its latency, so one warp per scheduler fills the pipe and what
// counts is how many lanes each instruction uses. Block sides are about c, 2 c, 4 c, ... with 16 < c <=
// 32, so one entry per lane left a third of them idle. An entry is evaluated as six items, one per
// quadrature point, spread over the CTA's threads (128 for sides up to 64, 256 above: 20 columns are
// 120 items); its owner adds them in order. The square roots and sums of the cross terms are formed
// once per value instead of on every lane, and the stopping test needs no division or square root.
// With a warp per block before: assembly 15.7 -> 11.5 ms on the 5280-triangle relief at 2 kHz, the three
// assemblies of the 1280-triangle sphere at a tolerance of 1e-10 about 5 ms each -> 1.2 ms.
#include <algorithm>
#include <mutex>

#include <math_constants.h>

#include "common.cuh"
#include "internal.h"
#include "listener.h"

namespace ac3d {

struct AcaF64Args {
  const double4* va;              // panel vertices a
  const ElemGeo<double>* eg;
  const double4* cen;             // centroids: the exactly-zero block test
  const double4* rowpts;          // rows: centroids or receivers
  const int4* blocks;
  const int* order;
  double k, eps, eps2;            // eps^2, -1 for eps < 0
  int maxk, zero_guard, iter_cap;
  int wide;                       // every block in the order of the wide ones (below)
  int chunk;                      // entries evaluated at a time: T, or what shared memory leaves room for
  cd* pool;
  long long pool_cap;
  unsigned long long* pool_used;
  long long* term_off;
  int* rank;
  int* status;
  int* passes;  // per block: rows (and columns) evaluated, or null
};

__constant__ double c_quad[3][6] = {
    {quad_m(0), quad_m(1), quad_m(2), quad_m(3), quad_m(4), quad_m(5)},
    {quad_n(0), quad_n(1), quad_n(2), quad_n(3), quad_n(4), quad_n(5)},
    {quad_w(0), quad_w(1), quad_w(2), quad_w(3), quad_w(4), quad_w(5)}};

namespace {
struct F64Item {
  double f, re, im;  // odd in eight-byte words: neither an item nor an entry per lane conflicts
};
// Shared memory: this, the coefficients and offsets of the terms, the items of a chunk of entries and a bit
// per row
template <int T>
struct F64Cta {
  double bv[2][T / 32];
  int bi[2][T / 32];
  double sd[2][T / 32];
  long long base;
  int ovf, pad;
};
template <int T>
size_t f64_smem(int iter_cap, int max_rows, int chunk) {
  return sizeof(F64Cta<T>) + (size_t)iter_cap * (sizeof(cd) + sizeof(long long) + sizeof(double)) +
         (size_t)chunk * sizeof(F64Item) * 6 + (size_t)((max_rows + 31) / 32) * 4;
}
constexpr size_t kF64SmemMax = 227 * 1024;
}  // namespace

// Items of cnt entries (point + e ps, panel + e es; ps and es 0 or 1): item 6 e + q is quadrature point q.
template <int T>
__device__ __noinline__ void f64_items(double k, const double4* __restrict__ pts, int ps,
                                       const double4* __restrict__ va, const ElemGeo<double>* __restrict__ eg, int es,
                                       int cnt, F64Item* items) {
#pragma unroll 1
  for (int it = threadIdx.x; it < 6 * cnt; it += T) {
    const int e = it / 6, q = it - 6 * e;
    const double4 p = pts[e * ps], a = va[e * es];
    const ElemGeo<double>& g = eg[e * es];
    const double dx = p.x - a.x, dy = p.y - a.y, dz = p.z - a.z;
    const double m = c_quad[0][q], n = c_quad[1][q], w = c_quad[2][q];
    // entry_from_d
    const double rx = dx - m * g.ab[0] - n * g.ac[0];
    const double ry = dy - m * g.ab[1] - n * g.ac[1];
    const double rz = dz - m * g.ab[2] - n * g.ac[2];
    const double r2 = rx * rx + ry * ry + rz * rz;
    const double r = sqrt(r2);
    const double rinv = 1.0 / r;
    const double s = rx * g.n[0] + ry * g.n[1] + rz * g.n[2];
    const double kr = k * r;
    double sn, cs;
    sincos(kr, &sn, &cs);
    items[it] = {w * s * rinv * rinv * rinv, cs + kr * sn, kr * cs - sn};
  }
}

// Entry e from its items, less the earlier terms, four loads in flight.
__device__ __forceinline__ cd f64_finish(const F64Item* items, int e, const cd* coef, const long long* toff,
                                         const cd* pool, int nst, bool swap = false) {
  double re = 0, im = 0;
#pragma unroll 1
  for (int it = 6 * e; it < 6 * e + 6; it++) {
    const F64Item t = items[it];
    re = fma(t.f, t.re, re);
    im = fma(t.f, t.im, im);
  }
  const double scale = 0.5 / (4.0 * kPi);
  cd acc(re * scale, im * scale);
#pragma unroll 1
  for (int p = 0; p < nst; p += 4) {
    cd a[4];
#pragma unroll
    for (int u = 0; u < 4; u++) a[u] = pool[toff[min(p + u, nst - 1)]];
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (p + u < nst) cfms(acc, swap ? a[u] : coef[p + u], swap ? coef[p + u] : a[u]);
  }
  return acc;
}

// (value, index) argmax over the CTA, first index on ties; values non-negative, or -1 for a thread
// without one, so that their bits order as integers. sv, si: free after the next barrier.
template <int T>
__device__ __forceinline__ void f64_argmax(double& val, int& idx, double* sv, int* si) {
  const unsigned long long key = val < 0.0 ? 0ull : (unsigned long long)__double_as_longlong(val + 0.0) + 1ull;
  const unsigned hk = (unsigned)(key >> 32), hm = __reduce_max_sync(0xffffffffu, hk);
  const unsigned lk = hk == hm ? (unsigned)key : 0u, lm = __reduce_max_sync(0xffffffffu, lk);
  idx = (int)__reduce_min_sync(0xffffffffu, hk == hm && lk == lm ? (unsigned)idx : 0xffffffffu);
  const unsigned long long best = ((unsigned long long)hm << 32) | lm;
  val = best == 0ull ? -1.0 : __longlong_as_double((long long)(best - 1ull));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    sv[w] = val;
    si[w] = idx;
  }
  __syncthreads();
  val = sv[0];
  idx = si[0];
#pragma unroll
  for (int i = 1; i < T / 32; i++)
    if (sv[i] > val || (sv[i] == val && si[i] < idx)) {
      val = sv[i];
      idx = si[i];
    }
}

// x^2 + y^2 with y^2 rounded by itself. On symmetric geometries many candidates for a pivot are equal but for
// rounding, and which of them is largest hangs on this order; another pivot is another approximation of the
// block (1.6% of the solution on two spheres of 80 panels in leaves of one). So it is fixed, as the results of
// the FP64 kernels before these have it: for rows and for wide blocks the imaginary part by itself, for the
// columns of the others the real part.
__device__ __forceinline__ double f64_abs2(double x, double y) { return fma(x, x, y * y); }

template <int T>
__global__ void __launch_bounds__(T) aca_f64_kernel(AcaF64Args A) {
  constexpr int W = T / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  F64Cta<T>& S = *reinterpret_cast<F64Cta<T>*>(smem);
  cd* coef = reinterpret_cast<cd*>(smem + sizeof(F64Cta<T>));
  long long* toff = reinterpret_cast<long long*>(coef + A.iter_cap);
  double* prod = reinterpret_cast<double*>(toff + A.iter_cap);
  F64Item* items = reinterpret_cast<F64Item*>(prod + A.iter_cap);
  unsigned* used = reinterpret_cast<unsigned*>(items + 6 * A.chunk);
  const int C = A.chunk;
  static_assert(sizeof(F64Cta<T>) % 16 == 0, "the coefficients follow");
  const int b = A.order[blockIdx.x];
  const int4 q = A.blocks[b];
  const int rs = q.x, cs = q.z, m = q.y - q.x, n = q.w - q.z;
  const int iter_lim = max(0, min(min(A.maxk, A.iter_cap), min(m - 1, n - 1)));
  // column residuals of wide blocks multiply term by coefficient, those of the others coefficient by term: the
  // order of the two products in the imaginary part, and so the last bits, as assemble.cu has them
  const bool wide = A.wide || m > kWarpAcaMaxDim || n > kWarpAcaMaxDim;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // exactly-zero block: all panels in one axis-aligned plane that holds every target point (see aca_kernel)
  if (A.zero_guard && iter_lim > 0) {
    for (int d = 0; d < 3; d++) {
      const double4 a0 = A.va[cs];
      const double v = d == 0 ? a0.x : (d == 1 ? a0.y : a0.z);
      bool ok = true;
      for (int j = tid; j < n && ok; j += T) {
        const double4 a = A.va[cs + j];
        ok = (d == 0 ? a.x : (d == 1 ? a.y : a.z)) == v && A.eg[cs + j].ab[d] == 0.0 && A.eg[cs + j].ac[d] == 0.0;
      }
      for (int i = tid; i < m && ok; i += T) {
        const double4 p = A.cen[rs + i];
        ok = (d == 0 ? p.x : (d == 1 ? p.y : p.z)) == v;
      }
      if (__syncthreads_and(ok)) {
        if (tid == 0) {
          A.rank[b] = 0;
          if (A.passes) A.passes[b] = 0;
        }
        return;
      }
    }
  }

  for (int w = tid; w < (m + 31) / 32; w += T) used[w] = w == 0 ? 1u : 0u;
  double err = 0;
  int i = 0, iter = 0, nst = 0, npass = 0;
  bool need_alloc = true;
  __syncthreads();
  while (iter < iter_lim) {
    if (need_alloc) {
      if (tid == 0) {
        const unsigned long long need = (unsigned long long)(m + n);
        const unsigned long long bb = atomicAdd(A.pool_used, need);
        S.ovf = bb + need > (unsigned long long)A.pool_cap;
        S.base = (long long)bb;
        if (S.ovf) atomicOr(A.status, 1);
      }
      __syncthreads();
      if (S.ovf) break;
      need_alloc = false;
    }
    npass++;
    const long long base = S.base;
    cd* unew = A.pool + base;
    cd* vnew = unew + m;
    for (int p = tid; p < nst; p += T) coef[p] = A.pool[toff[p] + i];

    // row residual v = M(i, :) - U(i, :) V and column pivot
    double best = -1.0;
    int bidx = 0;
    for (int c0 = 0; c0 < n; c0 += C) {
      if (c0) __syncthreads();  // the previous entries are finished
      f64_items<T>(A.k, A.rowpts + rs + i, 0, A.va + cs + c0, A.eg + cs + c0, 1, min(C, n - c0), items);
      __syncthreads();
      const int c = c0 + tid;
      if (tid < C && c < n) {
        const cd v = f64_finish(items, tid, coef, toff, A.pool + m + c, nst);
        vnew[c] = v;
        const double a = f64_abs2(wide ? v.re : v.im, wide ? v.im : v.re);
        if (a > best) {
          best = a;
          bidx = c;
        }
      }
    }
    f64_argmax<T>(best, bidx, S.bv[0], S.bi[0]);
    const int j = bidx;
    const cd vj = vnew[j];
    for (int p = tid; p < nst; p += T) coef[p] = A.pool[toff[p] + m + j];
    __syncthreads();  // v_j is read before it is divided
    const bool keep = A.zero_guard && vj.re == 0.0 && vj.im == 0.0;
    double vn = 0;
    for (int c = tid; c < n; c += T) {
      cd v = vnew[c];
      if (!keep) v = cdiv(v, vj);
      vnew[c] = v;
      vn += abs2(v);
    }
    // column residual u = M(:, j) - U V(:, j)
    double un = 0;
    for (int r0 = 0; r0 < m; r0 += C) {
      if (r0) __syncthreads();
      f64_items<T>(A.k, A.rowpts + rs + r0, 1, A.va + cs + j, A.eg + cs + j, 0, min(C, m - r0), items);
      __syncthreads();
      const int r = r0 + tid;
      if (tid < C && r < m) {
        const cd u = f64_finish(items, tid, coef, toff, A.pool + r, nst, wide);
        unew[r] = u;
        un += abs2(u);
      }
    }
    __syncthreads();
    // cross terms |u^T U_p| |v V_p^T|, a warp per earlier term: the four sums folded over the lanes (the upper
    // half of them dropped from a lane at each step), so that each is added and rooted once
    for (int p = warp; p < nst; p += W) {
      const cd* Up = A.pool + toff[p];
      const cd* Vp = Up + m;
      cd ud(0, 0), vd(0, 0);
#pragma unroll 2
      for (int r = lane; r < m; r += 32) cfma(ud, unew[r], Up[r]);
#pragma unroll 2
      for (int c = lane; c < n; c += 32) cfma(vd, vnew[c], Vp[c]);
      const bool up = (lane & 16) != 0;
      double x = (up ? vd.re : ud.re) + __shfl_xor_sync(0xffffffffu, up ? ud.re : vd.re, 16);
      double y = (up ? vd.im : ud.im) + __shfl_xor_sync(0xffffffffu, up ? ud.im : vd.im, 16);
      const bool im = (lane & 8) != 0;
      double s = (im ? y : x) + __shfl_xor_sync(0xffffffffu, im ? x : y, 8);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const double t = __shfl_xor_sync(0xffffffffu, s, 8);
      const double a = sqrt(s * s + t * t);  // lanes 0..15: |u^T U|, lanes 16..31: |v V^T|
      const double v = __shfl_xor_sync(0xffffffffu, a, 16);
      if (lane == 0) prod[p] = a * v;
    }
    un = warp_sum(un);
    vn = warp_sum(vn);
    if (lane == 0) {
      S.sd[0][warp] = un;
      S.sd[1][warp] = vn;
    }
    __syncthreads();
    double unt = S.sd[0][0], vnt = S.sd[1][0];
#pragma unroll 1
    for (int w = 1; w < W; w++) {
      unt += S.sd[0][w];
      vnt += S.sd[1][w];
    }
    double dots = 0;
    for (int p = lane; p < nst; p += 32) dots += prod[p];
    dots = warp_sum(dots);
    const double uv = unt * vnt;
    err += uv + 2 * dots;
    // sqrt(uv / err) <= eps, as it stands where err is 0, infinite or NaN
    if (err > 0.0 && err < CUDART_INF ? uv <= A.eps2 * err : sqrt(uv / err) <= A.eps) break;
    const bool zero_term = unt == 0.0 || vnt == 0.0;
    // next row pivot: first max |u|^2 over unused rows
    best = -1.0;
    bidx = 0;
    for (int r = tid; r < m; r += T) {
      if ((used[r >> 5] >> (r & 31)) & 1u) continue;
      const cd u = unew[r];
      const double a = f64_abs2(u.re, u.im);
      if (a > best) {
        best = a;
        bidx = r;
      }
    }
    f64_argmax<T>(best, bidx, S.bv[1], S.bi[1]);
    i = bidx;
    if (tid == 0) {
      used[i >> 5] |= 1u << (i & 31);
      if (!zero_term) {
        toff[nst] = base;
        A.term_off[(long long)b * A.maxk + nst] = base;
      }
    }
    if (!zero_term) {
      nst++;
      need_alloc = true;
    }
    iter++;
    __syncthreads();
  }
  if (tid == 0) {
    A.rank[b] = nst;
    if (A.passes) A.passes[b] = npass;
  }
}

template <int T>
static void aca_f64_launch(AcaF64Args a, const int* order, int nblocks, int max_rows, cudaStream_t s) {
  if (nblocks <= 0) return;
  size_t smem = f64_smem<T>(a.iter_cap, max_rows, a.chunk = T);
  if (smem > kF64SmemMax) {
    // millions of rows, or thousands of terms: fewer entries at a time
    const size_t rest = f64_smem<T>(a.iter_cap, max_rows, 0);
    a.chunk = rest < kF64SmemMax ? (int)((kF64SmemMax - rest) / (6 * sizeof(F64Item))) : 0;
    smem = f64_smem<T>(a.iter_cap, max_rows, a.chunk);
  }
  if (a.chunk < 1) throw Error(4, "ACA block too large for shared memory");
  // once per process, to the largest size any launch uses: contexts on other threads launch with others
  static std::once_flag once;
  std::call_once(once, [] {
    AC3D_CUDA(cudaFuncSetAttribute(aca_f64_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF64SmemMax));
  });
  a.order = order;
  note_launch();
  aca_f64_kernel<T><<<nblocks, T, smem, s>>>(a);
  AC3D_CUDA(cudaGetLastError());
}

void launch_aca_f64(const DevGeometry& G, const DevPartition& DP, DevHMat& H, double eps, int max_rows, cudaStream_t s,
                    cudaStream_t s_small) {
  if (DP.na == 0) return;
  AcaF64Args a{G.va.as<double4>(), G.eg64.as<ElemGeo<double>>(), G.cen.as<double4>(), G.cen.as<double4>(),
               DP.blocks_a.as<int4>(), nullptr, H.k, eps, eps < 0 ? -1.0 : eps * eps, H.maxk, 1, H.maxk, H.maxk > kWarpAcaTerms, 0, H.pool.as<cd>(), H.pool_cap,
               H.pool_used.as<unsigned long long>(), H.term_off.as<long long>(), H.rank.as<int>(),
               (int*)(H.pool_used.as<unsigned long long>() + 1), H.passes.as<int>()};
  // aca_order: blocks above 256, then up to 256, 128 and 64
  const int* order = DP.aca_order.as<int>();
  const int large = DP.aca_split[0] + DP.aca_split[1] + DP.aca_split[2];
  aca_f64_launch<256>(a, order, large, max_rows, s);
  aca_f64_launch<128>(a, order + large, DP.aca_split[3], 64, s_small);
}

void launch_listener_aca_f64(const DevGeometry& G, const double4* pts, int L, double k, double eps, int maxk, cd* pool,
                             long long pool_cap, unsigned long long* used, long long* term_off, int* rank, int* status,
                             const int4* block, const int* order, cudaStream_t s) {
  const int iter_lim = std::max(1, std::min(maxk, std::min(L - 1, G.ne - 1)));
  AcaF64Args a{G.va.as<double4>(), G.eg64.as<ElemGeo<double>>(), G.cen.as<double4>(), pts, block, nullptr, k,
               eps, eps < 0 ? -1.0 : eps * eps, maxk, 0, iter_lim, 1, 0, pool, pool_cap, used, term_off, rank, status, nullptr};
  aca_f64_launch<256>(a, order, 1, L, s);
}

}  // namespace ac3d
