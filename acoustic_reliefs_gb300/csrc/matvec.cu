// H-matrix matvec y = op(K - I/2) x (generic_product_impl::scaleAndAddTo, hmatrix.h:84-139),
// op = identity or the plain (non-conjugate) transpose.
//
// The matrix is held as per-leaf segments (R x K column-major, R = leaf size):
//   near segment of a row leaf   : its dense blocks side by side, columns indexing x;
//   U segment of a row leaf      : rows of the leaf of every admissible block above it, one column
//                                  per rank-1 term;
//   V segment of a column leaf   : columns of the leaf of every admissible block beside it.
// Forward:    p = per-column dots of the V segments with x   (dot pass, one to eight CTAs per leaf)
//             t[b, q] = sum over the column leaves of b of p (reduce, fixed leaf order)
//             y = -x/2 + near x + U t                         (gather pass, resident CTAs take the leaves)
// Transpose:  the same with U and V swapped, the near field from its transposed copy or, where the device
// has no room for that, from the blocks themselves.
// Both passes stream their segments through shared memory with bulk async copies, so the bytes
// in flight are set by the copy ring, not by how many loads a warp can issue. Every sum has a fixed
// order (atomics only count finished CTAs), so results are bit-reproducible. The FP64 H-matrix's
// passes are in matvec64.cu; the reduce pass is common.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "launch.cuh"
#include "segstream.cuh"

namespace ac3d {

namespace {
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
}  // namespace

// Double-float: the unevaluated sum hi + lo of two FP32 numbers, about 48 significant bits, used
// for the FP64-vector residual of iterative refinement so that it runs on the FP32 pipes (GB300's
// FP64 rate is a small fraction of its FP32 rate). Error-free transformations: two_sum (Knuth),
// two_prod by FMA (the double-double arithmetic of Dekker 1971, Hida-Li-Bailey 2001). The _rn
// intrinsics keep the compiler from contracting the exact splits into FMAs.
struct df32 {
  float hi, lo;
  __host__ __device__ df32(float h = 0.f, float l = 0.f) : hi(h), lo(l) {}
};

__device__ __forceinline__ df32 df_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return df32(s, e);
}
__device__ __forceinline__ df32 df_fast_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return df32(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ df32 df_add(df32 x, df32 y) {
  const df32 s = df_two_sum(x.hi, y.hi);
  return df_fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(x.lo, y.lo)));
}
// acc + a z for a float a: the product's rounding error and a z.lo go to the low word, which is
// renormalised when accumulators are combined (df_add).
__device__ __forceinline__ void df_mac(df32& acc, float a, df32 z) {
  const float p = __fmul_rn(a, z.hi);
  const float pe = __fmaf_rn(a, z.lo, __fmaf_rn(a, z.hi, -p));
  const df32 s = df_two_sum(acc.hi, p);
  acc = df32(s.hi, __fadd_rn(acc.lo, __fadd_rn(s.lo, pe)));
}

// Accumulator arithmetic of the matvec passes: plain FP32, or double-float.
template <typename AT, typename MT>
__device__ __forceinline__ void acc_mac(AT& ar, AT& ai, const cplx<MT>& a, const AT& zr, const AT& zi) {
  ar = fma((AT)a.re, zr, ar);
  ar = fma(-(AT)a.im, zi, ar);
  ai = fma((AT)a.re, zi, ai);
  ai = fma((AT)a.im, zr, ai);
}
__device__ __forceinline__ void acc_mac(df32& ar, df32& ai, const cplx<float>& a, const df32& zr, const df32& zi) {
  df_mac(ar, a.re, zr);
  df_mac(ar, -a.im, zi);
  df_mac(ai, a.re, zi);
  df_mac(ai, a.im, zr);
}
template <typename AT>
__device__ __forceinline__ AT acc_add(AT a, AT b) { return a + b; }
__device__ __forceinline__ df32 acc_add(df32 a, df32 b) { return df_add(a, b); }
template <typename AT>
__device__ __forceinline__ AT acc_shfl_xor(AT v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ df32 acc_shfl_xor(df32 v, int o) {
  return df32(__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o));
}
template <typename VT, typename AT>
__device__ __forceinline__ VT acc_to(AT v) { return (VT)v; }
template <>
__device__ __forceinline__ double acc_to<double, df32>(df32 v) { return (double)v.hi + (double)v.lo; }

// x (FP64) -> double-float multipliers
__global__ void to_df_kernel(int n, const cd* __restrict__ x, cplx<df32>* out) {
  grid_dep_wait();
  grid_dep_launch();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const cd v = x[i];
  const float rh = __double2float_rn(v.re), ih = __double2float_rn(v.im);
  out[i] = cplx<df32>(df32(rh, __double2float_rn(v.re - (double)rh)), df32(ih, __double2float_rn(v.im - (double)ih)));
}

// Lanes per column and rows per lane of the dot pass for leaves of up to 32 RPL rows: a group of G
// lanes shares one column, lane g summing rows g, g + G, g + 2G, ..., so one warp instruction
// covers 32 / G columns and the cross-lane sum takes log2(G) shuffle levels.
template <int RPL>
struct DotShape {
  static constexpr int G = RPL <= 2 ? 8 : RPL == 4 ? 16 : 32;
  static constexpr int RPG = 32 * RPL / G;
};

// Barrier of the consumer warps only (the producer keeps streaming): every consumer thread arrives
// on an mbarrier (release) and waits for the phase (acquire), with the bounded wait, so a failed
// pipeline cannot leave threads blocked. Returns false if the phase did not complete.
__device__ __forceinline__ bool consumer_sync(uint64_t* bar, uint32_t& phase) {
  mbar_arrive(bar);
  const bool ok = mbar_wait_bounded(bar, phase);
  phase ^= 1u;
  return ok;
}

// One step of a transposed butterfly: of 2 N values, a lane keeps N (the upper ones in the lanes with
// bit O set) and adds its partner's share of them: the bits of the butterfly on each.
template <int N, int O>
__device__ __forceinline__ void dot_fold(float* v) {
  const bool up = (threadIdx.x & O) != 0;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const float keep = up ? v[k + N] : v[k], give = up ? v[k] : v[k + N];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, O);
  }
}

// Dot pass: p[kptr[leaf] + k] = sum_rows S[k][row] x[leaf rows] for every column k of the leaf's
// low-rank segment (region B), gridDim.y CTAs per leaf. As the gather pass, eight consumer warps and one
// producer warp that streams the chunks, so that no barrier of the CTA stands between chunks, and sums over
// the lanes folded (4 shuffles for 12). Matvec, before and after: 29.4 and 27.7 us on 5280 triangles, 84.0 and
// 81.1 us on 20480, 145.8 and 143.0 us on 34340, 999 and 994 us on 118680.
template <typename MT, typename AT, int RPL>
__global__ void __launch_bounds__(kThreads + 32, 4) seg_dot_kernel(SegView V, const cplx<MT>* __restrict__ lrseg,
                                                                   const cplx<AT>* __restrict__ xm,
                                                                   cplx<AT>* __restrict__ p,
                                                                   const int* __restrict__ done) {
  constexpr int G = DotShape<RPL>::G, RPG = DotShape<RPL>::RPG;
  constexpr int CPW = 32 / G;             // columns per warp step
  constexpr int STEP = kWarps * CPW;      // columns per CTA step
  extern __shared__ __align__(128) unsigned char dsmem[];
  auto stage = reinterpret_cast<unsigned char(*)[kStageBytes]>(dsmem);
  __shared__ __align__(8) uint64_t full[kStages];
  __shared__ __align__(8) uint64_t empty[kStages];
  __shared__ __align__(8) uint64_t cbar;
  __shared__ int s_stop;
  // the segments and the partition are not written by any kernel of a solve: the first stages
  // stream in before the wait for the preceding kernel (which writes x and the done flag)
  const int leaf = V.order[blockIdx.x];
  if (threadIdx.x == 0) {
    for (int st = 0; st < kStages; st++) {
      mbar_init(&full[st], 1);
      mbar_init(&empty[st], kWarps);
    }
    mbar_init(&cbar, kThreads);
    s_stop = 0;
    fence_barrier_init();
  }
  // a set done flag stays set for the rest of the solve, so reading it before the wait can only
  // miss a flag that is being set (checked again after the wait). The Givens step beside this pass
  // may set it at any time, so the CTA votes: its threads must not part ways. The vote comes before the
  // leaf's places are loaded: a pass behind the end of a solve takes 2.4 instead of 2.9 us
  if (__syncthreads_or(done && *(volatile const int*)done)) {
    grid_dep_wait();
    grid_dep_launch();
    return;
  }
  const int ls = V.leaf_start[leaf], R = V.leaf_start[leaf + 1] - ls;
  int k0 = V.b_kptr[leaf], K = V.b_kptr[leaf + 1] - k0;
  const cplx<MT>* seg = lrseg + V.b_seg[leaf];
  if (gridDim.y > 1) {  // this CTA's part of the columns, from an even one on (16-byte aligned copies)
    const int lo = (int)((long long)K * blockIdx.y / gridDim.y) & ~1;
    const int hi = blockIdx.y + 1 == gridDim.y ? K : (int)((long long)K * (blockIdx.y + 1) / gridDim.y) & ~1;
    k0 += lo;
    K = hi - lo;
    seg += (long long)lo * R;
  }
  if (K == 0) {
    grid_dep_wait();
    grid_dep_launch();
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cpc = max(2, (int)(kStageBytes / sizeof(cplx<MT>)) / R & ~1);  // columns per chunk, even
  if (warp == kWarps) {
    int st = 0, issued = 0;
    uint32_t ph = 1;  // of the empty barriers: a fresh one lets pass
    for (int c0 = 0; c0 < K; c0 += cpc) {
      if (issued == kStages) {  // the ring is full: now the kernel before
        grid_dep_wait();
        grid_dep_launch();
      }
      const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&empty[st], ph));
      if (!got && lane == 0) atomicExch(V.err, 1);
      if (!got || *(volatile int*)&s_stop) break;
      if (lane == 0) {
        const uint32_t bytes = (uint32_t)(min(cpc, K - c0) * R * sizeof(cplx<MT>));
        fence_proxy_async();
        mbar_expect_tx(&full[st], bytes);
        bulk_copy_g2s(stage[st], seg + (size_t)c0 * R, bytes, &full[st]);
      }
      issued++;
      if (++st == kStages) {
        st = 0;
        ph ^= 1u;
      }
    }
    if (issued <= kStages) {
      grid_dep_wait();
      grid_dep_launch();
    }
    // the copies land before the CTA exits
    if (lane == 0)
      for (int cc = max(0, issued - kStages); cc < issued; cc++)
        mbar_wait_bounded(&full[cc % kStages], (uint32_t)(cc / kStages) & 1u);
    return;
  }
  const int g = lane % G, slot = lane / G;
  AT xr[RPG], xi[RPG];
  cplx<AT>* out = p + k0;
  grid_dep_wait();
  grid_dep_launch();
  if (done) {  // the consumers' vote; the producer sees it when a stage is given back
    if (*(volatile const int*)done) s_stop = 1;
    uint32_t cph = 0;
    if (!consumer_sync(&cbar, cph) || *(volatile int*)&s_stop) {
      if (lane == 0) mbar_arrive(&empty[0]);
      return;
    }
  }
#pragma unroll
  for (int t = 0; t < RPG; t++) {
    const int row = g + G * t;
    const cplx<AT> v = row < R ? xm[ls + row] : cplx<AT>();
    xr[t] = v.re;
    xi[t] = v.im;
  }
  int st = 0;
  uint32_t ph = 0;
  for (int c0 = 0; c0 < K; c0 += cpc) {
    const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&full[st], ph));
    if (!got) {
      if (lane == 0) atomicExch(V.err, 1);
      break;
    }
    const cplx<MT>* S = (const cplx<MT>*)stage[st];
    const int ncols = min(cpc, K - c0);
    // two columns per lane in flight: j and j + STEP
    for (int jb = warp * CPW; jb < ncols; jb += 2 * STEP) {
      AT a[4];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int j = jb + slot + u * STEP;
        AT ar = 0, ai = 0;
        if (j < ncols) {
          const cplx<MT>* col = S + j * R;
#pragma unroll
          for (int t = 0; t < RPG; t++) {
            const int row = g + G * t;
            if (row < R) acc_mac(ar, ai, col[row], xr[t], xi[t]);
          }
        }
        a[2 * u] = ar;
        a[2 * u + 1] = ai;
      }
      const int j = jb + slot;
      if constexpr (std::is_same<AT, float>::value) {
        dot_fold<2, G / 2>(a);
        dot_fold<1, G / 4>(a);
        float v = a[0];
#pragma unroll
        for (int o = G / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        // the quarters of the column's lanes: Re, Im of column j, Re, Im of column j + STEP
        const int jq = j + (g >= G / 2 ? STEP : 0);
        if (g % (G / 4) == 0 && jq < ncols) reinterpret_cast<float*>(out + c0 + jq)[g / (G / 4) & 1] = v;
      } else {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < 4; u++) a[u] = acc_add(a[u], acc_shfl_xor(a[u], o));
        if (g == 0) {
          if (j < ncols) out[c0 + j] = cplx<AT>(a[0], a[1]);
          if (j + STEP < ncols) out[c0 + j + STEP] = cplx<AT>(a[2], a[3]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
    if (++st == kStages) {
      st = 0;
      ph ^= 1u;
    }
  }
}

// t[task] = sum over the leaf entries of the task's block of p[kpos[e] + q], in leaf order
// (kpos is stored block-major, so a block's entries are consecutive). The grid covers the terms the
// blocks could have: the gather pass may start when this pass's last CTA has, and behind the CTAs
// that only return it does so when most sums are done. With a grid of the stored terms its streams
// slowed the sums' loads: 97 instead of 85 us per matvec on the 20480-triangle relief, 164 instead
// of 148 us on 34340; with the longer sums' entries in shared memory (cp.async) and the gather behind
// the last sum, 85 and 145 us, but 56 instead of 54 us on 10980 and 35 instead of 34 us on 5280.
template <typename AT>
__global__ void __launch_bounds__(256) seg_reduce_kernel(const int* __restrict__ task_b,
                                                         const int* __restrict__ t_off, int ntask_cap,
                                                         const int* __restrict__ t_total,
                                                         const int* __restrict__ ent_ptr,
                                                         const int* __restrict__ kpos,
                                                         const cplx<AT>* __restrict__ p, cplx<AT>* __restrict__ t,
                                                         const int* __restrict__ done) {
  grid_dep_wait();
  grid_dep_launch();
  if (done && *done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ntask_cap || i >= *t_total) return;
  const int b = task_b[i];
  const int q = i - t_off[b];
  const int e0 = ent_ptr[b], e1 = ent_ptr[b + 1];
  AT sr = 0, si = 0;
  int e = e0;
  // batches of 16: every load of a batch is issued before its first add (a block spans up to a
  // few hundred leaves); the adds keep the entry order, so any batching gives the same sums
  for (; e + 15 < e1; e += 16) {
    int kk[16];
#pragma unroll
    for (int u = 0; u < 16; u++) kk[u] = kpos[e + u];
    cplx<AT> v[16];
#pragma unroll
    for (int u = 0; u < 16; u++) v[u] = p[kk[u] + q];
#pragma unroll
    for (int u = 0; u < 16; u++) {
      sr = acc_add(sr, v[u].re);
      si = acc_add(si, v[u].im);
    }
  }
  for (; e + 3 < e1; e += 4) {
    const int k0 = kpos[e], k1 = kpos[e + 1], k2 = kpos[e + 2], k3 = kpos[e + 3];
    const cplx<AT> v0 = p[k0 + q], v1 = p[k1 + q], v2 = p[k2 + q], v3 = p[k3 + q];
    sr = acc_add(sr, v0.re);
    si = acc_add(si, v0.im);
    sr = acc_add(sr, v1.re);
    si = acc_add(si, v1.im);
    sr = acc_add(sr, v2.re);
    si = acc_add(si, v2.im);
    sr = acc_add(sr, v3.re);
    si = acc_add(si, v3.im);
  }
  for (; e < e1; e++) {
    const cplx<AT> v = p[kpos[e] + q];
    sr = acc_add(sr, v.re);
    si = acc_add(si, v.im);
  }
  t[i] = cplx<AT>(sr, si);
}

// Gather pass: y[leaf rows] = -x/2 + S_A x[a_idx] + S_B t[b_idx] (+ transposed dense blocks), or
// b - that; optional fused FP64 dot partials (conj(a).y, conj(y).b, |y|^2) per leaf.
//
// Warp-specialised: kWarps consumer warps compute, one producer warp feeds the copy ring. For
// each chunk (at most kPCols columns) the producer waits until the consumers have released the
// stage (its "empty" mbarrier, one arrival per consumer warp), issues the chunk's bulk copy, then
// gathers its column multipliers (x[idx] or t[idx]) into the stage's multiplier buffer with
// cp.async; the stage's "full" mbarrier expects the copy's bytes and one arrival per producer
// lane. A padding column (index -1) is zero in the segment, so it gathers any valid multiplier
// (element 0). The compute uses the dot pass's layout: G lanes per column, each lane summing RPG
// rows, 32 / G columns per warp step.
constexpr int kGatherThreads = kThreads + 32;
#ifndef AC3D_GATHER_MIN_CTAS
#define AC3D_GATHER_MIN_CTAS 4
#endif

// The grid is persistent: the CTAs that fit on the device at once (P) take the row leaves in the
// order V.order (decreasing work), CTA k the leaves k, 2P - 1 - k, 2P + k, ... (a serpentine over
// the sorted list). The producer goes on to the next leaf's chunks as soon as it has issued the
// current leaf's last one (it loads the next leaf's geometry while it streams the current one),
// so an SM slot never waits for an empty ring between leaves. Every stage carries its leaf slot,
// column count and first / last flags; the consumer warps finish a leaf (row sums, epilogue, dot
// partials) when they consume its last chunk, synchronising among themselves on an mbarrier
// while the producer keeps streaming. A leaf's row sums have a fixed order (each warp's columns
// in chunk order, then the warps in order), and the last CTA to finish reduces the per-leaf dot
// partials in fixed order, so results are reproducible. Against one CTA per leaf this takes 104
// instead of 101 us for back-to-back matvecs without overlap, but 6.7% less time per BiCGSTAB
// iteration inside the solve and 3% more served solves/s over the relief sweep.
constexpr int kPCols = 128;                  // multiplier columns per stage (chunks are capped at it)
constexpr int kPProdCols = kPCols / 32;      // per producer lane
constexpr int kLeafSlots = kStages + 1;      // leaves whose chunks can be in the ring at once

// The gather pass's directions: A x, and A^T x with the near field from its transposed copy or in place
enum : int { kForward = 0, kTransposed = 1, kInPlace = 2 };

struct StageMeta {
  int slot, ncols, first, last;  // slot < 0: no more leaves
};

template <typename MT, typename VT, typename AT, int TRANS, int RPL>
__global__ void __launch_bounds__(kGatherThreads, AC3D_GATHER_MIN_CTAS) seg_gather_persist_kernel(
    SegView V, int nleaf, const cplx<MT>* __restrict__ near, const cplx<MT>* __restrict__ lrseg,
    const cplx<AT>* __restrict__ t, const cplx<VT>* __restrict__ x, const cplx<AT>* __restrict__ xm,
    cplx<VT>* __restrict__ y, const cplx<VT>* __restrict__ bminus, const cplx<VT>* __restrict__ dot_a,
    const cplx<VT>* __restrict__ dot_b, double* partials, double* red5, unsigned* ticket,
    const int* __restrict__ done) {
  constexpr int G = DotShape<RPL>::G, RPG = DotShape<RPL>::RPG;
  constexpr int CPW = 32 / G;
  constexpr int STEP = kWarps * CPW;
  constexpr int RMAX = 32 * RPL;
  extern __shared__ __align__(128) unsigned char dsmem[];
  auto stage = reinterpret_cast<unsigned char(*)[kStageBytes]>(dsmem);
  __shared__ __align__(8) uint64_t full[kStages];
  __shared__ __align__(8) uint64_t empty[kStages];
  __shared__ __align__(8) uint64_t cbar;  // consumer barrier, kThreads arrivals per phase
  __shared__ __align__(16) unsigned char zraw[kStages * kPCols * sizeof(cplx<AT>)];
  auto zbuf = reinterpret_cast<cplx<AT>(*)[kPCols]>(zraw);
  __shared__ __align__(16) unsigned char praw[kWarps * RMAX * sizeof(cplx<AT>)];
  cplx<AT>* part = reinterpret_cast<cplx<AT>*>(praw);
  __shared__ StageMeta meta[kStages];
  __shared__ int slot_leaf[kLeafSlots], slot_ls[kLeafSlots], slot_R[kLeafSlots];
  __shared__ double sdot[kWarps][5];
  __shared__ int s_fail;
  __shared__ bool s_last;
  grid_dep_launch();  // as in the one-CTA-per-leaf pass
  // the vote of the CTA: the Givens step beside this pass may set the flag while its warps read it
  if (__syncthreads_or(done && *(volatile const int*)done)) {
    grid_dep_wait();
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int P = gridDim.x, kc = blockIdx.x;
  // geometry of the n-th leaf of this CTA in the serpentine (leaf -1: none left)
  struct LeafGeo {
    int leaf, ls, R, a_cols, b_cols, a_k, b_k;
    long long a_seg, b_seg;
  };
  auto leaf_geo = [&](int n) -> LeafGeo {
    LeafGeo o{-1, 0, 0, 0, 0, 0, 0, 0, 0};
    const long long li = (long long)n * P + ((n & 1) ? P - 1 - kc : kc);
    if (li >= nleaf) return o;
    o.leaf = V.order[li];
    o.ls = V.leaf_start[o.leaf];
    o.R = V.leaf_start[o.leaf + 1] - o.ls;
    if (!TRANS) {
      o.a_k = V.a_kptr[o.leaf];
      o.a_cols = V.a_kptr[o.leaf + 1] - o.a_k;
      o.a_seg = V.a_seg[o.leaf];
    }
    o.b_k = V.b_kptr[o.leaf];
    o.b_cols = V.b_kptr[o.leaf + 1] - o.b_k;
    o.b_seg = V.b_seg[o.leaf];
    return o;
  };
  if (tid == 0) {
    for (int st = 0; st < kStages; st++) {
      mbar_init(&full[st], 1 + 32);
      mbar_init(&empty[st], kWarps);
    }
    mbar_init(&cbar, kThreads);
    s_fail = 0;
    fence_barrier_init();
  }
  __syncthreads();

  if (warp == kWarps) {
    // ---- producer warp: every leaf's chunks in order, with no gap between leaves. Its own time per
    // chunk bounds the pass on small meshes, so places advance by additions (no divisions per chunk) and
    // the column indices are loaded a chunk ahead (the multipliers' addresses wait for them).
    // Matvec, before and after: 30.9 and 29.5 us on 5280 triangles, 118 and 105 us on 10680 in 128
    // leaves, 1019 and 1005 us on 118680
    bool waited = false, failed = false;
    int st = 0, nissued = 0;
    uint32_t ph = 1;  // of the empty barriers: a fresh one lets pass
    int kk[kPProdCols];
    auto load_idx = [&](const int* idx, int ncols) {
#pragma unroll
      for (int u = 0; u < kPProdCols; u++) kk[u] = lane + 32 * u < ncols ? idx[lane + 32 * u] : 0;
    };
    auto acquire = [&]() {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&empty[st], ph))) {
        if (lane == 0) atomicExch(&s_fail, 1);
        failed = true;
      }
      return !failed;
    };
    auto advance = [&]() {
      nissued++;
      if (++st == kStages) {
        st = 0;
        ph ^= 1u;
      }
    };
    int slot = 0;
    auto chunk_cols = [](const LeafGeo& o) { return min(kPCols, max(2, (int)(kStageBytes / sizeof(cplx<MT>)) / o.R & ~1)); };
    LeafGeo nxt = leaf_geo(0);
    int ncpc = nxt.leaf >= 0 ? chunk_cols(nxt) : 2;
    load_idx(nxt.a_cols ? V.a_idx + nxt.a_k : V.b_idx + nxt.b_k, min(ncpc, nxt.a_cols ? nxt.a_cols : nxt.b_cols));
    for (int n = 0; !failed && nxt.leaf >= 0; n++) {
      const LeafGeo cur = nxt;
      const int R = cur.R, cpc = ncpc;
      nxt = leaf_geo(n + 1);  // in flight while this leaf streams
      if (lane == 0) {
        slot_leaf[slot] = cur.leaf;
        slot_ls[slot] = cur.ls;
        slot_R[slot] = R;
      }
      const bool two = cur.a_cols > 0 && cur.b_cols > 0;
      bool first = true;
      for (int region = cur.a_cols > 0 ? 0 : 1; region < 2 && !failed; region++) {
        int left = region ? cur.b_cols : cur.a_cols;
        if (region && left == 0 && cur.a_cols > 0) break;
        const cplx<MT>* src = region ? lrseg + cur.b_seg : near + cur.a_seg;
        const int* idx = region ? V.b_idx + cur.b_k : V.a_idx + cur.a_k;
        const cplx<AT>* z = region ? t : xm;
        // (a leaf with no columns still gets one stage)
        do {
          if (!acquire()) break;
          const int ncols = min(cpc, left);
          left -= ncols;
          if (lane == 0) {
            meta[st] = StageMeta{slot, ncols, first, left == 0 && (region || !two)};
            const uint32_t bytes = (uint32_t)(ncols * R * sizeof(cplx<MT>));
            fence_proxy_async();
            mbar_expect_tx(&full[st], bytes);  // zero bytes: a plain arrival
            if (bytes) bulk_copy_g2s(stage[st], src, bytes, &full[st]);
          }
          if (region && ncols > 0 && !waited) {  // t comes from the preceding kernel
            grid_dep_wait();
            waited = true;
          }
#pragma unroll
          for (int u = 0; u < kPProdCols; u++) {
            const int col = lane + 32 * u;
            if (col < ncols) cp_async_elem<sizeof(cplx<AT>)>(&zbuf[st][col], z + max(kk[u], 0));
          }
          cp_async_arrive_noinc(&full[st]);
          advance();
          first = false;
          src += (size_t)ncols * R;
          idx += ncols;
          if (left > 0) {
            load_idx(idx, min(cpc, left));
          } else if (region == 0 && two) {
            load_idx(V.b_idx + cur.b_k, min(cpc, cur.b_cols));
          } else if (nxt.leaf >= 0) {
            ncpc = chunk_cols(nxt);
            load_idx(nxt.a_cols ? V.a_idx + nxt.a_k : V.b_idx + nxt.b_k, min(ncpc, nxt.a_cols ? nxt.a_cols : nxt.b_cols));
          }
        } while (left > 0);
      }
      if (++slot == kLeafSlots) slot = 0;
    }
    if (!failed && acquire()) {  // the end marker
      if (lane == 0) {
        meta[st] = StageMeta{-1, 0, 1, 1};
        mbar_expect_tx(&full[st], 0);
      }
      cp_async_arrive_noinc(&full[st]);
      advance();
    }
    if (!waited) grid_dep_wait();
    cp_async_wait_all();
    if (lane == 0)
      for (int cc = max(0, nissued - kStages); cc < nissued; cc++)
        mbar_wait_bounded(&full[cc % kStages], (uint32_t)(cc / kStages) & 1u);
  } else {
    // ---- consumer warps
    const int g = lane % G, slot = lane / G;
    AT ar[RPG], ai[RPG];
#pragma unroll
    for (int q = 0; q < RPG; q++) ar[q] = ai[q] = 0;
    int leaf = -1, ls = 0, R = 0;
    uint32_t cphase = 0;
    bool cok = true;
    int s = kStages - 1;
    uint32_t ph = 1;
    for (;;) {
      if (++s == kStages) s = 0;
      if (s == 0) ph ^= 1u;
      const bool got = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], ph));
      if (!got) {
        if (lane == 0) atomicExch(&s_fail, 1);
        break;
      }
      const StageMeta mt = meta[s];
      if (mt.slot < 0) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        break;
      }
      if (mt.first) {
        leaf = slot_leaf[mt.slot];
        ls = slot_ls[mt.slot];
        R = slot_R[mt.slot];
      }
      const int ncols = mt.ncols;
      const cplx<MT>* S = (const cplx<MT>*)stage[s];
      const cplx<AT>* Z = zbuf[s];
      for (int jb = warp * CPW; jb < ncols; jb += 2 * STEP) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int j = jb + slot + u * STEP;
          if (j < ncols) {
            const cplx<AT> zz = Z[j];
            const cplx<MT>* col = S + j * R;
#pragma unroll
            for (int q = 0; q < RPG; q++) {
              const int row = g + G * q;
              if (row < R) acc_mac(ar[q], ai[q], col[row], zz.re, zz.im);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (!mt.last) continue;
      // ---- the leaf is complete: its row sums and epilogue
#pragma unroll
      for (int o = G; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < RPG; q++) {
          ar[q] = acc_add(ar[q], acc_shfl_xor(ar[q], o));
          ai[q] = acc_add(ai[q], acc_shfl_xor(ai[q], o));
        }
      if (slot == 0) {
#pragma unroll
        for (int q = 0; q < RPG; q++) {
          const int row = g + G * q;
          if (row < R) part[warp * R + row] = cplx<AT>(ar[q], ai[q]);
        }
      }
#pragma unroll
      for (int q = 0; q < RPG; q++) ar[q] = ai[q] = 0;
      __syncwarp();
      if (TRANS) {
        AT tr[RPL], ti[RPL];
#pragma unroll
        for (int jr = 0; jr < RPL; jr++) tr[jr] = ti[jr] = 0;
        // near: the transposed copy, so that the lanes' columns of a row are consecutive; the rows of a
        // warp's blocks in order, U loads in flight (as many as the 56 registers hold). The blocks
        // themselves (kInPlace: the device has no room for the copy) are read a column per lane.
        // Transposed matvec, from the blocks and from the copy: 149.6 and 101.3 us on the
        // 20480-triangle relief, 65.7 and 37.5 us on 5280 triangles
        for (int it = V.trn_ptr[leaf] + warp; it < V.trn_ptr[leaf + 1]; it += kWarps) {
          const int b = V.trn[it];
          const int4 blk = V.blocks_d[b];
          const int m = blk.y - blk.x;
          const cplx<AT>* xs = xm + blk.x;
          const cplx<MT>* D = near + V.near_off[b];
          if constexpr (TRANS == kInPlace) {
#pragma unroll
            for (int jr = 0; jr < RPL; jr++) {
              const int col = lane + 32 * jr;
              if (col < R) {
                const cplx<MT>* Dc = D + (long long)col * m;
                for (int r = 0; r < m; r++) {
                  const cplx<AT> zz = xs[r];
                  acc_mac(tr[jr], ti[jr], Dc[r], zz.re, zz.im);
                }
              }
            }
            continue;
          }
          constexpr int U = sizeof(AT) > 4 ? 2 : RPL > 2 ? 4 : 8;
          for (int r0 = 0; r0 < m; r0 += U) {
#pragma unroll
            for (int jr = 0; jr < RPL; jr++) {
              const int col = min(lane + 32 * jr, R - 1);
              cplx<MT> d[U];
              cplx<AT> z[U];
#pragma unroll
              for (int u = 0; u < U; u++) {
                const int r = min(r0 + u, m - 1);
                d[u] = D[(long long)r * R + col];
                z[u] = xs[r];
              }
#pragma unroll
              for (int u = 0; u < U; u++)
                if (r0 + u < m) acc_mac(tr[jr], ti[jr], d[u], z[u].re, z[u].im);
            }
          }
        }
#pragma unroll
        for (int jr = 0; jr < RPL; jr++) {
          const int col = lane + 32 * jr;
          if (col < R) {
            cplx<AT>& pc = part[warp * R + col];
            pc = cplx<AT>(acc_add(pc.re, tr[jr]), acc_add(pc.im, ti[jr]));
          }
        }
      }
      if (!(cok = consumer_sync(&cbar, cphase))) break;
      double d[5] = {0, 0, 0, 0, 0};
      if (tid < R) {
        const int r = tid;
        AT sr = 0, si = 0;
        for (int w = 0; w < kWarps; w++) {
          sr = acc_add(sr, part[w * R + r].re);
          si = acc_add(si, part[w * R + r].im);
        }
        const cplx<VT> xv = x[ls + r];
        VT yr = acc_to<VT>(sr) - VT(0.5) * xv.re;
        VT yi = acc_to<VT>(si) - VT(0.5) * xv.im;
        if (bminus) {
          const cplx<VT> bv = bminus[ls + r];
          yr = bv.re - yr;
          yi = bv.im - yi;
        }
        const cplx<VT> o(yr, yi);
        y[ls + r] = o;
        const double oyr = (double)o.re, oyi = (double)o.im;
        if (dot_a) {
          const cplx<VT> a = dot_a[ls + r];
          d[0] += (double)a.re * oyr + (double)a.im * oyi;
          d[1] += (double)a.re * oyi - (double)a.im * oyr;
        }
        if (dot_b) {
          const cplx<VT> bb = dot_b[ls + r];
          d[2] += oyr * (double)bb.re + oyi * (double)bb.im;
          d[3] += oyr * (double)bb.im - oyi * (double)bb.re;
        }
        d[4] += oyr * oyr + oyi * oyi;
      }
      if (partials) {
        warp_sum5(d, sdot[warp], 32 * warp < R);
        if (!(cok = consumer_sync(&cbar, cphase))) break;
        if (tid < 5) {
          double sum = 0;
          for (int w = 0; w < kWarps; w++) sum += sdot[w][tid];
          partials[(size_t)leaf * 5 + tid] = sum;
        }
      }
      if (!(cok = consumer_sync(&cbar, cphase))) break;  // part and sdot are free for the next leaf
    }
    if (!cok && lane == 0) atomicExch(&s_fail, 1);
  }
  __syncthreads();
  if (s_fail && tid == 0) atomicExch(V.err, 1);
  if (partials && red5) {
    // the last CTA to finish reduces all leaves' partials in fixed order into red5
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      const bool consumer = warp < kWarps;
      double acc[5] = {0, 0, 0, 0, 0};
      if (consumer)
        for (int l = tid; l < nleaf; l += kThreads)
          for (int i = 0; i < 5; i++) acc[i] += __ldcg(&partials[(size_t)l * 5 + i]);
      __syncthreads();
      if (consumer) warp_sum5(acc, sdot[warp], 32 * warp < nleaf);
      __syncthreads();
      if (tid < 5) {
        double sum = 0;
        for (int w = 0; w < kWarps; w++) sum += sdot[w][tid];
        red5[tid] = sum;
      }
      if (tid == 0) *ticket = 0u;
    }
  }
}

static std::atomic<int> g_sms{0};
int device_sm_count() {
  int n = g_sms.load();
  if (!n) {
    int dev = 0;
    AC3D_CUDA(cudaGetDevice(&dev));
    AC3D_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    g_sms.store(n);
  }
  return n;
}

constexpr size_t kRingBytes = (size_t)kStages * kStageBytes;

template <typename MT, typename VT, typename AT, int RPL>
static void set_smem_attrs_rpl() {
  AC3D_CUDA(cudaFuncSetAttribute(seg_dot_kernel<MT, AT, RPL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kRingBytes));
  // the largest shared-memory carveout, so that four CTAs of the ring size fit on an SM
  AC3D_CUDA(cudaFuncSetAttribute(seg_dot_kernel<MT, AT, RPL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 100));
  for (auto kern : {seg_gather_persist_kernel<MT, VT, AT, kForward, RPL>, seg_gather_persist_kernel<MT, VT, AT, kTransposed, RPL>,
                    seg_gather_persist_kernel<MT, VT, AT, kInPlace, RPL>}) {
    AC3D_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    AC3D_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRingBytes));
  }
}

template <typename MT, typename VT, typename AT>
static void set_smem_attrs() {
  set_smem_attrs_rpl<MT, VT, AT, 1>();
  set_smem_attrs_rpl<MT, VT, AT, 2>();
  set_smem_attrs_rpl<MT, VT, AT, 4>();
  set_smem_attrs_rpl<MT, VT, AT, 8>();
}

void prepare_matvec_kernels() {
  // once per process (one device per process); contexts on other threads wait for the first call
  static std::once_flag once;
  std::call_once(once, [] {
    set_smem_attrs<float, float, float>();
    set_smem_attrs<float, double, df32>();
    set_smem_attrs<float, double, float>();
  });
}

// CTAs per leaf of the dot pass (a column's dot is the same in any of them). Below two CTAs per SM
// always more: 256 leaves of 5280 triangles 35.6 us a matvec with one CTA each and 31.0 with two, 64 leaves of
// 1280 triangles 14.3 and 13.3 with eight. Up to a full wave of four per SM while a part keeps twice
// the ring's bytes: 512 leaves of 10980 triangles (190 KB) 55.0 and 51.1 us with two, but four for
// the 256 leaves of 5280 (150 KB) 34.7 us.
static int dot_parts(int nleaf, size_t bytes) {
  const int sms = device_sm_count();
  int parts = 1;
  while (parts < 8 && (nleaf * parts < 2 * sms ||
                       (nleaf * parts < 4 * sms && bytes / ((size_t)nleaf * parts) >= 2 * kRingBytes)))
    parts *= 2;
  return parts;
}

template <typename AT>
static void launch_reduce(const DevPartition& DP, const DevHMat& H, bool tr, const cplx<AT>* p, cplx<AT>* t,
                          const int* done, cudaStream_t s, bool pdl) {
  launch_k(pdl, seg_reduce_kernel<AT>, dim3((int)((H.task_cap + 255) / 256)), dim3(256), 0, s, H.task_b.as<int>(),
           H.t_off.as<int>(), (int)H.task_cap, H.t_off.as<int>() + DP.na,
           tr ? DP.blk_fw_ptr.as<int>() : DP.blk_tr_ptr.as<int>(), tr ? H.kpos_f.as<int>() : H.kpos_t.as<int>(), p, t,
           done);
}
void launch_reduce_f64(const DevPartition& DP, const DevHMat& H, bool tr, const void* p, void* t, const int* done,
                       cudaStream_t s, bool pdl) {
  launch_reduce<double>(DP, H, tr, (const cd*)p, (cd*)t, done, s, pdl);
}

template <typename MT, typename VT, typename AT, int RPL>
static void mv_t(const DevPartition& DP, const DevHMat& H, bool tr, const void* x, void* y, const void* bminus,
                 const MatvecEpilogue& ep, const int* done, void* tvec, cudaStream_t s, const void* x32, bool pdl) {
  SegView v;
  v.leaf_start = DP.leaf_start.as<int>();
  v.a_seg = DP.near_seg.as<long long>();
  v.a_kptr = DP.didx_ptr.as<int>();
  v.a_idx = DP.didx.as<int>();
  v.blocks_d = DP.blocks_d.as<int4>();
  const int mode = !tr ? kForward : H.nearT.p ? kTransposed : kInPlace;
  v.near_off = mode == kTransposed ? DP.near_off_t.as<long long>() : DP.near_off.as<long long>();
  v.trn_ptr = DP.tr_near_ptr.as<int>();
  v.trn = DP.tr_near.as<int>();
  v.err = H.err.as<int>();
  const cplx<MT>* useg = H.useg.as<cplx<MT>>();
  const cplx<MT>* vseg = H.vseg.as<cplx<MT>>();
  cplx<AT>* t = (cplx<AT>*)tvec;
  cplx<AT>* p = H.pbuf.as<cplx<AT>>();
  // column multipliers taken from x in the accumulator type: x itself, its FP32 shadow x32 (FP64
  // vectors on FP32 arithmetic) or its double-float copy
  const cplx<AT>* xm = x32 ? (const cplx<AT>*)x32 : (const cplx<AT>*)x;
  if constexpr (std::is_same<AT, df32>::value) {
    launch_k(pdl, to_df_kernel, dim3((DP.ne + 255) / 256), dim3(256), 0, s, DP.ne, (const cd*)x,
             H.xdf.as<cplx<df32>>());
    xm = H.xdf.as<cplx<df32>>();
  }
  if (DP.na > 0) {
    // dot pass over the segments on the input side: V by column leaf (forward), U by row leaf
    SegView d = v;
    d.b_seg = tr ? H.seg_f.as<long long>() : H.seg_t.as<long long>();
    d.b_kptr = tr ? H.kseg_f.as<int>() : H.kseg_t.as<int>();
    d.order = tr ? H.order_rows.as<int>() : H.order_cols.as<int>();
    launch_k(pdl, seg_dot_kernel<MT, AT, RPL>, dim3(DP.nleaf, dot_parts(DP.nleaf, (tr ? H.useg : H.vseg).bytes)),
             dim3(kThreads + 32), kRingBytes, s, d,
             tr ? useg : vseg, xm, p, done);
    launch_reduce<AT>(DP, H, tr, p, t, done, s, pdl);
  }
  v.b_seg = tr ? H.seg_t.as<long long>() : H.seg_f.as<long long>();
  v.b_kptr = tr ? H.kseg_t.as<int>() : H.kseg_f.as<int>();
  v.b_idx = tr ? H.vidx.as<int>() : H.uidx.as<int>();
  v.order = tr ? H.order_cols.as<int>() : H.order_rows.as<int>();
  const cplx<AT>* tc = t;
  // the gather reads x and the done flag before its wait, which needs the dot and reduce passes
  // between it and the kernel that wrote them; without low-rank blocks it is an ordinary launch
  // one resident wave: as many CTAs as fit on the device at once (each takes a share of the leaves)
  auto kern = mode == kForward      ? seg_gather_persist_kernel<MT, VT, AT, kForward, RPL>
              : mode == kTransposed ? seg_gather_persist_kernel<MT, VT, AT, kTransposed, RPL>
                                    : seg_gather_persist_kernel<MT, VT, AT, kInPlace, RPL>;
  static std::atomic<int> per_sm[3] = {{0}, {0}, {0}};
  int nb = per_sm[mode].load();
  if (!nb) {
    AC3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, kGatherThreads, kRingBytes));
    nb = std::max(nb, 1);
    per_sm[mode].store(nb);
  }
  const int P = std::min(DP.nleaf, nb * device_sm_count());
  launch_k(pdl && DP.na > 0, kern, dim3(P), dim3(kGatherThreads), kRingBytes, s, v, DP.nleaf,
           (const cplx<MT>*)(mode == kTransposed ? H.nearT : H.near).as<cplx<MT>>(),
           tr ? vseg : useg, tc, (const cplx<VT>*)x, xm, (cplx<VT>*)y, (const cplx<VT>*)bminus,
           (const cplx<VT>*)ep.dot_a, (const cplx<VT>*)ep.dot_b, ep.partials, ep.red5, H.ticket.as<unsigned>(), done);

}

template <typename MT, typename VT, typename AT>
static void mv_rpl(const DevPartition& DP, const DevHMat& H, bool tr, const void* x, void* y, const void* bminus,
                   const MatvecEpilogue& ep, const int* done, void* tvec, cudaStream_t s, const void* x32,
                   bool pdl) {
  const int rpl = (DP.max_leaf + 31) / 32;
  if (rpl <= 1)
    mv_t<MT, VT, AT, 1>(DP, H, tr, x, y, bminus, ep, done, tvec, s, x32, pdl);
  else if (rpl <= 2)
    mv_t<MT, VT, AT, 2>(DP, H, tr, x, y, bminus, ep, done, tvec, s, x32, pdl);
  else if (rpl <= 4)
    mv_t<MT, VT, AT, 4>(DP, H, tr, x, y, bminus, ep, done, tvec, s, x32, pdl);
  else
    mv_t<MT, VT, AT, 8>(DP, H, tr, x, y, bminus, ep, done, tvec, s, x32, pdl);
}

// vec64: 0 FP32 vectors; 1 FP64 vectors (FP64 storage: FP64 arithmetic, matvec64.cu; FP32 storage: the
// double-float residual); 2 FP64 vectors on FP32 storage with FP32 arithmetic, the multipliers
// taken from the FP32 shadow x32 of x. pdl: launch the passes as programmatic dependents (the
// kernel before the first pass then must follow the same protocol, see launch.cuh).
void launch_matvec_ex(const DevPartition& DP, const DevHMat& H, bool transposed, int vec64, const void* x, void* y,
                      const void* b_minus, const MatvecEpilogue& ep, const int* done, cudaStream_t s,
                      const void* x32, bool pdl) {
  if (H.prec == PREC_FP64) {
    if (!vec64) throw Error(3, "internal: FP64 H-matrix needs FP64 vectors");
    launch_matvec_f64(DP, H, transposed, x, y, b_minus, ep, done, s, pdl);
  } else if (vec64 == 2) {
    if (!x32) throw Error(3, "internal: FP32 shadow of the matvec input missing");
    mv_rpl<float, double, float>(DP, H, transposed, x, y, b_minus, ep, done, H.tvec.p, s, x32, pdl);
  } else if (vec64) {
    // FP32 H-matrix with FP64 vectors (refinement residuals): double-float arithmetic
    mv_rpl<float, double, df32>(DP, H, transposed, x, y, b_minus, ep, done, H.tvec64.p, s, nullptr, pdl);
  } else {
    mv_rpl<float, float, float>(DP, H, transposed, x, y, b_minus, ep, done, H.tvec.p, s, nullptr, pdl);
  }
}

void launch_matvec(const DevPartition& DP, const DevHMat& H, int ne, bool transposed, int vec64, const void* x,
                   void* y, const void* b_minus, const MatvecEpilogue& ep, cudaStream_t s) {
  (void)ne;
  launch_matvec_ex(DP, H, transposed, vec64, x, y, b_minus, ep, nullptr, s, nullptr, false);
}

int matvec_grid(const DevPartition& DP, bool) { return DP.nleaf; }

}  // namespace ac3d
