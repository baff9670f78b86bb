// Mixed-precision assembly with FP64-accurate entries: near-field entries, and the admissible
// blocks' rows and columns with the ACA recursion, evaluated in double-float arithmetic (about 47
// bits, on the FP32 pipes); everything is stored in complex FP32. Near-field entries of nearly
// coplanar neighbours cancel in r.n, so FP32 evaluation from FP64 displacements is not enough
// there (5.6e-5 instead of 1.3e-5 from the FP64 path on a 5280-triangle relief at 3.5 kHz).
//
// The ACA sequence is the reference's (compute_ACA_block, aca.cpp:38-82, argmax rules
// aca.cpp:9-36) exactly as the FP32 / FP64 kernels of assemble.cu run it: first row pivot 0;
// v = row - U(i,:) V; column pivot j = first index of max |v|^2; V row = v / v_j (v itself when
// v_j == 0); u = column - U V(:, j); err += |u|^2 |v|^2 + 2 sum_q |u^T U_q| |v V_q^T|; stop when
// sqrt(|u|^2 |v|^2 / err) <= eps, dropping the converging term; next row pivot = first max of
// |u|^2 over unused rows. Entries, residuals, the pivot magnitudes and the norms are double-float,
// so the pivots and ranks are the FP64 path's (the two differ only where two candidates agree to
// about 1e-12); the cross terms of the error estimate are FP32 sums of the leading parts (they
// only scale err). The estimate, the norms and the stopping test are double-float too (the FP64
// pipes of GB300 are too slow to hold them), the test as |u|^2 |v|^2 <= eps^2 err. The terms live in a double-float pool while the recursion needs them; packing
// rounds them to the FP32 per-leaf segments the matvec streams.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "df2.cuh"
#include "entry_df.cuh"
#include "internal.h"

namespace ac3d {

namespace {
constexpr int kDfThreads = 256;
constexpr int kDfWarps = kDfThreads / 32;
constexpr int kSmallThreads = 128;  // CTAs of the 1-, 2- and 4-warp groups
// Blocks are run by groups of W warps, W by the block's larger side: 1 up to 64, 2 up to 128, 4 up to
// 256 (so that a thread owns at most two rows and two columns), 8 above.
constexpr int kGroups = 4;
}  // namespace

struct AcaDfArgs {
  const double4* cen;          // FP64 centroids and vertices: the exactly-zero block test
  const double4* va;
  const ElemGeo<double>* eg;
  const DfPt* pts;             // double-float centroids (rows)
  const DfElem* el;            // double-float quadrature points and normals (columns)
  const float4* tab;           // df_sincos table in global memory (copied to shared memory)
  const int4* blocks;
  const int* order;            // blocks grouped by W = 8, 4, 2, 1
  int split[kGroups];          // blocks per group
  df64 k;
  df64 eps2;       // eps^2 as a double-float (the stopping test)
  int maxk;
  int iter_cap;
  df2* pool;       // terms u | v, complex double-floats packed as (re, im)
  long long pool_cap;
  unsigned long long* pool_used;
  long long* term_off;
  int* rank;
  int* status;
  int* passes;     // per block: rows (and columns) evaluated, or null
  unsigned* next;  // of each class of small blocks: the first one not taken
  int zero_guard;  // boundary blocks: v kept when v_j == 0 and exactly-zero blocks skipped
};

// The CTA's copy of the df_sincos table. A function's own shared variable, so that out-of-line code
// reads it with shared-memory loads.
__device__ __forceinline__ float4* s_table() {
  __shared__ float4 s_tab[kDfTab];
  return s_tab;
}
__device__ __forceinline__ void load_table(const float4* __restrict__ g) {
  float4* s = s_table();
  for (int i = threadIdx.x; i < kDfTab; i += blockDim.x) s[i] = g[i];
  __syncthreads();
}

// Exactly-zero block (all source elements in one axis-aligned plane that holds every target
// point, judged on the FP64 geometry; see aca_kernel): evaluated by the `count` threads
// t0, t0 + step, ... of a warp or CTA; `all` reduces the verdict over them.
template <typename All>
__device__ __forceinline__ bool zero_block(const AcaDfArgs& A, int rs, int m, int cs, int n, int t0, int step,
                                           All all) {
  // the three planes together, the points first: almost every block fails there, after one round of loads
  const double4 a0 = A.va[cs];
  bool x = true, y = true, z = true;
  for (int j = t0; j < n; j += step) {
    const double4 a = A.va[cs + j];
    x = x && a.x == a0.x;
    y = y && a.y == a0.y;
    z = z && a.z == a0.z;
  }
  for (int i = t0; i < m; i += step) {
    const double4 p = A.cen[rs + i];
    x = x && p.x == a0.x;
    y = y && p.y == a0.y;
    z = z && p.z == a0.z;
  }
  for (int d = 0; d < 3; d++) {
    bool ok = d == 0 ? x : (d == 1 ? y : z);
    if (!all(ok)) continue;
    for (int j = t0; j < n && ok; j += step) ok = A.eg[cs + j].ab[d] == 0.0 && A.eg[cs + j].ac[d] == 0.0;
    if (all(ok)) return true;
  }
  return false;
}

__device__ __forceinline__ df64 shfl_df(df64 v, int src) {
  return {__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src)};
}

// a * b of two FP32 values, exactly, as a double-float
__device__ __forceinline__ df64 df_prod_ff(float a, float b) {
  float p, e;
  two_prod(a, b, p, e);
  return {p, e};
}

// The ACA stopping test of the FP64 path, sqrt(|u|^2 |v|^2 / err) <= eps, as uv <= eps^2 err
// without a square root or a division; with err = 0 (then uv = 0) the FP64 test sees 0 / 0 and
// does not stop, and neither does this one.
__device__ __forceinline__ bool aca_converged(df64 uv, df64 err, df64 eps2) {
  return !df_is_zero(err) && !(uv > eps2 * err);
}

// (value, index) argmax over the warp: larger value wins, smaller index on ties. Values are
// non-negative double-floats, or -1 for a lane without one; three integer reductions on keys in
// the values' order (-1 below 0, the low part with -0 = +0) instead of a butterfly of triples.
__device__ __forceinline__ void warp_argmax_df(df64& val, int& idx) {
  const unsigned hk = val.hi < 0.0f ? 0u : __float_as_uint(val.hi + 0.0f) + 1u;
  const unsigned hm = __reduce_max_sync(0xffffffffu, hk);
  const unsigned lb = __float_as_uint(val.lo + 0.0f);
  const unsigned lk = hk == hm ? ((lb >> 31) ? ~lb : lb | 0x80000000u) : 0u;
  const unsigned lm = __reduce_max_sync(0xffffffffu, lk);
  const unsigned best = hk == hm && lk == lm ? (unsigned)idx : 0xffffffffu;
  idx = (int)__reduce_min_sync(0xffffffffu, best);
  val.hi = hm == 0u ? -1.0f : __uint_as_float(hm - 1u);
  val.lo = __uint_as_float((lm >> 31) ? lm & 0x7fffffffu : ~lm);
}

// Sums of two double-floats over the warp by butterfly; every lane ends with the same values (the
// double-float add is commutative bit for bit: TwoSum's error term is exact).
__device__ __forceinline__ void warp_sum2_df(df64& x, df64& y) {
  df2 v = df2_make(x, y);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = v + df2{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
  x = df2_x(v);
  y = df2_y(v);
}

// FP32 complex product of the leading parts (re, im): acc += a b
__device__ __forceinline__ void lead_fma(float& re, float& im, f2 a, f2 b) {
  re = fmaf(f2_x(a), f2_x(b), re);
  re = fmaf(-f2_y(a), f2_y(b), re);
  im = fmaf(f2_x(a), f2_y(b), im);
  im = fmaf(f2_y(a), f2_x(b), im);
}

// The three quadrature-point pairs of cnt entries, 3 cnt items spread over the T threads of a
// group: entry e is the pair (pts + e ps, el + e es), ps and es 0 or 1; item 3 e + h goes to
// b0[3 e + h] (first point) and b1[3 e + h] (second point), shared-memory addresses. One out-of-line
// copy serves every group width and both directions.
__device__ __noinline__ void eval_items(df64 k, const DfPt* __restrict__ pts, int ps, const DfElem* __restrict__ el,
                                        int es, int cnt, int tid, int T, uint32_t b0, uint32_t b1) {
  const df2 kk = df2_dup(k);
  const float4* tab = s_table();
#pragma unroll 1
  for (int it = tid; it < 3 * cnt; it += T) {
    const int e = it / 3, h = it - 3 * e;
    const DfItem d = entry_item(kk, pts + e * ps, el + e * es, h, tab);
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(b0 + 16 * it), "l"(d.p0), "l"(d.e0) : "memory");
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(b1 + 16 * it), "l"(d.p1), "l"(d.e1) : "memory");
  }
}
__device__ __forceinline__ uint32_t shared_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// One step of the transposed butterfly below: of 2 N values, a lane keeps N (the upper ones in the
// lanes with bit O set) and adds its partner's share of them.
template <int N, int O>
__device__ __forceinline__ void fold(float* v) {
  const bool up = (threadIdx.x & O) != 0;
#pragma unroll
  for (int k = 0; k < N; k++) {
    const float keep = up ? v[k + N] : v[k], give = up ? v[k] : v[k + N];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, O);
  }
}

// |u^T U_p| |v V_p^T| of the NT earlier terms p0 .. p0 + NT - 1 that exist (FP32 on the leading parts,
// each dot product summed over rows l, l + 32, ... by lane l and then over the lanes in the order of
// a xor butterfly) into prod[p]. uh, vh: leading parts of the new u and v, us and vs apart. The 4 NT
// sums are folded together, half of them dropped from a lane at each step: 4 NT shuffles and
// 5 - log2(4 NT) more instead of 20 NT.
template <int NT>
__device__ __forceinline__ void cross_terms(int p0, int nst, int m, int n, const f2* uh, int us, const f2* vh, int vs,
                                            const df2* pool, const long long* toff, df64* prod) {
  const int lane = threadIdx.x & 31;
  float s[4 * NT];
#pragma unroll
  for (int k = 0; k < 4 * NT; k++) s[k] = 0.f;
  const df2* P[NT];
#pragma unroll
  for (int t = 0; t < NT; t++) P[t] = pool + toff[min(p0 + t, nst - 1)];
#pragma unroll(4 / NT)
  for (int r = lane; r < m; r += 32) {
    const f2 u = uh[r * us];
#pragma unroll
    for (int t = 0; t < NT; t++) lead_fma(s[4 * t], s[4 * t + 1], u, P[t][r].hi);
  }
#pragma unroll(4 / NT)
  for (int c = lane; c < n; c += 32) {
    const f2 v = vh[c * vs];
#pragma unroll
    for (int t = 0; t < NT; t++) lead_fma(s[4 * t + 2], s[4 * t + 3], v, P[t][m + c].hi);
  }
  // the butterfly's steps in its order: lanes 16 apart, 8, 4, 2, 1
  if constexpr (NT == 4) {
    fold<8, 16>(s);
    fold<4, 8>(s);
    fold<2, 4>(s);
    fold<1, 2>(s);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
  } else if constexpr (NT == 2) {
    fold<4, 16>(s);
    fold<2, 8>(s);
    fold<1, 4>(s);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
  } else {
    fold<2, 16>(s);
    fold<1, 8>(s);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 4);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
  }
  // the 32 / NT lanes of a term hold Re, Im of u^T U, then Re, Im of v V^T, 8 / NT lanes each
  constexpr int Q = 8 / NT;
  const float im = __shfl_down_sync(0xffffffffu, s[0], Q);
  const float a = sqrtf(s[0] * s[0] + im * im);
  const float b = __shfl_down_sync(0xffffffffu, a, 2 * Q);
  const int p = p0 + lane / (4 * Q);
  if (lane % (4 * Q) == 0 && p < nst) prod[p] = df_prod_ff(a, b);
}

// Every earlier term, spread over the W warps of a group: as many at a time per warp as leave no
// warp idle
template <int W>
__device__ __forceinline__ void cross_all(int w, int nst, int m, int n, const f2* uh, int us, const f2* vh, int vs,
                                          const df2* pool, const long long* toff, df64* prod) {
  if (W > 1 && nst <= W) {
    for (int p = w; p < nst; p += W) cross_terms<1>(p, nst, m, n, uh, us, vh, vs, pool, toff, prod);
  } else if (W > 1 && nst <= 2 * W) {
    for (int p = 2 * w; p < nst; p += 2 * W) cross_terms<2>(p, nst, m, n, uh, us, vh, vs, pool, toff, prod);
  } else {
    for (int p = 4 * w; p < nst; p += 4 * W) cross_terms<4>(p, nst, m, n, uh, us, vh, vs, pool, toff, prod);
  }
}

// 16 bytes from global to shared memory behind the entry evaluation; visible to the group after
// cp_async_wait and the group's barrier
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ ulonglong2 lds_pair(uint32_t a) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(a) : "memory");
  return v;
}
// Entry e from its items (the six points in order), less the earlier terms:
// - sum_{p < nst} coef[p] * pool[toff[p] + off], D loads in flight, with AHEAD under the arithmetic of the D
// terms before (and the first under the items' sum). Out of line like eval_items: the warps of an SM
// are at different places of the recursion, and its straight-line code in every caller overran the
// instruction caches (21% of the stalls; 8.9 -> 7.9 ms on the 20480-triangle relief). There, loading
// ahead costs more instructions than it hides; the one block of the receiver ACA has hundreds of
// terms and nothing else to run.
// (terms past the last one load the last one again: a load behind a branch waits for the ones before)
template <int D>
__device__ __forceinline__ void load_terms(df2 (&a)[D], const df2* pool, uint32_t toff, int p, int nst) {
#pragma unroll
  for (int u = 0; u < D; u++) {
    long long o;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(o) : "r"(toff + 8 * min(p + u, nst - 1)) : "memory");
    a[u] = df2_ldc(pool + o);
  }
}
template <int D, bool AHEAD>
__device__ __noinline__ df2 finish_entry(uint32_t b0, uint32_t b1, int e, uint32_t coef, uint32_t toff,
                                         const df2* pool, int nst) {
  df2 a[D], nx[D];
  if (AHEAD && nst > 0) load_terms<D>(a, pool, toff, 0, nst);
  df2 acc{f2_dup(0.0f), f2_dup(0.0f)};
#pragma unroll 1
  for (int h = 3 * e; h < 3 * e + 3; h++) {
    const ulonglong2 x = lds_pair(b0 + 16 * h), y = lds_pair(b1 + 16 * h);
    acc = df2_add_prod(x.x, x.y, acc);
    acc = df2_add_prod(y.x, y.y, acc);
  }
  acc = entry_scale(acc);
#pragma unroll 1
  for (int p = 0; p < nst; p += D) {
    load_terms<D>(AHEAD ? nx : a, pool, toff, AHEAD ? p + D : p, nst);
#pragma unroll
    for (int u = 0; u < D; u++)
      if (p + u < nst) {
        const ulonglong2 c = lds_pair(coef + 16 * (p + u));
        df2_cfms(acc, df2{c.x, c.y}, a[u]);
      }
    if (AHEAD) {
#pragma unroll
      for (int u = 0; u < D; u++) a[u] = nx[u];
    }
  }
  return acc;
}

// Synchronises the W warps of group `grp` of the CTA.
template <int W>
__device__ __forceinline__ void group_sync(int grp) {
  if (W == 1)
    __syncwarp();
  else if (W == kDfWarps)
    __syncthreads();
  else {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * W) : "memory");
  }
}

// (value, index) argmax over the group, first index on ties; sv, si: W slots, free after the next
// group_sync
template <int W>
__device__ __forceinline__ void group_argmax(df64& val, int& idx, df64* sv, int* si, int grp) {
  warp_argmax_df(val, idx);
  if (W == 1) return;
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % W;
  if (lane == 0) {
    sv[w] = val;
    si[w] = idx;
  }
  group_sync<W>(grp);
  val = sv[0];
  idx = si[0];
#pragma unroll
  for (int k = 1; k < W; k++)
    if (sv[k] > val || (sv[k] == val && si[k] < idx)) {
      val = sv[k];
      idx = si[k];
    }
}

// Shared memory of one group of W <= 4 warps (the rows and columns fit in 64 W).
template <int W>
struct AcaGroup {
  static constexpr int kTerms = W == 1 ? 64 : kWarpAcaTerms;  // terms < min(m, n)
  ulonglong2 b0[96 * W], b1[96 * W];  // items of 32 W entries
  df2 coef[kTerms];
  df2 vs[64 * W];                     // the row residual
  f2 uh[64 * W], vh[64 * W];          // leading parts of the new u and v
  df64 su[64 * W], sv[64 * W];        // |u_r|^2, |v_c|^2
  long long toff[kTerms];
  df64 prod[kTerms];
  df64 bv[2][W];
  int bi[2][W];
  long long base;
  int ovf;
};
static_assert(sizeof(AcaGroup<1>) % 16 == 0 && sizeof(AcaGroup<2>) % 16 == 0 && sizeof(AcaGroup<4>) % 16 == 0,
              "groups follow one another in shared memory");

// ------------------------------------------------------------------------------------------
// W warps per block, sides up to 64 W: thread t owns rows and columns t and t + 32 W. The entries of a
// row or column are evaluated as 3 items each (pairs of quadrature points) spread evenly over the
// group's threads, because the sides rarely fill the threads: clusters halve from the root, so a
// mesh's sides are about c, 2 c, 4 c, ... with 16 < c <= 32, and one entry per lane left up to half
// of the lanes idle (20480 triangles: c = 20). Each entry is then finished by its owner. Sums are
// taken in one order whatever W: rows and columns l, l + 32, ... by lane l, then the butterfly.
//
// Bound by the FP32 pipe (55% busy) and, beside it, by instruction supply and latency: the warps
// are at different places of a long recursion. Four CTAs of 128 threads per SM (128 registers)
// beat six (80 registers, spills) 4.9 to 6.2 ms on the 20480-triangle relief: more warps thrash L1 and
// the instruction caches. With the 8-warp blocks' kernel the assembly takes 8.0 instead of 11.0 ms
// there, 1.65 instead of 2.95 ms on 5280 triangles and 89 instead of 106 ms on 118680 (2 kHz), against
// one warp per block with scalar arithmetic up to sides of 256.
// ------------------------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ void aca_small(const AcaDfArgs& A, unsigned char* smem, int b) {
  constexpr int T = 32 * W;
  const int grp = (threadIdx.x >> 5) / W;
  AcaGroup<W>& S = reinterpret_cast<AcaGroup<W>*>(smem)[grp];
  const uint32_t b0 = shared_addr(S.b0), b1 = shared_addr(S.b1), coef = shared_addr(S.coef), toff = shared_addr(S.toff);
  const int tid = threadIdx.x % T, lane = threadIdx.x & 31, gw = tid >> 5;
  const int4 q = A.blocks[b];
  const int rs = q.x, cs = q.z, m = q.y - q.x, n = q.w - q.z;
  int iter_lim = min(A.maxk, min(m - 1, n - 1));
  if (iter_lim < 0) iter_lim = 0;
  if (iter_lim > AcaGroup<W>::kTerms) iter_lim = AcaGroup<W>::kTerms;  // the host routes only blocks that fit

  // every warp of the group reaches the same verdict by itself
  if (iter_lim > 0 &&
      zero_block(A, rs, m, cs, n, lane, 32, [](bool ok) { return __all_sync(0xffffffffu, ok) != 0; })) {
    if (tid == 0) {
      A.rank[b] = 0;
      if (A.passes) A.passes[b] = 0;
    }
    return;
  }

  unsigned used = tid == 0 ? 1u : 0u;  // bit k: row tid + T k is used (row 0 first)
  df64 err{0.0f, 0.0f};
  int i = 0, iter = 0, nst = 0, npass = 0;
  bool need_alloc = true;
  long long base = 0;
  int nfree = 0;
  while (iter < iter_lim) {
    if (need_alloc) {
      // a term's place in the pool; taken for several terms at a time (never more than the block
      // can have), because every iteration would wait for the atomic's round trip
      if (nfree == 0) {
        nfree = min(kAcaAllocTerms, iter_lim - iter);
        if (tid == 0) {
          const unsigned long long need = (unsigned long long)(m + n) * nfree;
          const unsigned long long bb = atomicAdd(A.pool_used, need);
          S.ovf = bb + need > (unsigned long long)A.pool_cap;
          S.base = (long long)bb;
          if (S.ovf) atomicOr(A.status, 1);
        }
        group_sync<W>(grp);
        if (S.ovf) break;
        base = S.base;
      } else {
        base += m + n;
      }
      nfree--;
      need_alloc = false;
    }
    npass++;
    df2* unew = A.pool + base;
    df2* vnew = unew + m;
    // row residual v = M(i, :) - U(i, :) V and column pivot
    for (int p = tid; p < nst; p += T) cp_async_16(coef + 16 * p, A.pool + S.toff[p] + i);
    df64 best{-1.0f, 0.0f};
    int bidx = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < n; c0 += T) {
      if (c0) group_sync<W>(grp);  // the first entries are finished
      eval_items(A.k, A.pts + rs + i, 0, A.el + cs + c0, 1, min(T, n - c0), tid, T, b0, b1);
      cp_async_wait();
      group_sync<W>(grp);
      const int c = c0 + tid;
      if (c < n) {
        const df2 v = finish_entry<4, false>(b0, b1, tid, coef, toff, A.pool + m + c, nst);
        df2_stc(&S.vs[c], v);
        const df64 a = df2_abs2(v);
        if (a > best) {
          best = a;
          bidx = c;
        }
      }
    }
    if (W == 1) __syncwarp();
    group_argmax<W>(best, bidx, S.bv[0], S.bi[0], grp);
    const int j = bidx;
    const cdf vj = df2_to_cdf(df2_ldc(&S.vs[j]));
    for (int p = tid; p < nst; p += T) cp_async_16(coef + 16 * p, A.pool + S.toff[p] + m + j);
    const bool keep = df_is_zero(vj.re) && df_is_zero(vj.im);
    const CdfDivisor dv = keep ? CdfDivisor{cdf{}, 1.0f} : cdf_divisor(vj);
#pragma unroll 1
    for (int c = tid; c < n; c += T) {
      df2 v = df2_ldc(&S.vs[c]);
      if (!keep) v = df2_cdivide(v, dv);
      df2_stc(vnew + c, v);
      S.vh[c] = v.hi;
      S.sv[c] = df2_abs2(v);
    }
    // column residual u = M(:, j) - U V(:, j)
#pragma unroll 1
    for (int r0 = 0; r0 < m; r0 += T) {
      if (r0) group_sync<W>(grp);
      eval_items(A.k, A.pts + rs + r0, 1, A.el + cs + j, 0, min(T, m - r0), tid, T, b0, b1);
      cp_async_wait();
      group_sync<W>(grp);
      const int r = r0 + tid;
      if (r < m) {
        const df2 u = finish_entry<4, false>(b0, b1, tid, coef, toff, A.pool + r, nst);
        df2_stc(unew + r, u);
        S.uh[r] = u.hi;
        S.su[r] = df2_abs2(u);
      }
    }
    group_sync<W>(grp);
    // norms, every warp the same sums; cross terms sum_q |u^T U_q| |v V_q^T| (FP32 on the leading
    // parts, exact products summed as double-floats), the earlier terms over the warps
    df64 un{0.0f, 0.0f}, vn{0.0f, 0.0f};
    for (int c = lane; c < n; c += 32) vn += S.sv[c];
    for (int r = lane; r < m; r += 32) un += S.su[r];
    warp_sum2_df(un, vn);
    const df64 unt = un, vnt = vn;
    cross_all<W>(gw, nst, m, n, S.uh, 1, S.vh, 1, A.pool, S.toff, S.prod);
    group_sync<W>(grp);
    df64 dots{0.0f, 0.0f};
    for (int p = 0; p < nst; p++) dots += S.prod[p];
    const df64 uv = unt * vnt;
    err += uv + df_ldexp(dots, 2.0f);
    if (aca_converged(uv, err, A.eps2)) break;
    const bool zero_term = df_is_zero(unt) || df_is_zero(vnt);
    // next row pivot over unused rows
    best = df64{-1.0f, 0.0f};
    bidx = 0;
#pragma unroll 1
    for (int kk = 0; kk < 2; kk++) {
      const int r = tid + kk * T;
      if (r < m && !((used >> kk) & 1u)) {
        const df64 a = S.su[r];
        if (a > best) {
          best = a;
          bidx = r;
        }
      }
    }
    if (!zero_term && tid == 0) {
      S.toff[nst] = base;
      A.term_off[(long long)b * A.maxk + nst] = base;
    }
    group_argmax<W>(best, bidx, S.bv[1], S.bi[1], grp);
    i = bidx;
    if (tid == (i % T)) used |= 1u << (i / T);
    if (!zero_term) {
      nst++;
      need_alloc = true;
    }
    iter++;
    if (W == 1) __syncwarp();
  }
  if (tid == 0) {
    A.rank[b] = nst;
    if (A.passes) A.passes[b] = npass;
  }
}

// ------------------------------------------------------------------------------------------
// One CTA per block (blocks with a side above 256, or more terms than the groups hold): thread t
// owns rows and columns t + 256 k, kept in the pool. Sums: by thread, then over the warps.
// ------------------------------------------------------------------------------------------
// Shared memory of a CTA block beside its coefficients, term offsets and used-row bits; C entries are
// evaluated at a time, kDfThreads or half as many
template <int C>
struct AcaCta {
  ulonglong2 b0[3 * C], b1[3 * C];
  df64 bv[2][kDfWarps];
  int bi[2][kDfWarps];
  df64 sd[2][kDfWarps];
  long long base;
  int ovf, pad;
};
static_assert(sizeof(AcaCta<kDfThreads>) % 16 == 0 && sizeof(AcaCta<kDfThreads / 2>) % 16 == 0,
              "the coefficients follow");

template <int C>
static size_t aca_cta_smem(int iter_cap, int max_rows) {
  return sizeof(AcaCta<C>) + (size_t)iter_cap * (sizeof(df2) + sizeof(long long) + sizeof(df64)) + (size_t)((max_rows + 31) / 32) * 4;
}

template <int C>
__device__ __forceinline__ void aca_cta(const AcaDfArgs& A, unsigned char* smem, int b) {
  AcaCta<C>& S = *reinterpret_cast<AcaCta<C>*>(smem);
  df2* coef = reinterpret_cast<df2*>(smem + sizeof(AcaCta<C>));
  long long* toff = reinterpret_cast<long long*>(coef + A.iter_cap);
  df64* prod = reinterpret_cast<df64*>(toff + A.iter_cap);
  unsigned* used = reinterpret_cast<unsigned*>(prod + A.iter_cap);
  const uint32_t b0 = shared_addr(S.b0), b1 = shared_addr(S.b1), coef_a = shared_addr(coef), toff_a = shared_addr(toff);
  const int4 q = A.blocks[b];
  const int rs = q.x, cs = q.z, m = q.y - q.x, n = q.w - q.z;
  int iter_lim = min(A.maxk, min(m - 1, n - 1));
  if (iter_lim < 0) iter_lim = 0;
  if (iter_lim > A.iter_cap) iter_lim = A.iter_cap;  // host guarantees iter_cap >= every iter_lim
  const int tid = threadIdx.x, T = kDfThreads, lane = tid & 31, warp = tid >> 5;

  if (A.zero_guard && iter_lim > 0 &&
      zero_block(A, rs, m, cs, n, tid, T, [](bool ok) { return __syncthreads_and(ok) != 0; })) {
    if (tid == 0) {
      A.rank[b] = 0;
      if (A.passes) A.passes[b] = 0;
    }
    return;
  }

  for (int w = tid; w < (m + 31) / 32; w += T) used[w] = w == 0 ? 1u : 0u;
  df64 err{0.0f, 0.0f};
  int i = 0, iter = 0, nst = 0, npass = 0;
  bool need_alloc = true;
  __syncthreads();

  while (iter < iter_lim) {
    if (need_alloc) {
      if (tid == 0) {
        const unsigned long long need = (unsigned long long)(m + n);
        const unsigned long long bb = atomicAdd(A.pool_used, need);
        S.ovf = (bb + need > (unsigned long long)A.pool_cap) ? 1 : 0;
        S.base = (long long)bb;
        if (S.ovf) atomicOr(A.status, 1);
      }
      __syncthreads();
      if (S.ovf) break;
      need_alloc = false;
    }
    npass++;
    const long long base = S.base;
    df2* unew = A.pool + base;
    df2* vnew = unew + m;
    for (int p = tid; p < nst; p += T) df2_stc(&coef[p], df2_ldc(A.pool + toff[p] + i));

    // row residual v = M(i, :) - U(i, :) V
    df64 best{-1.0f, 0.0f};
    int bidx = 0;
    for (int c0 = 0; c0 < n; c0 += C) {
      if (c0) __syncthreads();  // the previous entries are finished
      eval_items(A.k, A.pts + rs + i, 0, A.el + cs + c0, 1, min(C, n - c0), tid, T, b0, b1);
      __syncthreads();
      const int e = C == kDfThreads ? tid : tid - c0 % T, c = c0 + e;  // (thread t owns t, t + T, ...)
      if (e >= 0 && e < C && c < n) {
        const df2 v = finish_entry<4, false>(b0, b1, e, coef_a, toff_a, A.pool + m + c, nst);
        df2_stc(vnew + c, v);
        const df64 a = df2_abs2(v);
        if (a > best) {
          best = a;
          bidx = c;
        }
      }
    }
    group_argmax<kDfWarps>(best, bidx, S.bv[0], S.bi[0], 0);
    const int j = bidx;
    const cdf vj = df2_to_cdf(df2_ldc(vnew + j));
    for (int p = tid; p < nst; p += T) df2_stc(&coef[p], df2_ldc(A.pool + toff[p] + m + j));
    __syncthreads();  // v_j is read before it is divided
    const bool keep = A.zero_guard && df_is_zero(vj.re) && df_is_zero(vj.im);
    const CdfDivisor dv = keep ? CdfDivisor{cdf{}, 1.0f} : cdf_divisor(vj);
    df64 vn{0.0f, 0.0f};
    for (int c = tid; c < n; c += T) {
      df2 v = df2_ldc(vnew + c);
      if (!keep) v = df2_cdivide(v, dv);
      df2_stc(vnew + c, v);
      vn += df2_abs2(v);
    }

    // column residual u = M(:, j) - U V(:, j)
    df64 un{0.0f, 0.0f};
    for (int r0 = 0; r0 < m; r0 += C) {
      if (r0) __syncthreads();
      eval_items(A.k, A.pts + rs + r0, 1, A.el + cs + j, 0, min(C, m - r0), tid, T, b0, b1);
      __syncthreads();
      const int e = C == kDfThreads ? tid : tid - r0 % T, r = r0 + e;
      if (e >= 0 && e < C && r < m) {
        const df2 u = finish_entry<4, false>(b0, b1, e, coef_a, toff_a, A.pool + r, nst);
        df2_stc(unew + r, u);
        un += df2_abs2(u);
      }
    }
    __syncthreads();

    // cross terms and the norms; then the products in the order of one
    // running sum per warp w over the terms w, w + 8, ..., and the eight sums in order
    cross_all<kDfWarps>(warp, nst, m, n, &unew->hi, 2, &vnew->hi, 2, A.pool, toff, prod);
    warp_sum2_df(un, vn);
    if (lane == 0) {
      S.sd[0][warp] = un;
      S.sd[1][warp] = vn;
    }
    __syncthreads();
    df64 unt = S.sd[0][0], vnt = S.sd[1][0];
#pragma unroll 1
    for (int k = 1; k < kDfWarps; k++) {
      unt += S.sd[0][k];
      vnt += S.sd[1][k];
    }
    df64 part{0.0f, 0.0f};
    if (lane < kDfWarps)
      for (int p = lane; p < nst; p += kDfWarps) part += prod[p];
    df64 dots = shfl_df(part, 0);
#pragma unroll 1
    for (int k = 1; k < kDfWarps; k++) dots += shfl_df(part, k);
    const df64 uv = unt * vnt;
    err += uv + df_ldexp(dots, 2.0f);
    if (aca_converged(uv, err, A.eps2)) break;
    const bool zero_term = df_is_zero(unt) || df_is_zero(vnt);

    // next row pivot: first max |u|^2 over unused rows
    best = df64{-1.0f, 0.0f};
    bidx = 0;
    for (int r = tid; r < m; r += T) {
      if ((used[r >> 5] >> (r & 31)) & 1u) continue;
      const df64 a = df2_abs2(df2_ldc(unew + r));
      if (a > best) {
        best = a;
        bidx = r;
      }
    }
    group_argmax<kDfWarps>(best, bidx, S.bv[1], S.bi[1], 0);
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

template <int C>
__global__ void __launch_bounds__(kDfThreads, 2) aca_df_cta_kernel(AcaDfArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_table(A.tab);
  aca_cta<C>(A, smem_raw, A.order[blockIdx.x]);
}

// The blocks next, next + 1, ... of a class by the CTA's groups, each as it gets free
template <int W>
__device__ __forceinline__ void run_groups(const AcaDfArgs& A, unsigned char* smem, const int* order, int count,
                                           unsigned* next) {
  __shared__ int s_block[kSmallThreads / 32];
  const int grp = (threadIdx.x >> 5) / W, tid = threadIdx.x % (32 * W);
  for (;;) {
    if (tid == 0) {
      const unsigned t = atomicAdd(next, 1u);
      s_block[grp] = t < (unsigned)count ? order[t] : -1;
    }
    group_sync<W>(grp);
    const int b = s_block[grp];
    if (b < 0) break;
    aca_small<W>(A, smem, b);
    group_sync<W>(grp);  // the group's shared memory is free for the next block
  }
}

// The blocks of sides up to 256 in one launch, longest first. As many CTAs as are resident take them,
// first as one 4-warp group each, then as two 2-warp and four 1-warp groups: with four blocks to a
// CTA that ends with the longest of them, 12.6 of 16 warps per SM were running (4.94 -> 4.67 ms on the
// 20480-triangle relief).
__global__ void __launch_bounds__(kSmallThreads, 4) aca_df_kernel(AcaDfArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_table(A.tab);
  const int* order = A.order + A.split[0];
  run_groups<4>(A, smem_raw, order, A.split[1], A.next);
  __syncthreads();
  order += A.split[1];
  run_groups<2>(A, smem_raw, order, A.split[2], A.next + 1);
  __syncthreads();
  order += A.split[2];
  run_groups<1>(A, smem_raw, order, A.split[3], A.next + 2);
}

// ------------------------------------------------------------------------------------------
// Near field: one CTA per block, one thread per entry, rounded to complex FP32.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) near_df_kernel(const DfPt* __restrict__ pts, const DfElem* __restrict__ el,
                                                      const float4* __restrict__ tab, const int4* __restrict__ blocks,
                                                      const long long* __restrict__ near_off, df64 k, cf* out) {
  load_table(tab);
  const float4* s_tab = s_table();
  const int b = blockIdx.x;
  const int4 q = blocks[b];
  const int m = q.y - q.x, n = q.w - q.z;
  cf* dst = out + near_off[b];
  const int mn = m * n;
  for (int t = threadIdx.x; t < mn; t += blockDim.x) {
    const int c = t / m, r = t - c * m;
    const df2 v = entry_df(k, pts + q.x + r, el + q.z + c, s_tab);
    dst[t] = cf(f2_x(v.hi), f2_y(v.hi));
  }
}

void launch_near_assembly_df(const DevGeometry& G, const DevPartition& DP, DevHMat& H, cudaStream_t s) {
  if (DP.nd == 0) return;
  note_launch();
  near_df_kernel<<<DP.nd, 256, 0, s>>>(G.cen_df.as<DfPt>(), G.el_df.as<DfElem>(), G.df_tab.as<float4>(),
                                       DP.blocks_d.as<int4>(), DP.near_off.as<long long>(), df_from_double(H.k),
                                       H.near.as<cf>());
  AC3D_CUDA(cudaGetLastError());
}

// What a CTA can have beside the static shared memory of these kernels (the table, a few words).
constexpr size_t kAcaSmemMax = 227 * 1024 - kDfTab * sizeof(float4) - 256;
// The blocks that are taken: 40 bytes a term and a bit a row in 200 KB, or all of a CTA's in 200 KB. The
// first kind fits with half of the entries at a time; with kDfThreads all do but those of 1.57 million rows
// and more.
constexpr size_t kAcaBlockMax = 200 * 1024;
static_assert(sizeof(AcaCta<kDfThreads / 2>) + kAcaBlockMax <= kAcaSmemMax, "every block that is taken fits");

// kernels[1] (half of the entries at a time) where kernels[0] does not fit; false: not taken
template <typename K>
static bool pick_aca_kernel(const K (&kernels)[2], int iter_cap, int max_rows, K& kernel, size_t& smem) {
  smem = aca_cta_smem<kDfThreads>(iter_cap, max_rows);
  if ((size_t)iter_cap * 40 + (size_t)((max_rows + 31) / 32) * 4 > kAcaBlockMax && smem > kAcaBlockMax) return false;
  kernel = kernels[0];
  if (smem > kAcaSmemMax) {
    smem = aca_cta_smem<kDfThreads / 2>(iter_cap, max_rows);
    kernel = kernels[1];
  }
  return true;
}

// Blocks above 256 on s_large, the others on s_small.
static void launch_aca_kernels(const AcaDfArgs& a, int max_rows, cudaStream_t s_large, cudaStream_t s_small) {
  if (a.split[0] > 0) {
    static void (*const kernels[2])(AcaDfArgs) = {aca_df_cta_kernel<kDfThreads>, aca_df_cta_kernel<kDfThreads / 2>};
    void (*kernel)(AcaDfArgs);
    size_t smem;
    if (!pick_aca_kernel(kernels, a.iter_cap, max_rows, kernel, smem)) throw Error(4, "ACA block too large for shared memory");
    // once per process, to the largest size any launch uses: contexts on other threads launch with
    // other sizes
    static std::once_flag once;
    std::call_once(once, [] {
      for (auto k : kernels) AC3D_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAcaSmemMax));
    });
    note_launch();
    kernel<<<a.split[0], kDfThreads, smem, s_large>>>(a);
    AC3D_CUDA(cudaGetLastError());
  }
  const int ctas = a.split[1] + (a.split[2] + 1) / 2 + (a.split[3] + 3) / 4;
  if (ctas > 0) {
    constexpr size_t smem = std::max({sizeof(AcaGroup<4>), 2 * sizeof(AcaGroup<2>), 4 * sizeof(AcaGroup<1>)});
    static_assert(smem <= 48 * 1024, "no opt-in needed");
    note_launch();
    aca_df_kernel<<<std::min(ctas, 4 * device_sm_count()), kSmallThreads, smem, s_small>>>(a);
    AC3D_CUDA(cudaGetLastError());
  }
}

void launch_aca_df(const DevGeometry& G, const DevPartition& DP, DevHMat& H, double eps, int max_rows, cudaStream_t s,
                   cudaStream_t s_small) {
  if (DP.na == 0) return;
  AcaDfArgs a{G.cen.as<double4>(), G.va.as<double4>(), G.eg64.as<ElemGeo<double>>(), G.cen_df.as<DfPt>(),
              G.el_df.as<DfElem>(), G.df_tab.as<float4>(), DP.blocks_a.as<int4>(), DP.aca_order.as<int>(),
              {DP.aca_split[0], DP.aca_split[1], DP.aca_split[2], DP.aca_split[3]},
              df_from_double(H.k), df_from_double(eps * eps), H.maxk, H.maxk, H.pool.as<df2>(), H.pool_cap,
              H.pool_used.as<unsigned long long>(), H.term_off.as<long long>(), H.rank.as<int>(),
              &H.pool_used.as<AsmTotals>()->status, H.passes.as<int>(), H.pool_used.as<AsmTotals>()->next, 1};
  launch_aca_kernels(a, max_rows, s, s_small);
}

// ------------------------------------------------------------------------------------------
// One block over the whole GPU: the receiver ACA (L receivers x Ne elements, a single block of high
// rank). A cooperative kernel; CTA c owns a contiguous range of the columns and one of the rows. An
// iteration has three grid barriers: after the row (every CTA then finds the pivot among the CTAs'
// best), after the divided row and the column, and after the cross terms (one warp per earlier
// term and side) and the norms. The stopping test and the next row pivot are computed by every CTA
// alike. Sums are taken in the order of aca_cta. Data that other SMs write in the iteration is read
// past L1 (ld.cg); terms are a multiple of 128 bytes apart, so that no line of an earlier term holds
// part of a later one.
//
// Bound by latency: an iteration takes 37 us (1297 receivers x 10680 elements, tolerance 1e-5, 135 to 168
// terms); when it was split up, at 40 us, the chain over the earlier terms took 15 us, the longest dot
// product 12 us, the barriers 5 us, the entries 3 us. 5.6 ms instead of 168 ms by one CTA, which is where it
// began (146 ms with the entries' items spread over its threads).
// ------------------------------------------------------------------------------------------
struct alignas(16) AcaBest {
  df2 v;      // the entry
  df64 a;     // |v|^2
  int idx;
  int pad;
};

struct AcaGridBufs {
  unsigned long long* bar;  // arrivals, zero at launch
  int* fail;                // a wait gave up
  AcaBest* best;            // per CTA
  df64* sq_v;               // |v_c|^2 (n)
  df64* sq_u;               // |u_r|^2 (m)
  df64* norm;               // |u|^2, |v|^2
  float2* dots;             // per earlier term: u^T U_p, v V_p^T
  int stride;               // entries between terms
};

constexpr uint32_t kGridSpin = 1u << 24;  // polls of an L2 line, seconds in all

__device__ __forceinline__ bool aca_grid_sync(const AcaGridBufs& X) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned long long t = atomicAdd(X.bar, 1ull);
    const unsigned long long target = (t / gridDim.x + 1) * (unsigned long long)gridDim.x;
    volatile unsigned long long* c = X.bar;
    int ok = 1;
    uint32_t it = 0;
    while (*c < target) {
      if (++it > kGridSpin) {
        ok = 0;
        atomicExch(X.fail, 1);
        break;
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ df2 df2_ldcg(const df2* p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
  return {v.x, v.y};
}
__device__ __forceinline__ df64 df64_ldcg(const df64* p) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
  return {v.x, v.y};
}

// sum_r a_r b_r of the leading parts, a new vector against an earlier term, by one warp: lane 0 gets the
// real part, lane 16 the imaginary part
__device__ __noinline__ float grid_dot(const df2* a, const df2* b, int len) {
  const int lane = threadIdx.x & 31;
  float s[2] = {0.f, 0.f};
  constexpr int D = 32;  // pairs of loads in flight
  for (int r0 = lane; r0 < len; r0 += 32 * D) {
    f2 x[D], y[D];
#pragma unroll
    for (int k = 0; k < D; k++) {
      const int r = min(r0 + 32 * k, len - 1);
      x[k] = __ldcg(&a[r].hi);
      y[k] = b[r].hi;
    }
#pragma unroll
    for (int k = 0; k < D; k++)
      if (r0 + 32 * k < len) lead_fma(s[0], s[1], x[k], y[k]);
  }
  fold<1, 16>(s);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
  return s[0];
}

template <int C>
__global__ void __launch_bounds__(kDfThreads, 1) aca_df_grid_kernel(AcaDfArgs A, AcaGridBufs X) {
  extern __shared__ __align__(16) unsigned char smem[];
  load_table(A.tab);
  AcaCta<C>& S = *reinterpret_cast<AcaCta<C>*>(smem);
  df2* coef = reinterpret_cast<df2*>(smem + sizeof(AcaCta<C>));
  long long* toff = reinterpret_cast<long long*>(coef + A.iter_cap);
  df64* prod = reinterpret_cast<df64*>(toff + A.iter_cap);
  unsigned* used = reinterpret_cast<unsigned*>(prod + A.iter_cap);
  const uint32_t b0 = shared_addr(S.b0), b1 = shared_addr(S.b1), coef_a = shared_addr(coef), toff_a = shared_addr(toff);
  const int4 q = A.blocks[A.order[0]];
  const int rs = q.x, cs = q.z, m = q.y - q.x, n = q.w - q.z;
  const int iter_lim = max(0, min(min(A.maxk, A.iter_cap), min(m - 1, n - 1)));
  const int tid = threadIdx.x, T = kDfThreads, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, cta = blockIdx.x;
  const int pc = (n + G - 1) / G, pr = (m + G - 1) / G;
  const int c_lo = min(n, cta * pc), c_hi = min(n, c_lo + pc), r_lo = min(m, cta * pr), r_hi = min(m, r_lo + pr);
  for (int w = tid; w < (m + 31) / 32; w += T) used[w] = w == 0 ? 1u : 0u;
  __syncthreads();
  df64 err{0.0f, 0.0f};
  int i = 0, nst = 0;
  bool ok = true;
  for (int iter = 0; iter < iter_lim; iter++) {
    const long long base = (long long)nst * X.stride;
    df2* unew = A.pool + base;
    df2* vnew = unew + m;
    // row residual of this CTA's columns
    for (int p = tid; p < nst; p += T) df2_stc(&coef[p], df2_ldcg(A.pool + toff[p] + i));
    df64 best{-1.0f, 0.0f};
    df2 bv{0, 0};
    int bidx = 0;
    for (int c0 = c_lo; c0 < c_hi; c0 += C) {
      if (c0 > c_lo) __syncthreads();
      eval_items(A.k, A.pts + rs + i, 0, A.el + cs + c0, 1, min(C, c_hi - c0), tid, T, b0, b1);
      __syncthreads();
      const int c = c0 + tid;
      if (tid < C && c < c_hi) {
        const df2 v = finish_entry<8, true>(b0, b1, tid, coef_a, toff_a, A.pool + m + c, nst);
        df2_stc(vnew + c, v);
        const df64 a = df2_abs2(v);
        if (a > best) {
          best = a;
          bidx = c;
          bv = v;
        }
      }
    }
    {
      df64 val = best;
      int idx = bidx;
      group_argmax<kDfWarps>(val, idx, S.bv[0], S.bi[0], 0);
      AcaBest* o = X.best + cta;
      if (tid == 0) {
        o->a = val;
        o->idx = idx;
      }
      if (idx == bidx && !(best.hi < 0.0f)) df2_stc(&o->v, bv);  // the one thread that holds it
    }
    if (!(ok = aca_grid_sync(X))) break;
    // column pivot: the best of the CTAs' bests
    best = df64{-1.0f, 0.0f};
    bidx = 0;
    for (int k = tid; k < G; k += T) {
      const df64 a = df64_ldcg(&X.best[k].a);
      const int idx = __ldcg(&X.best[k].idx);
      if (a > best) {  // ascending ranges: the first of equals is the smallest index
        best = a;
        bidx = idx;
      }
    }
    group_argmax<kDfWarps>(best, bidx, S.bv[1], S.bi[1], 0);
    const int j = bidx;
    const cdf vj = df2_to_cdf(df2_ldcg(&X.best[min(G - 1, j / pc)].v));
    for (int p = tid; p < nst; p += T) df2_stc(&coef[p], df2_ldcg(A.pool + toff[p] + m + j));
    const bool keep = A.zero_guard && df_is_zero(vj.re) && df_is_zero(vj.im);
    const CdfDivisor dv = keep ? CdfDivisor{cdf{}, 1.0f} : cdf_divisor(vj);
    for (int c = c_lo + tid; c < c_hi; c += T) {
      df2 v = df2_ldcg(vnew + c);
      if (!keep) v = df2_cdivide(v, dv);
      df2_stc(vnew + c, v);
      X.sq_v[c] = df2_abs2(v);
    }
    // column residual of this CTA's rows
    for (int r0 = r_lo; r0 < r_hi; r0 += C) {
      if (r0 > r_lo) __syncthreads();
      eval_items(A.k, A.pts + rs + r0, 1, A.el + cs + j, 0, min(C, r_hi - r0), tid, T, b0, b1);
      __syncthreads();
      const int r = r0 + tid;
      if (tid < C && r < r_hi) {
        const df2 u = finish_entry<8, true>(b0, b1, tid, coef_a, toff_a, A.pool + r, nst);
        df2_stc(unew + r, u);
        X.sq_u[r] = df2_abs2(u);
      }
    }
    if (!(ok = aca_grid_sync(X))) break;
    // norms by the first CTA; cross terms by the warps of the others
    if (cta == 0) {
      df64 un{0.0f, 0.0f}, vn{0.0f, 0.0f};
      for (int c0 = tid; c0 < n; c0 += 8 * T) {
        df64 x[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (c0 + k * T < n) x[k] = df64_ldcg(X.sq_v + c0 + k * T);
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (c0 + k * T < n) vn += x[k];
      }
      for (int r = tid; r < m; r += T) un += df64_ldcg(X.sq_u + r);
      warp_sum2_df(un, vn);
      if (lane == 0) {
        S.sd[0][warp] = un;
        S.sd[1][warp] = vn;
      }
      __syncthreads();
      if (tid == 0) {
        un = S.sd[0][0];
        vn = S.sd[1][0];
        for (int k = 1; k < kDfWarps; k++) {
          un += S.sd[0][k];
          vn += S.sd[1][k];
        }
        X.norm[0] = un;
        X.norm[1] = vn;
      }
    }
    if (cta > 0 || G == 1) {
      const int ng = max(1, G - 1), w0 = warp * ng + (G == 1 ? 0 : cta - 1), nw = ng * kDfWarps;  // over the SMs first
      for (int t = w0; t < 2 * nst; t += nw) {
        // the long sides first
        const int p = t < nst ? t : t - nst;
        const bool row = t < nst;
        const int o0 = row ? m : 0;
        const float d = grid_dot(unew + o0, A.pool + toff[p] + o0, row ? n : m);
        float* o = reinterpret_cast<float*>(X.dots + 2 * p + (row ? 1 : 0));
        if (lane == 0) o[0] = d;
        if (lane == 16) o[1] = d;
      }
    }
    if (!(ok = aca_grid_sync(X))) break;
    // stopping test and next row pivot, alike in every CTA
    const df64 unt = df64_ldcg(X.norm), vnt = df64_ldcg(X.norm + 1);
    for (int p = tid; p < nst; p += T) {
      const float2 u = __ldcg(X.dots + 2 * p), v = __ldcg(X.dots + 2 * p + 1);
      prod[p] = df_prod_ff(sqrtf(u.x * u.x + u.y * u.y), sqrtf(v.x * v.x + v.y * v.y));
    }
    __syncthreads();
    df64 part{0.0f, 0.0f};
    if (lane < kDfWarps)
      for (int p = lane; p < nst; p += kDfWarps) part += prod[p];
    df64 dots = shfl_df(part, 0);
#pragma unroll 1
    for (int k = 1; k < kDfWarps; k++) dots += shfl_df(part, k);
    const df64 uv = unt * vnt;
    err += uv + df_ldexp(dots, 2.0f);
    if (aca_converged(uv, err, A.eps2)) break;
    const bool zero_term = df_is_zero(unt) || df_is_zero(vnt);
    best = df64{-1.0f, 0.0f};
    bidx = 0;
    for (int r0 = tid; r0 < m; r0 += 8 * T) {
      df64 x[8];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (r0 + k * T < m) x[k] = df64_ldcg(X.sq_u + r0 + k * T);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int r = r0 + k * T;
        if (r < m && !((used[r >> 5] >> (r & 31)) & 1u) && x[k] > best) {
          best = x[k];
          bidx = r;
        }
      }
    }
    group_argmax<kDfWarps>(best, bidx, S.bv[0], S.bi[0], 0);
    i = bidx;
    if (tid == 0) {
      used[i >> 5] |= 1u << (i & 31);
      if (!zero_term) {
        toff[nst] = base;
        if (cta == 0) A.term_off[nst] = base;
      }
    }
    if (!zero_term) nst++;
    __syncthreads();
  }
  if (cta == 0 && tid == 0) {
    A.rank[0] = nst;
    *A.pool_used = (unsigned long long)nst * X.stride;
    if (!ok) atomicOr(A.status, 2);
  }
}

// Receiver ACA (compute_ACA_listener, aca.cpp:84-134: one block of L receivers x Ne elements, no
// zero guard) in double-float, then the terms converted in place to complex FP64 (same size).
__global__ void df_to_cd_kernel(df2* pool, const unsigned long long* used) {
  const unsigned long long n = *used;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const cdf v = df2_to_cdf(df2_ldc(pool + i));
    reinterpret_cast<cd*>(pool)[i] = cd(df_to_double(v.re), df_to_double(v.im));
  }
}

// Entries of a receiver term in the pool: rounded up so that terms start on 128-byte lines.
int listener_term_stride(int L, int ne) { return (L + ne + 7) & ~7; }

void launch_listener_aca_df(const DevGeometry& G, const void* pts_df, int L, double k, double eps, int maxk,
                            void* pool, long long pool_cap, unsigned long long* used, long long* term_off, int* rank,
                            int* status, const int4* block, const int* order, DevBuf& scratch, cudaStream_t s) {
  int iter_lim = std::min(maxk, std::min(L - 1, G.ne - 1));
  if (iter_lim < 1) iter_lim = 1;
  AcaDfArgs a{G.cen.as<double4>(), G.va.as<double4>(), G.eg64.as<ElemGeo<double>>(), (const DfPt*)pts_df,
              G.el_df.as<DfElem>(), G.df_tab.as<float4>(), block, order, {1, 0, 0, 0}, df_from_double(k),
              df_from_double(eps * eps), maxk, iter_lim,
              (df2*)pool, pool_cap, used, term_off, rank, status, nullptr, nullptr, 0};
  static void (*const kernels[2])(AcaDfArgs, AcaGridBufs) = {aca_df_grid_kernel<kDfThreads>, aca_df_grid_kernel<kDfThreads / 2>};
  void (*kernel)(AcaDfArgs, AcaGridBufs);
  size_t smem;
  if (!pick_aca_kernel(kernels, iter_lim, L, kernel, smem))
    throw Error(4, "receiver ACA too large for shared memory (at most about 5000 receivers)");
  static std::once_flag once;
  std::call_once(once, [] {
    for (auto k : kernels) AC3D_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAcaSmemMax));
  });
  int per_sm = 0;
  AC3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kDfThreads, smem));
  // about 64 columns (192 items) per CTA, at most one CTA per SM
  const int grid = std::max(1, std::min((per_sm > 0 ? 1 : 0) * device_sm_count(), (G.ne + 63) / 64));
  if (grid <= 2 || L + G.ne <= 384) {
    // barriers would cost more than the entries. By the grid and by one CTA: 0.33 and 0.24 ms on 180
    // elements and 37 receivers, 0.30 and 0.23 on 240 and 37, 0.09 and 0.08 on 384 and 5; the same on 308 and
    // 37 (0.29, 0.30) and on 240 and 181; 0.29 and 0.36 on 468 and 37, 0.44 and 0.73 on 140 and 1297
    launch_aca_kernels(a, L, s, s);
    note_launch();
    df_to_cd_kernel<<<4 * device_sm_count(), 256, 0, s>>>((df2*)pool, used);
    AC3D_CUDA(cudaGetLastError());
    return;
  }
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t o_best = 256, o_v = o_best + up(grid * sizeof(AcaBest)), o_u = o_v + up((size_t)G.ne * sizeof(df64)),
               o_n = o_u + up((size_t)L * sizeof(df64)), o_d = o_n + 256,
               total = o_d + up((size_t)iter_lim * 2 * sizeof(float2));
  scratch.alloc(total, s);
  AC3D_CUDA(cudaMemsetAsync(scratch.p, 0, 256, s));
  char* sp = (char*)scratch.p;
  AcaGridBufs x{(unsigned long long*)sp, (int*)(sp + 8), (AcaBest*)(sp + o_best), (df64*)(sp + o_v), (df64*)(sp + o_u),
                (df64*)(sp + o_n), (float2*)(sp + o_d), listener_term_stride(L, G.ne)};
  void* args[] = {&a, &x};
  note_launch();
  AC3D_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3(grid), dim3(kDfThreads), args, smem, s));
  note_launch();
  df_to_cd_kernel<<<4 * device_sm_count(), 256, 0, s>>>((df2*)pool, used);
  AC3D_CUDA(cudaGetLastError());
}

}  // namespace ac3d
