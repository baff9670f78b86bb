// Double-float (about 47-bit) evaluation of the collocation entry M(p, element) for the
// mixed-precision path's near-field blocks and ACA rows and columns. The entries agree with the
// FP64 path's to about 1e-13 relative, so ACA picks the FP64 path's pivots and ranks, and only
// the stored factors are rounded to FP32.
//
// Per element the six quadrature points y_q = a + m_q (b - a) + n_q (c - a) are formed in FP64
// and kept as double-floats with the unnormalised normal n = (b - a) x (c - a); per collocation
// point the centroid is kept as a double-float. The entry is
//   M = 1/2 sum_q w_q e^{-ikr}(1 + ikr) (r.n) / (4 pi r^3),  r = p - y_q,
// the dGdr(k, r) (-(r.n)/r) of integrate.h:11-19 summed over the rule of integrate.cpp:5-14.
#pragma once

#include "common.cuh"
#include "df2.cuh"
#include "df64.cuh"

namespace ac3d {

struct alignas(16) DfPt {
  df64 x, y, z;
  float pad[2];
};

// Quadrature points 2 h and 2 h + 1 side by side: yq[h][d] = {hi, hi', lo, lo'} of coordinate d, so
// that one 16-byte load fills the two register pairs of the packed arithmetic.
struct alignas(16) DfElem {
  float4 yq[3][3];
  df64 n[3];
  float pad[2];
};
static_assert(sizeof(DfElem) == 176, "DfElem layout");
static_assert(sizeof(DfPt) == 32, "DfPt layout");

__device__ __forceinline__ df2 df2_load(const float4* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}

// Contributions of the quadrature points 2 h and 2 h + 1 to an entry, as exact-product pairs: point
// 2 h adds p0 + e0 and point 2 h + 1 adds p1 + e1 to (re, im).
struct DfItem {
  f2 p0, e0, p1, e1;
};

// Two quadrature points at once through the geometry, the phase and the weights: about 400 packed
// operations, bound by the FP32 pipe (two clocks each).
__device__ __forceinline__ DfItem entry_item(df2 kk, const DfPt* __restrict__ pp, const DfElem* __restrict__ ge, int h,
                                             const float4* __restrict__ tab) {
  const DfPt p = *pp;
  const df2 rx = df2_dup(p.x) - df2_load(&ge->yq[h][0]);
  const df2 ry = df2_dup(p.y) - df2_load(&ge->yq[h][1]);
  const df2 rz = df2_dup(p.z) - df2_load(&ge->yq[h][2]);
  const df2 r = df2_sqrt(df2_norm2_3(rx, ry, rz));
  const df2 rinv = df2_rcp(r);
  const df2 s = df2_fma(rz, df2_dup(ge->n[2]), df2_fma(ry, df2_dup(ge->n[1]), rx * df2_dup(ge->n[0])));
  const df2 kr = kk * r;
  df2 cs, sn;
  df2_sincos(kr, tab, cs, sn);
  const df64 w0 = df_from_double(quad_w(0)), w3 = df_from_double(quad_w(3));
  const df2 w = df2_make(h < 2 ? w0 : w3, h < 1 ? w0 : w3);
  const df2 f = (s * (rinv * df2_sqr(rinv))) * w;
  // e^{-ikr}(1 + ikr) = (cs + kr sn) + i (kr cs - sn)
  f2 pr, er, pi, ei;
  df2_prod(f, df2_fma(kr, sn, cs), pr, er);
  df2_prod(f, df2_fms(kr, cs, sn), pi, ei);
  return {f2_make(f2_x(pr), f2_x(pi)), f2_make(f2_x(er), f2_x(ei)), f2_make(f2_y(pr), f2_y(pi)),
          f2_make(f2_y(er), f2_y(ei))};
}

__device__ __forceinline__ df2 entry_scale(df2 acc) { return acc * df2_dup(df_from_double(0.5 / (4.0 * kPi))); }

// The entry as (re, im): bit for bit the sum over the six points in order in scalar double-float
// arithmetic.
__device__ __forceinline__ df2 entry_df(df64 k, const DfPt* __restrict__ pp, const DfElem* __restrict__ ge,
                                        const float4* __restrict__ tab) {
  const df2 kk = df2_dup(k);
  df2 acc{f2_dup(0.0f), f2_dup(0.0f)};
#pragma unroll 1
  for (int h = 0; h < 3; h++) {
    const DfItem t = entry_item(kk, pp, ge, h, tab);
    acc = df2_add_prod(t.p0, t.e0, acc);
    acc = df2_add_prod(t.p1, t.e1, acc);
  }
  return entry_scale(acc);
}

}  // namespace ac3d
