// Two double-floats at a time on the packed FP32 instructions of sm_100 and later (add, sub, mul and
// fma .rn.f32x2: two IEEE operations on a 64-bit register pair). Each half of a packed operation
// rounds as the scalar instruction does, so the functions below give, half by half, the bits of
// their scalar namesakes in df64.cuh, which say what each computes and how exactly.
//
// Why: the packed forms issue one instruction for two operations. Their lane rate is the scalar
// one (measured 112-123 against 118 lane operations per clock and SM, the same 4.2 clocks of
// latency), but the double-float code is a long dependent chain that a few resident warps could
// not issue fast enough; packed, each instruction holds the pipe for two clocks and four warps per
// scheduler fill it.
#pragma once

#include "df64.cuh"

namespace ac3d {

typedef unsigned long long f2;  // two FP32 values: low half .x, high half .y

__device__ __forceinline__ f2 f2_make(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ f2 f2_dup(float x) { return f2_make(x, x); }
__device__ __forceinline__ float f2_x(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x;
}
__device__ __forceinline__ float f2_y(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return y;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_neg(f2 a) { return f2_make(-f2_x(a), -f2_y(a)); }

__device__ __forceinline__ void two_sum2(f2 a, f2 b, f2& s, f2& e) {
  s = f2_add(a, b);
  const f2 bb = f2_sub(s, a);
  e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
}
// two_sum(a, -b)
__device__ __forceinline__ void two_diff2(f2 a, f2 b, f2& s, f2& e) {
  s = f2_sub(a, b);
  const f2 bb = f2_sub(s, a);
  e = f2_sub(f2_sub(a, f2_sub(s, bb)), f2_add(b, bb));
}
__device__ __forceinline__ void fast_two_sum2(f2 a, f2 b, f2& s, f2& e) {
  s = f2_add(a, b);
  e = f2_sub(b, f2_sub(s, a));
}
__device__ __forceinline__ void two_prod2(f2 a, f2 b, f2& p, f2& e) {
  p = f2_mul(a, b);
  e = f2_fma(a, b, f2_neg(p));
}

struct alignas(16) df2 {
  f2 hi, lo;
};

__device__ __forceinline__ df2 df2_dup(df64 a) { return {f2_dup(a.hi), f2_dup(a.lo)}; }
__device__ __forceinline__ df2 df2_make(df64 x, df64 y) { return {f2_make(x.hi, y.hi), f2_make(x.lo, y.lo)}; }
__device__ __forceinline__ df64 df2_x(df2 a) { return {f2_x(a.hi), f2_x(a.lo)}; }
__device__ __forceinline__ df64 df2_y(df2 a) { return {f2_y(a.hi), f2_y(a.lo)}; }

__device__ __forceinline__ df2 operator+(df2 a, df2 b) {
  f2 s, e;
  two_sum2(a.hi, b.hi, s, e);
  e = f2_add(e, f2_add(a.lo, b.lo));
  fast_two_sum2(s, e, s, e);
  return {s, e};
}
__device__ __forceinline__ df2 operator-(df2 a, df2 b) {
  f2 s, e;
  two_diff2(a.hi, b.hi, s, e);
  e = f2_add(e, f2_sub(a.lo, b.lo));
  fast_two_sum2(s, e, s, e);
  return {s, e};
}
__device__ __forceinline__ df2 operator*(df2 a, df2 b) {
  f2 p, e;
  two_prod2(a.hi, b.hi, p, e);
  e = f2_fma(a.hi, b.lo, e);
  e = f2_fma(a.lo, b.hi, e);
  fast_two_sum2(p, e, p, e);
  return {p, e};
}
__device__ __forceinline__ df2 df2_add_f(df2 a, f2 b) {
  f2 s, e;
  two_sum2(a.hi, b, s, e);
  e = f2_add(e, a.lo);
  fast_two_sum2(s, e, s, e);
  return {s, e};
}
__device__ __forceinline__ df2 df2_sub_f(df2 a, f2 b) {
  f2 s, e;
  two_diff2(a.hi, b, s, e);
  e = f2_add(e, a.lo);
  fast_two_sum2(s, e, s, e);
  return {s, e};
}
// the sum of an exact product p + e and c with one normalisation (the second half of df_fma)
__device__ __forceinline__ df2 df2_add_prod(f2 p, f2 e, df2 c) {
  f2 s, t;
  two_sum2(p, c.hi, s, t);
  t = f2_add(t, f2_add(e, c.lo));
  fast_two_sum2(s, t, s, t);
  return {s, t};
}
__device__ __forceinline__ void df2_prod(df2 a, df2 b, f2& p, f2& e) {
  two_prod2(a.hi, b.hi, p, e);
  e = f2_fma(a.hi, b.lo, e);
  e = f2_fma(a.lo, b.hi, e);
}
__device__ __forceinline__ df2 df2_fma(df2 a, df2 b, df2 c) {
  f2 p, e;
  df2_prod(a, b, p, e);
  return df2_add_prod(p, e, c);
}
// a * b - c
__device__ __forceinline__ df2 df2_fms(df2 a, df2 b, df2 c) {
  f2 p, e, s, t;
  df2_prod(a, b, p, e);
  two_diff2(p, c.hi, s, t);
  t = f2_add(t, f2_sub(e, c.lo));
  fast_two_sum2(s, t, s, t);
  return {s, t};
}
__device__ __forceinline__ df2 df2_sqr(df2 a) {
  f2 p, e;
  two_prod2(a.hi, a.hi, p, e);
  e = f2_fma(f2_add(a.hi, a.hi), a.lo, e);
  fast_two_sum2(p, e, p, e);
  return {p, e};
}
__device__ __forceinline__ df2 df2_norm2_3(df2 x0, df2 x1, df2 x2) {
  f2 p0, e0, p1, e1, p2, e2;
  two_prod2(x0.hi, x0.hi, p0, e0);
  two_prod2(x1.hi, x1.hi, p1, e1);
  two_prod2(x2.hi, x2.hi, p2, e2);
  f2 s, t0, t1;
  two_sum2(p0, p1, s, t0);
  two_sum2(s, p2, s, t1);
  const f2 c = f2_fma(x0.hi, x0.lo, f2_fma(x1.hi, x1.lo, f2_mul(x2.hi, x2.lo)));
  f2 lo = f2_add(f2_add(f2_add(e0, e1), f2_add(e2, t0)), f2_fma(f2_dup(2.0f), c, t1));
  fast_two_sum2(s, lo, s, lo);
  return {s, lo};
}

// Correctly rounded 1 / x and sqrt(x) of normal FP32 values well inside the exponent range (here
// distances of 1e-9 to 1e9), two at a time: the approximation instruction, then Newton steps with
// fused multiply-adds, the last one with an exact residual (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990). Compared with
// 1.0f / x and sqrtf(x) for every significand.
__device__ __forceinline__ f2 f2_rcp(f2 x) {
  float a, b;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(f2_x(x)));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(f2_y(x)));
  f2 y = f2_make(a, b);
  const f2 e = f2_fma(f2_neg(x), y, f2_dup(1.0f));
  return f2_fma(y, e, y);
}
__device__ __forceinline__ f2 f2_sqrt(f2 x) {
  float a, b;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(f2_x(x)));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(b) : "f"(f2_y(x)));
  const f2 y = f2_make(a, b);
  const f2 g = f2_mul(x, y), h = f2_mul(y, f2_dup(0.5f));
  const f2 d = f2_fma(f2_neg(g), g, x);
  return f2_fma(d, h, g);
}

__device__ __forceinline__ df2 df2_sqrt(df2 x) {
  const f2 s0 = f2_sqrt(x.hi);
  f2 p, e;
  two_prod2(s0, s0, p, e);
  const f2 d = f2_add(f2_sub(f2_sub(x.hi, p), e), x.lo);
  const f2 c = f2_mul(d, f2_mul(f2_dup(0.5f), f2_rcp(s0)));
  f2 h, l;
  fast_two_sum2(s0, c, h, l);
  return {h, l};
}
__device__ __forceinline__ df2 df2_rcp(df2 x) {
  const f2 y0 = f2_rcp(x.hi);
  f2 p, e;
  two_prod2(x.hi, y0, p, e);
  const f2 h = f2_fma(f2_neg(x.lo), y0, f2_sub(f2_sub(f2_dup(1.0f), p), e));
  f2 r, l;
  fast_two_sum2(y0, f2_mul(y0, h), r, l);
  return {r, l};
}

// t + (a b - c d), or t + (a b + c d) with PLUS (df_add_prod_diff with -c)
template <bool PLUS>
__device__ __forceinline__ df2 df2_add_prod_pair(df2 t, df2 a, df2 b, df2 c, df2 d) {
  f2 p, pe, q, qe, dd, de;
  two_prod2(a.hi, b.hi, p, pe);
  two_prod2(c.hi, d.hi, q, qe);
  const f2 x = f2_fma(c.hi, d.lo, f2_mul(c.lo, d.hi));
  f2 lo;
  if (PLUS) {
    two_sum2(p, q, dd, de);
    lo = f2_add(f2_add(f2_add(pe, qe), de), f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, x)));
  } else {
    two_diff2(p, q, dd, de);
    lo = f2_add(f2_add(f2_sub(pe, qe), de), f2_fma(a.hi, b.lo, f2_fma(a.lo, b.hi, f2_neg(x))));
  }
  f2 h, he;
  two_sum2(t.hi, dd, h, he);
  lo = f2_add(f2_add(lo, he), t.lo);
  fast_two_sum2(h, lo, h, lo);
  return {h, lo};
}

__device__ __forceinline__ void df2_sincos(df2 t, const float4* __restrict__ tab, df2& c, df2& s) {
  const float step0 = (float)kDfStep;
  const float step1 = (float)(kDfStep - (double)step0);
  const float step2 = (float)(kDfStep - (double)step0 - (double)step1);
  const float inv_step = (float)(1.0 / kDfStep);
  const f2 u = f2_mul(t.hi, f2_dup(inv_step));
  const float j0 = rintf(f2_x(u)), j1 = rintf(f2_y(u));
  const f2 jf = f2_make(j0, j1);
  f2 p0, e0, p1, e1;
  two_prod2(jf, f2_dup(step0), p0, e0);
  two_prod2(jf, f2_dup(step1), p1, e1);
  df2 r{f2_sub(t.hi, p0), f2_dup(0.0f)};
  r = df2_add_f(r, t.lo);
  r = df2_sub_f(r, e0);
  r = df2_sub_f(r, p1);
  r.lo = f2_sub(r.lo, f2_fma(jf, f2_dup(step2), e1));
  df2 sv;
  fast_two_sum2(r.hi, r.lo, sv.hi, sv.lo);
  const df2 s2 = df2_sqr(sv);
  const f2 z = s2.hi, mh = f2_dup(-0.5f);
  const f2 c_small = f2_mul(f2_mul(z, z), f2_fma(f2_neg(z), f2_dup(1.0f / 720.0f), f2_dup(1.0f / 24.0f)));
  const df2 cp = df2_add_f(df2{f2_mul(s2.hi, mh), f2_mul(s2.lo, mh)}, c_small);
  const f2 s_small =
      f2_mul(f2_mul(f2_neg(sv.hi), z), f2_fma(f2_neg(z), f2_dup(1.0f / 120.0f), f2_dup(1.0f / 6.0f)));
  const df2 sn = df2_add_f(sv, s_small);
  const float4 T0 = tab[((int)j0) & (kDfTab - 1)], T1 = tab[((int)j1) & (kDfTab - 1)];
  const df2 tc{f2_make(T0.x, T1.x), f2_make(T0.y, T1.y)}, ts{f2_make(T0.z, T1.z), f2_make(T0.w, T1.w)};
  c = df2_add_prod_pair<false>(tc, tc, cp, ts, sn);
  s = df2_add_prod_pair<true>(ts, ts, cp, tc, sn);
}


// ------------------------------------------------------------------------------------------
// Complex double-floats packed as (re, im): {re.hi, im.hi}, {re.lo, im.lo}; 16 bytes in memory.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ f2 f2_swap(f2 a) { return f2_make(f2_y(a), f2_x(a)); }
__device__ __forceinline__ df2 df2_swap(df2 a) { return {f2_swap(a.hi), f2_swap(a.lo)}; }
__device__ __forceinline__ df2 df2_ldc(const df2* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void df2_stc(df2* p, df2 v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.hi, v.lo);
}
// acc -= a * b (cdf_fms): first -Re a (b.re, b.im), then (Im a, -Im a) (b.im, b.re)
__device__ __forceinline__ void df2_cfms(df2& acc, df2 a, df2 b) {
  const float rh = -f2_x(a.hi), rl = -f2_x(a.lo), ih = f2_y(a.hi), il = f2_y(a.lo);
  acc = df2_fma(df2{f2_dup(rh), f2_dup(rl)}, b, acc);
  acc = df2_fma(df2{f2_make(ih, -ih), f2_make(il, -il)}, df2_swap(b), acc);
}
// |a|^2 (cdf_abs2)
__device__ __forceinline__ df64 df2_abs2(df2 a) {
  const df2 q = df2_sqr(a);
  return df2_x(q) + df2_y(q);
}
// a * b (the cdf product)
__device__ __forceinline__ df2 df2_cmul(df2 a, df2 b) {
  const float rh = f2_x(a.hi), rl = f2_x(a.lo), ih = f2_y(a.hi), il = f2_y(a.lo);
  const df2 u = df2{f2_dup(rh), f2_dup(rl)} * b;
  const df2 v = df2{f2_make(-ih, ih), f2_make(-il, il)} * df2_swap(b);
  return u + v;
}
__device__ __forceinline__ df2 df2_from_cdf(cdf a) { return df2_make(a.re, a.im); }
__device__ __forceinline__ cdf df2_to_cdf(df2 a) { return {df2_x(a), df2_y(a)}; }
__device__ __forceinline__ df2 df2_cdivide(df2 a, const CdfDivisor& D) {
  const f2 sc = f2_dup(D.sc);
  return df2_cmul(df2{f2_mul(a.hi, sc), f2_mul(a.lo, sc)}, df2_from_cdf(D.inv));
}

}  // namespace ac3d
