// Self-check of the packed double-float arithmetic (df2.cuh) against the scalar one (df64.cuh), bit
// for bit, and of the packed reciprocal and square root against 1.0f / x and sqrtf(x) for every
// significand.
#include <cuda_runtime.h>

#include "../../include/ac3d.h"
#include "df2.cuh"
#include "internal.h"

namespace ac3d {

__device__ __forceinline__ bool same(df64 a, df64 b) {
  return __float_as_uint(a.hi) == __float_as_uint(b.hi) && __float_as_uint(a.lo) == __float_as_uint(b.lo);
}

__global__ void df_round_selftest_kernel(unsigned exponent, int root, unsigned long long* bad) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  const float x = __uint_as_float((exponent << 23) | m);
  // the other half of the pair holds another significand
  const float y = __uint_as_float((exponent << 23) | (m ^ 0x5a5a5au));
  const f2 r = root ? f2_sqrt(f2_make(x, y)) : f2_rcp(f2_make(x, y));
  const float wx = root ? sqrtf(x) : 1.0f / x, wy = root ? sqrtf(y) : 1.0f / y;
  if (__float_as_uint(f2_x(r)) != __float_as_uint(wx) || __float_as_uint(f2_y(r)) != __float_as_uint(wy))
    atomicAdd(bad, 1ull);
}

// a value of about 1e-3 to 1e3 with a low part below half an ulp, from a hash of (i, k)
__device__ __forceinline__ df64 hashed(unsigned i, unsigned k) {
  unsigned h = i * 2654435761u ^ (k * 0x9e3779b9u + 0x7f4a7c15u);
  h ^= h >> 16, h *= 0x85ebca6bu, h ^= h >> 13, h *= 0xc2b2ae35u, h ^= h >> 16;
  const float hi = __uint_as_float((h & 0x807fffffu) | ((117u + ((h >> 24) & 0x7fu) % 20u) << 23));
  h = h * 1664525u + 1013904223u;
  const float lo = hi * (float)(int)(h >> 8) * 0x1p-50f * ((h & 1u) ? 1.0f : -1.0f);
  df64 r;
  fast_two_sum(hi, lo, r.hi, r.lo);
  return r;
}

// The scalar operations out of line: inlined beside one another they share exact products, and the
// compiler then contracts one of them into a sum, which the functions by themselves do not have.
__device__ __noinline__ df64 r_add(df64 a, df64 b) { return a + b; }
__device__ __noinline__ df64 r_mul(df64 a, df64 b) { return a * b; }
__device__ __noinline__ df64 r_fma(df64 a, df64 b, df64 c) { return df_fma(a, b, c); }
__device__ __noinline__ df64 r_sqr(df64 a) { return df_sqr(a); }
__device__ __noinline__ df64 r_norm(df64 a, df64 b, df64 c) { return df_norm2_3(a, b, c); }
__device__ __noinline__ df64 r_sqrt(df64 a) { return df_sqrt(a); }
__device__ __noinline__ df64 r_rcp(df64 a) { return df_rcp(a); }
__device__ __noinline__ void r_sincos(df64 t, const float4* tab, df64& c, df64& s) { df_sincos(t, tab, c, s); }
__device__ __noinline__ cdf r_fms(cdf acc, cdf a, cdf b) {
  cdf_fms(acc, a, b);
  return acc;
}
__device__ __noinline__ df64 r_abs2(cdf a) { return cdf_abs2(a); }
__device__ __noinline__ cdf r_divide(cdf a, CdfDivisor d) { return cdf_divide(a, d); }

__global__ void df_ops_selftest_kernel(unsigned long long* bad) {
  __shared__ float4 tab[kDfTab];
  for (int j = threadIdx.x; j < kDfTab; j += blockDim.x) {
    double sn, cs;
    sincos(j * kDfStep, &sn, &cs);
    const df64 c = df_from_double(cs), s = df_from_double(sn);
    tab[j] = make_float4(c.hi, c.lo, s.hi, s.lo);
  }
  __syncthreads();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  df64 a[2], b[2], c[2];
  for (int k = 0; k < 2; k++) {
    a[k] = hashed(i, 3 * k);
    b[k] = hashed(i, 3 * k + 1);
    c[k] = hashed(i, 3 * k + 2);
  }
  const df2 A = df2_make(a[0], a[1]), B = df2_make(b[0], b[1]), C = df2_make(c[0], c[1]);
  const df2 P{f2_make(fabsf(a[0].hi), fabsf(a[1].hi)), f2_dup(0.0f)};
  const df2 sum = A + B, dif = A - B, mul = A * B, fm = df2_fma(A, B, C), ms = df2_fms(A, B, C), sq = df2_sqr(A);
  const df2 nm = df2_norm2_3(A, B, C), rt = df2_sqrt(nm), rc = df2_rcp(A);
  df2 cs, sn;
  df2_sincos(P, tab, cs, sn);
  bool ok = true;
  for (int k = 0; k < 2; k++) {
    auto half = [&](df2 v) { return k ? df2_y(v) : df2_x(v); };
    ok = ok && same(half(sum), r_add(a[k], b[k])) && same(half(dif), r_add(a[k], df_neg(b[k]))) && same(half(mul), r_mul(a[k], b[k]));
    ok = ok && same(half(fm), r_fma(a[k], b[k], c[k])) && same(half(ms), r_fma(a[k], b[k], df_neg(c[k])));
    ok = ok && same(half(sq), r_sqr(a[k])) && same(half(nm), r_norm(a[k], b[k], c[k]));
    ok = ok && same(half(rt), r_sqrt(half(nm))) && same(half(rc), r_rcp(a[k]));
    df64 wc, ws;
    r_sincos(half(P), tab, wc, ws);
    ok = ok && same(half(cs), wc) && same(half(sn), ws);
  }
  // complex values packed as (re, im)
  const cdf x{a[0], a[1]}, y{b[0], b[1]}, z{c[0], c[1]};
  df2 acc = C;
  df2_cfms(acc, A, B);
  cdf want = r_fms(z, x, y);
  ok = ok && same(df2_x(acc), want.re) && same(df2_y(acc), want.im) && same(df2_abs2(A), r_abs2(x));
  const CdfDivisor d = cdf_divisor(y);
  const df2 q = df2_cdivide(A, d);
  want = r_divide(x, d);
  ok = ok && same(df2_x(q), want.re) && same(df2_y(q), want.im);
  if (!ok) atomicAdd(bad, 1ull);
}

}  // namespace ac3d

extern "C" int ac3d_packed_selftest(int op, long long* mismatches) {
  using namespace ac3d;
  if (op < 0 || op > 2 || !mismatches) return AC3D_ERR_ARG;
  unsigned long long* bad = nullptr;
  cudaError_t e = cudaMalloc(&bad, sizeof(*bad));
  if (e == cudaSuccess) e = cudaMemset(bad, 0, sizeof(*bad));
  if (e == cudaSuccess) {
    if (op < 2) {
      // the exponents of 1e-9, 1/2, 1, 2 and 1e9 (both parities for the root)
      for (unsigned exponent : {97u, 126u, 127u, 128u, 156u}) {
        note_launch();
        df_round_selftest_kernel<<<(1u << 23) / 256, 256>>>(exponent, op, bad);
      }
    } else {
      note_launch();
      df_ops_selftest_kernel<<<4096, 256>>>(bad);
    }
    e = cudaGetLastError();
  }
  unsigned long long n = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&n, bad, sizeof(n), cudaMemcpyDeviceToHost);
  cudaFree(bad);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return AC3D_ERR_CUDA;
  }
  *mismatches = (long long)n;
  return AC3D_OK;
}
