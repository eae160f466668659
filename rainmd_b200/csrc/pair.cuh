// The pair arithmetic of the direct-space kernels, written once for one pair (float) and for two
// pairs side by side (Pair2: the packed f32x2 instructions of sm_100, one issue slot for two
// operations, each half rounded as the scalar instruction rounds it). Every operation and
// contraction is spelled out, so both kernels compute a pair's force to the same bits. The
// group-pair kernel went from 49.7 to 46.7 us at 23,558 atoms, 169 to 160 at 99,999 and 442 to 429 at
// 250,000 with the packed form.
#pragma once

#include "common.cuh"

namespace rmd {

struct Pair2 {
  unsigned long long v;
};
__device__ __forceinline__ Pair2 pack2(float lo, float hi) {
  Pair2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(Pair2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}

__device__ __forceinline__ float op_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float op_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float op_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ Pair2 op_fma(Pair2 a, Pair2 b, Pair2 c) {
  Pair2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ Pair2 op_mul(Pair2 a, Pair2 b) {
  Pair2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair2 op_add(Pair2 a, Pair2 b) {
  Pair2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
// The hardware approximations (their arguments here are never subnormal within the cutoff).
__device__ __forceinline__ float op_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float op_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float op_rcp(float x) { return rcp_approx(x); }
__device__ __forceinline__ Pair2 op_rsqrt(Pair2 a) {
  const float2 u = unpack2(a);
  return pack2(op_rsqrt(u.x), op_rsqrt(u.y));
}
__device__ __forceinline__ Pair2 op_exp2(Pair2 a) {
  const float2 u = unpack2(a);
  return pack2(op_exp2(u.x), op_exp2(u.y));
}
__device__ __forceinline__ Pair2 op_rcp(Pair2 a) {
  const float2 u = unpack2(a);
  return pack2(op_rcp(u.x), op_rcp(u.y));
}
template <class V>
__device__ __forceinline__ V op_const(float c);
template <>
__device__ __forceinline__ float op_const<float>(float c) {
  return c;
}
template <>
__device__ __forceinline__ Pair2 op_const<Pair2>(float c) {
  return pack2(c, c);
}

template <class V>
__device__ __forceinline__ V pair_r2(V dx, V dy, V dz) {
  return op_fma(dx, dx, op_fma(dy, dy, op_mul(dz, dz)));
}

template <class V>
struct PairTerms {
  V scalar;        // force along the pair's vector, over its length
  V a12, b6;       // A/r^12, B/r^6
  V charge;        // k_e q_i q_j erfc(alpha r)
  V inv_r;
};

// Lennard-Jones and Ewald-screened Coulomb at squared distance r2. erfc and the Gaussian share one
// exponential (common.cuh erfc_and_gauss holds the fit); the reciprocal square root is refined by
// one Newton-Raphson step (rsqrt_refined).
template <class V>
__device__ __forceinline__ PairTerms<V> pair_terms(V r2, V A, V B, V qiqj, V alpha, V gauss_k) {
  auto c = [](float x) { return op_const<V>(x); };
  PairTerms<V> t;
  const V y = op_rsqrt(r2);
  t.inv_r = op_mul(y, op_fma(op_mul(op_mul(c(-0.5f), r2), y), y, c(1.5f)));
  const V inv_r2 = op_mul(t.inv_r, t.inv_r);
  const V inv_r6 = op_mul(op_mul(inv_r2, inv_r2), inv_r2);
  t.a12 = op_mul(op_mul(A, inv_r6), inv_r6);
  t.b6 = op_mul(B, inv_r6);
  const V lj = op_mul(op_fma(c(12.0f), t.a12, op_mul(c(-6.0f), t.b6)), inv_r2);
  const V z = op_mul(alpha, op_mul(r2, t.inv_r));
  const V gauss = op_exp2(op_mul(op_mul(z, z), c(-1.4426950408889634f)));
  const V u = op_rcp(op_fma(c(0.5f), z, c(1.0f)));
  V p = op_fma(c(-4.967514911e-02f), u, c(2.366592171e-01f));
  p = op_fma(p, u, c(-3.827331461e-01f));
  p = op_fma(p, u, c(1.511331490e-01f));
  p = op_fma(p, u, c(6.722758340e-02f));
  p = op_fma(p, u, c(1.595169610e-01f));
  p = op_fma(p, u, c(2.551498949e-01f));
  p = op_fma(p, u, c(2.805130003e-01f));
  p = op_fma(p, u, c(2.822084696e-01f));
  const V screened = op_mul(op_mul(u, p), gauss);
  const V qq = op_mul(c((float)ONE_4PI_EPS0), qiqj);
  t.charge = op_mul(qq, screened);
  t.scalar = op_fma(op_mul(qq, op_fma(screened, t.inv_r, op_mul(gauss_k, gauss))), inv_r2, lj);
  return t;
}

}  // namespace rmd
