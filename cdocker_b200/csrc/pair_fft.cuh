// pair_fft.cuh -- the butterflies of fft.cuh on pairs of independent complex values, one
// packed FP32 instruction (add / mul / fma .f32x2) for the two members of a pair.
//
// On sm_100a a packed instruction takes the FP32 pipe as long as its two scalar halves but one
// issue slot instead of two (measured on a B200: 36.2 T scalar FMAs/s, 37.0 T as packed FMAs), so
// kernels whose loads, stores and address arithmetic compete with the butterflies for issue
// slots gain from it. Every rounding is written out (no contraction left to the compiler) and
// follows the fused forms of fft.cuh's expressions, so the results are bit-identical to the
// scalar butterflies.
#pragma once
#include <cuda_runtime.h>

#include "fft.cuh"

namespace cdk {

// two floats in one 64-bit register pair
using pair_t = unsigned long long;

__device__ __forceinline__ pair_t pk(float lo, float hi) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpk(pair_t p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ pair_t p_add(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t p_sub(pair_t a, pair_t b) {
  pair_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t p_mul(pair_t a, pair_t b) {
  pair_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t p_fma(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// a pair of complex values: x the two real parts, y the two imaginary parts
struct cpair {
  pair_t x, y;
};
__device__ __forceinline__ cpair cp_add(cpair a, cpair b) { return {p_add(a.x, b.x), p_add(a.y, b.y)}; }
__device__ __forceinline__ cpair cp_sub(cpair a, cpair b) { return {p_sub(a.x, b.x), p_sub(a.y, b.y)}; }
// a + rot90(b), a - rot90(b) with rot90 the product with SIGN * i (c_rot90)
template <int SIGN>
__device__ __forceinline__ cpair cp_add_rot(cpair a, cpair b) {
  return SIGN < 0 ? cpair{p_add(a.x, b.y), p_sub(a.y, b.x)} : cpair{p_sub(a.x, b.y), p_add(a.y, b.x)};
}
template <int SIGN>
__device__ __forceinline__ cpair cp_sub_rot(cpair a, cpair b) {
  return cp_add_rot<-SIGN>(a, b);
}

// the radix-4 DFT (Radix<4, SIGN>)
template <int SIGN>
__device__ __forceinline__ void pair_radix4(cpair& v0, cpair& v1, cpair& v2, cpair& v3) {
  const cpair s02 = cp_add(v0, v2), d02 = cp_sub(v0, v2);
  const cpair s13 = cp_add(v1, v3), e13 = cp_sub(v1, v3);
  v0 = cp_add(s02, s13);
  v2 = cp_sub(s02, s13);
  v1 = cp_add_rot<SIGN>(d02, e13);
  v3 = cp_sub_rot<SIGN>(d02, e13);
}

template <int R, int SIGN>
struct PairRadix;

template <int SIGN>
struct PairRadix<4, SIGN> {
  __device__ __forceinline__ static void run(cpair* v) { pair_radix4<SIGN>(v[0], v[1], v[2], v[3]); }
};

template <int SIGN>
struct PairRadix<8, SIGN> {
  __device__ __forceinline__ static void run(cpair* v) {
    const float r2 = 0.70710678118654752440f;
    const pair_t pr = pk(r2, r2), nr = pk(-r2, -r2);
    cpair u[4], w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      u[j] = cp_add(v[j], v[j + 4]);
      w[j] = cp_sub(v[j], v[j + 4]);
    }
    pair_radix4<SIGN>(u[0], u[1], u[2], u[3]);
    // w1 e^(SIGN i pi/4) = r2 t1, w3 e^(SIGN 3 i pi/4) = r2 t3; their sum and difference as
    // fma(r2, t1, +-(r2 t3)), the difference kept negated (exact)
    const pair_t t1x = SIGN < 0 ? p_add(w[1].x, w[1].y) : p_sub(w[1].x, w[1].y);
    const pair_t t1y = SIGN < 0 ? p_sub(w[1].y, w[1].x) : p_add(w[1].y, w[1].x);
    // t3 = (-w3.x - SIGN w3.y, -w3.y + SIGN w3.x); the all-negative sum through -(x + y)
    cpair m3;
    if (SIGN < 0) {
      m3.x = p_mul(pr, p_sub(w[3].y, w[3].x));
      m3.y = p_mul(nr, p_add(w[3].y, w[3].x));
    } else {
      m3.x = p_mul(nr, p_add(w[3].x, w[3].y));
      m3.y = p_mul(pr, p_sub(w[3].x, w[3].y));
    }
    const cpair s13 = {p_fma(pr, t1x, m3.x), p_fma(pr, t1y, m3.y)};
    const cpair n13 = {p_fma(nr, t1x, m3.x), p_fma(nr, t1y, m3.y)};  // -(w1' - w3')
    const cpair s02 = cp_add_rot<SIGN>(w[0], w[2]), d02 = cp_sub_rot<SIGN>(w[0], w[2]);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[2 * j] = u[j];
    v[1] = cp_add(s02, s13);
    v[5] = cp_sub(s02, s13);
    v[3] = cp_sub_rot<SIGN>(d02, n13);
    v[7] = cp_add_rot<SIGN>(d02, n13);
  }
};

// u times exp(SIGN 2 pi i m / R) for the composite radices; the roots +-i are exact rotations.
// Which of a component's two products is rounded first is the scalar form's (its compiler folds
// the constants' signs: real part u.x c first and u.y s rounded, except m = 6 of R = 16 forward;
// imaginary part u.x s rounded, except m = 2 of R = 16).
template <int R, int SIGN>
__device__ __forceinline__ cpair cp_root(cpair u, int m) {
  const float2 b = unit_root<R, SIGN>(m);
  const pair_t pm1 = pk(-1.f, -1.f);
  if (4 * m == R) return SIGN < 0 ? cpair{u.y, p_mul(u.x, pm1)} : cpair{p_mul(u.y, pm1), u.x};
  if (2 * m == R) return {p_mul(u.x, pm1), p_mul(u.y, pm1)};
  const pair_t c = pk(b.x, b.x), s = pk(b.y, b.y), n = pk(-b.y, -b.y);
  cpair r;
  r.x = (R == 16 && m == 6 && SIGN < 0) ? p_fma(u.y, n, p_mul(u.x, c)) : p_fma(u.x, c, p_mul(u.y, n));
  r.y = (R == 16 && m == 2) ? p_fma(u.x, s, p_mul(u.y, c)) : p_fma(u.y, c, p_mul(u.x, s));
  return r;
}

template <int SIGN>
struct PairRadix<16, SIGN> {
  __device__ __forceinline__ static void run(cpair* v) {
    cpair u[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) u[n2][n1] = v[4 * n1 + n2];
      pair_radix4<SIGN>(u[n2][0], u[n2][1], u[n2][2], u[n2][3]);
#pragma unroll
      for (int k1 = 1; k1 < 4; ++k1)
        if (n2 > 0) u[n2][k1] = cp_root<16, SIGN>(u[n2][k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      pair_radix4<SIGN>(u[0][k1], u[1][k1], u[2][k1], u[3][k1]);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = u[k2][k1];
    }
  }
};

template <int SIGN>
struct PairRadix<12, SIGN> {
  __device__ __forceinline__ static void run(cpair* v) {
    const float h = 0.86602540378443864676f;  // sin(2 pi / 3)
    const pair_t ph = pk(h, h), nh = pk(-h, -h), mh = pk(-0.5f, -0.5f);
    cpair u[3][4];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) u[n2][n1] = v[3 * n1 + n2];
      pair_radix4<SIGN>(u[n2][0], u[n2][1], u[n2][2], u[n2][3]);
#pragma unroll
      for (int k1 = 1; k1 < 4; ++k1)
        if (n2 > 0) u[n2][k1] = cp_root<12, SIGN>(u[n2][k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      // Radix<3, SIGN>
      const cpair t = cp_add(u[1][k1], u[2][k1]), d = cp_sub(u[1][k1], u[2][k1]);
      const cpair m = {p_fma(mh, t.x, u[0][k1].x), p_fma(mh, t.y, u[0][k1].y)};
      v[k1] = cp_add(u[0][k1], t);
      // m + h rot90(d), m - h rot90(d)
      const pair_t a = SIGN < 0 ? ph : nh, b = SIGN < 0 ? nh : ph;
      v[k1 + 4] = {p_fma(a, d.y, m.x), p_fma(b, d.x, m.y)};
      v[k1 + 8] = {p_fma(b, d.y, m.x), p_fma(a, d.x, m.y)};
    }
  }
};

}  // namespace cdk
