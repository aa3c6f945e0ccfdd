// pair_math.cuh — the arithmetic of one neighbour pair, two pairs at a time.
//
// Correctly rounded square roots and quotients (the bits of sqrtf and of the IEEE
// division) for arguments that the host has bounded (pair_math_ranges), so that no
// range test, rescaling or slow path runs per pair. The method is Markstein's
// ("Computation of elementary functions on the IBM RISC System/6000 processor", IBM J.
// Res. Dev. 34, 1990): from an approximation y of 1 / sqrt(x), g = x y and h = y / 2,
// s = g + h (x - g g) is the rounded root; a Newton step turns y into the reciprocal
// of s; and a quotient a / s is q = a y corrected once by the exact remainder,
// q + y (a - s q), which is the rounded quotient whenever y is the rounded reciprocal.
// Checked on the device (p4a_test_pair_math) over every float: in [2^-96, 2^100] every
// root is sqrtf's, in [2^-60, 2^60] every recip() is the rounded reciprocal; the
// reciprocal of a root is the rounded one but for 10 or 24 roots per binade, and for each
// of those the quotients of all 2^23 numerators equal the IEEE division's (the
// approximation is taken one ulp up because the all-ones root fails that check without
// it).
//
// Blackwell's packed f32x2 instructions do two independent binary32 operations in one
// issue slot, each rounded as the scalar instruction rounds it (the FMA pipe is as
// busy as with two scalar ones: measured 8.1 cycles for four packed against 8.3 for
// eight scalar FMAs). The walks are bound by issue slots, so everything from r^2 on
// runs on the pair of entries (F2), and only the differences, the dot products and
// the ordered sums are scalar. The packed forms have no free negation, so the
// reciprocals are kept negated and quotients come out negated; the callers negate a
// constant factor instead. There is no packed add here: a packed product added to
// another value comes out contracted to one rounding in some kernels, so such sums are
// scalar.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace p4a {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 splat2(float a) { return pack2(a, a); }
__device__ __forceinline__ void unpack2(F2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

constexpr float kOneUp = -1.00000012f;  // -(1 + 2^-23)

// s = sqrt(x) rounded, yn = -1 / s for quot2.
struct Root2 {
  F2 s, yn;
};
__device__ __forceinline__ Root2 root2(F2 x) {
  float a, b;
  unpack2(x, a, b);
  const F2 y = pack2(rsqrt_approx(a), rsqrt_approx(b));
  Root2 r;
  const F2 g = mul2(x, y);
  r.s = fma2(fma2(g, g, mul2(x, splat2(-1.0f))), mul2(y, splat2(-0.5f)), g);
  const F2 yn = mul2(y, splat2(kOneUp));
  r.yn = fma2(fma2(r.s, yn, splat2(1.0f)), yn, yn);
  return r;
}
// -1 / d rounded, for quot2.
__device__ __forceinline__ F2 recip2(F2 d) {
  float a, b;
  unpack2(d, a, b);
  const F2 y = pack2(rcp_approx(a), rcp_approx(b)), yn = mul2(y, splat2(-1.0f));
  return fma2(fma2(d, y, splat2(-1.0f)), y, yn);
}
// -(a / s) rounded, yn = -1 / s from root2 or recip2.
__device__ __forceinline__ F2 quot2(F2 a, F2 s, F2 yn) {
  const F2 qn = mul2(a, yn);
  return fma2(fma2(s, qn, a), yn, qn);
}

// The same for one pair: s = sqrt(x) rounded, -1 / s, -1 / d, and a / s.
struct Root1 {
  float s, yn;
};
__device__ __forceinline__ Root1 root1(float x) {
  const float y = rsqrt_approx(x), g = x * y, s = fmaf(fmaf(-g, g, x), 0.5f * y, g), yn = y * kOneUp;
  return {s, fmaf(fmaf(s, yn, 1.0f), yn, yn)};
}
__device__ __forceinline__ float recip1(float d) {
  const float y = rcp_approx(d);
  return fmaf(fmaf(d, y, -1.0f), y, -y);
}
__device__ __forceinline__ float quot1(float a, float s, float yn) {
  const float qn = a * yn;
  return -fmaf(fmaf(s, qn, a), yn, qn);
}

}  // namespace p4a
