// The tanh of tanh_f32.cuh for two values at once, the same bit for bit (NaN for NaN), on the packed FP32 pipe.
//
// tanh_f32 branches between its two formulas, and a warp whose values fall on both sides of 0.8
// runs both of them one value at a time (about 55 instructions). Here both are computed for a pair of values with
// the packed instructions of sm_100 (add / mul / fma .rn.f32x2: two FP32 operations, each rounded as
// the scalar one) and the result is selected: about 20 instructions per value. The operations and
// their order are those of tanh_f32, with two exact substitutions:
//   * rint(t) as (t + 1.5 2^23) - 1.5 2^23, exact for |t| < 2^22 under round-to-nearest; the low bits of the
//     sum are the integer, shifted into the exponent of 2^k;
//   * 2 / d as 2 RN(1 / d) (a power of two changes no rounding here: 5.9 < d < 1.8e8), with RN(1 / d)
//     by one Newton step on the hardware approximation, y + y (1 - d y): with a y that is good to an
//     ulp and an exact fused residual the result is the correctly rounded reciprocal except where
//     d's significand is all ones (Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", IBM J. Res. Dev. 34, 1990); the tests compare the
//     two functions for every input.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace hignn {

struct f2 {  // two FP32 values in a 64-bit register pair
  uint64_t v;
};
__device__ __forceinline__ f2 f2_make(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 f2_dup(float x) { return f2_make(x, x); }
__device__ __forceinline__ float f2_lo(f2 a) {
  float lo;
  asm("{\n.reg .f32 h;\nmov.b64 {%0, h}, %1;\n}\n" : "=f"(lo) : "l"(a.v));
  return lo;
}
__device__ __forceinline__ float f2_hi(f2 a) {
  float hi;
  asm("{\n.reg .f32 l;\nmov.b64 {l, %0}, %1;\n}\n" : "=f"(hi) : "l"(a.v));
  return hi;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ f2 tanh_f32x2(f2 x) {
  const float x0 = f2_lo(x), x1 = f2_hi(x);
  const float a0 = fabsf(x0), a1 = fabsf(x1);
  const f2 a = f2_make(a0, a1);
  // |x| < 0.8
  const f2 s = f2_mul(a, a);
  f2 p = f2_fma(f2_dup(0x1.a19af4p-10f), s, f2_dup(-0x1.e69e6cp-8f));
  p = f2_fma(p, s, f2_dup(0x1.5d356ep-6f));
  p = f2_fma(p, s, f2_dup(-0x1.b92feap-5f));
  p = f2_fma(p, s, f2_dup(0x1.110b7ep-3f));
  p = f2_fma(p, s, f2_dup(-0x1.55553ep-2f));
  const f2 ts = f2_fma(a, f2_mul(s, p), a);
  // 0.8 <= |x| < 9.5
  const f2 y = f2_add(a, a);
  const f2 km = f2_add(f2_mul(y, f2_dup(0x1.715476p+0f)), f2_dup(12582912.f));
  const f2 kf = f2_add(km, f2_dup(-12582912.f));
  const f2 r = f2_fma(kf, f2_dup(-0x1.7f7d1cp-20f), f2_fma(kf, f2_dup(-0x1.62e4p-1f), y));
  f2 q = f2_fma(f2_dup(0x1.a01a02p-13f), r, f2_dup(0x1.6c16c2p-10f));
  q = f2_fma(q, r, f2_dup(0x1.111112p-7f));
  q = f2_fma(q, r, f2_dup(0x1.555556p-5f));
  q = f2_fma(q, r, f2_dup(0x1.555556p-3f));
  q = f2_fma(q, r, f2_dup(0.5f));
  q = f2_fma(q, r, f2_dup(1.0f));
  q = f2_fma(q, r, f2_dup(1.0f));
  const f2 scale = f2_make(__int_as_float((__float_as_int(f2_lo(km)) << 23) + 0x3f800000),
                           __int_as_float((__float_as_int(f2_hi(km)) << 23) + 0x3f800000));
  const f2 d = f2_add(f2_mul(q, scale), f2_dup(1.0f));
  const f2 i0 = f2_make(rcp_approx(f2_lo(d)), rcp_approx(f2_hi(d)));
  const f2 nd = f2_make(-f2_lo(d), -f2_hi(d));
  const f2 i1 = f2_fma(i0, f2_fma(nd, i0, f2_dup(1.0f)), i0);
  const f2 tb = f2_fma(i1, f2_dup(-2.0f), f2_dup(1.0f));
  // a NaN takes the first formula, which keeps it
  const float t0 = a0 >= 0.8f ? (a0 < 9.5f ? f2_lo(tb) : 1.0f) : f2_lo(ts);
  const float t1 = a1 >= 0.8f ? (a1 < 9.5f ? f2_hi(tb) : 1.0f) : f2_hi(ts);
  return f2_make(copysignf(t0, x0), copysignf(t1, x1));
}

}  // namespace hignn
