// adv_math.cuh -- correctly rounded scalar ops that the compiler may not contract into FMAs.
// The heat stage and the FP64 WENO path evaluate their expressions in the reference's operand
// order with these, so results match the CPU oracle (built with -ffp-contract=off) bit for bit.
#pragma once
#include <cuda_runtime.h>

namespace adv {

__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }

// Two FP32 lanes at once with Blackwell's paired instructions (FADD2 / FMUL2 / FFMA2): each lane
// is rounded exactly as the scalar operation, so packed code gives the scalar results bit for
// bit (as long as no paired product goes into a paired sum: the compiler fuses the two, which it
// does not do to the scalar ones). a - b is issued as fma(b, -1, a) (one rounding of the exact
// difference).
__device__ __forceinline__ float2 add_rn(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub_rn(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 mul_rn(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 div_rn(float2 a, float2 b) {
  return make_float2(__fdiv_rn(a.x, b.x), __fdiv_rn(a.y, b.y));
}
__device__ __forceinline__ float2 operator-(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ float fma_rn_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn_(double a, double b, double c) { return __fma_rn(a, b, c); }

// A constant of type T (both lanes for float2).
template <class T> __device__ __forceinline__ T bc(double v) { return T(v); }
template <> __device__ __forceinline__ float2 bc<float2>(double v) { return make_float2((float)v, (float)v); }

// x / 3, correctly rounded: the quotient x RN(1/3) corrected once by its residual (Markstein, IBM J.
// Res. Dev. 34 (1990) 111-119: exact rounding from a correctly rounded reciprocal and a quotient within
// one ulp), three operations instead of a compiled division's ten. Far from underflow and overflow only;
// other values (zeros apart) take the division.
__device__ __forceinline__ double div3(double x) {
  const double r = 1.0 / 3.0;
  const double q = __dmul_rn(x, r);
  const double y = __fma_rn(__fma_rn(-3.0, q, x), r, q);
  if ((((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 64u < 1900u) return y;
  return x == 0.0 ? x : __ddiv_rn(x, 3.0);
}
__device__ __forceinline__ float2 div3(float2 x) {
  const float2 r = make_float2(1.f / 3.f, 1.f / 3.f);
  const float2 q = __fmul2_rn(x, r);
  float2 y = __ffma2_rn(__ffma2_rn(make_float2(-3.f, -3.f), q, x), r, q);
  auto in = [](float v) { return ((__float_as_uint(v) >> 23) & 0xffu) - 32u < 190u; };
  if (!in(x.x)) y.x = x.x == 0.f ? x.x : __fdiv_rn(x.x, 3.f);
  if (!in(x.y)) y.y = x.y == 0.f ? x.y : __fdiv_rn(x.y, 3.f);
  return y;
}
__device__ __forceinline__ float div3(float x) { return __fdiv_rn(x, 3.f); }

// x / h, correctly rounded, from the correctly rounded reciprocal r = RN(1/h) (an IEEE division on the
// host): one correction makes the quotient faithful, the second rounds it exactly (Markstein, as above);
// five operations instead of a compiled division's ten. Other ranges (zeros apart) divide.
__device__ __forceinline__ double div_by(double x, double h, double r) {
  const double q0 = __dmul_rn(x, r);
  const double q1 = __fma_rn(__fma_rn(-h, q0, x), r, q0);
  const double q = __fma_rn(__fma_rn(-h, q1, x), r, q1);
  const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu, eh = ((unsigned)__double2hiint(h) >> 20) & 0x7ffu;
  if (ex - 512u < 1024u && eh - 768u < 512u) return q;
  return x == 0.0 ? x : __ddiv_rn(x, h);
}

// SSP-RK3 stage combination (stage 1 is forward Euler), operand order of
// SingleGPU/Diffusion3d_baselineCode/kernels.cu:130-138:
//   1: un + dt*L;  2: 0.75*un + 0.25*(uin + dt*L);  3: (un + 2*(uin + dt*L)) / 3
// (un + 2 x in one fused operation: 2 x is exact).
template <class T>
__device__ __forceinline__ T stage_combine(int stage, T un, T uin, T dt, T L) {
  if (stage == 2) return add_rn(mul_rn(T(0.75), un), mul_rn(T(0.25), add_rn(uin, mul_rn(dt, L))));
  if (stage == 3) return div3(fma_rn_(T(2), add_rn(uin, mul_rn(dt, L)), un));
  return add_rn(un, mul_rn(dt, L));
}

}  // namespace adv
