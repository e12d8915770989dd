// weno.cuh -- WENO5-JS / WENO5-Z face reconstruction for the Lax-Friedrichs split Burgers flux.
//
// Face flux at i+1/2:  F = R(f+_{i-2..i+2}) + R(f-_{i+3..i-1} reversed), where R is the
// left-biased 5-point reconstruction of SingleGPU/Burgers3d_WENO5/kernels.cu:142-192 (WENO5-Z)
// and :92-140 (WENO5-JS); the right-biased half of those functions is R applied to the
// mirrored stencil (same smoothness indicators, linear weights 0.1/0.6/0.3 reversed).
//
// Three forms:
//  * weno_face_ref<double>: the reference's own expression, operand for operand, with
//    correctly rounded intrinsics -> equal to the FP64 oracle bit for bit.
//  * weno_face2 / WenoLine: the same weights with the common denominator b0*b1*b2 (WENO5-Z) or
//    (b0*b1*b2)^2 (WENO5-JS) multiplied through, leaving ONE division per side instead of four,
//    and everything expressed in the cells' first and second differences, on two faces at once.
//    Used for the FP32 state and for an FP64 state with ADV_DIV_FAST.
//  * weno_face_mean (Candidates): the weighted mean of the three candidates, for FP32 WENO5-Z runs that are
//    differentiated.
#pragma once
#include <type_traits>

#include "adv_math.cuh"

namespace adv {

// Lax-Friedrichs split of f(u) = u^2/2 (kernels.cu:224-238): f+- = (f +- a u)/2.
// lf_split: the reference's operand order, correctly rounded (FP64 path, reference operators).
template <class T>
__device__ __forceinline__ void lf_split(T u, T a, T& fp, T& fm) {
  const T f = mul_rn(mul_rn(T(0.5), u), u);
  const T au = mul_rn(a, u);
  fp = mul_rn(T(0.5), add_rn(f, au));
  fm = mul_rn(T(0.5), sub_rn(f, au));
}

// ------------------------------------------------------------------ two values at once
// A pair of values: float2 operations are Blackwell's paired FP32 instructions (FFMA2 / FADD2 /
// FMUL2: one instruction, each lane rounded like the scalar operation), double2 operations two
// scalar ones. Every operation is explicit, but the compiler fuses a paired product into a paired sum that takes it
// (vmul_alone keeps one apart). The single-grid and the batched kernels round alike all the same: the only products
// that their stages add are by powers of two, which are exact.
template <class T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tsub.rn.f32x2 r, a, b;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
// a product that stays one: the paired multiplication is fused into a paired sum that follows, even with .rn
__device__ __forceinline__ float2 vmul_alone(float2 a, float2 b) { return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vabs(float2 a) { return make_float2(fabsf(a.x), fabsf(a.y)); }
__device__ __forceinline__ double2 vadd(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ double2 vmul(double2 a, double2 b) { return make_double2(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)); }
__device__ __forceinline__ double2 vfma(double2 a, double2 b, double2 c) {
  return make_double2(__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 vabs(double2 a) { return make_double2(fabs(a.x), fabs(a.y)); }
template <class V> __device__ __forceinline__ V vc(double v);  // a constant in both lanes
template <> __device__ __forceinline__ float2 vc<float2>(double v) { return make_float2((float)v, (float)v); }
template <> __device__ __forceinline__ double2 vc<double2>(double v) { return make_double2(v, v); }

// f+- = u (u/4 +- a/2).
template <class V>
__device__ __forceinline__ void lf_split2(V u, V a, V& fp, V& fm) {
  const V hu = vmul(vc<V>(0.25), u), ha = vmul(vc<V>(0.5), a);
  fp = vmul(u, vadd(hu, ha));
  fm = vmul(u, vsub(hu, ha));
}

struct FastDiv {};  // division tag: reciprocal approximation, <= 2 ulp (FP32 state)

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Negated quotient -num / den of the weight sums (den at least 6.4e-16 with WENO5-Z, 10 (4e-6)^3, and 2.5e-21 with JS,
// 10 (4e-6)^4: far from the subnormals). FP32: FastDiv multiplies by the reciprocal approximation; otherwise one
// Newton step on the reciprocal and one residual correction of the quotient in fused multiply-adds (Markstein,
// IBM J. Res. Dev. 34 (1990) 111-119). The quotient is correctly rounded where the residual is exact (|num| from
// 2^-102 on) -- what an FP64 division rounded to FP32 also returns, so both division kinds of an FP32 state share
// it: the reciprocal is the correctly rounded one for each of the 2^23 significands, which leaves only quotients
// within 2^-22 ulp of a tie in question, and all of those come out right (both compared on the GPU by
// tests/test_gpu_quotients.py). 3.5 issue slots per quotient in paired instructions; compiled IEEE divisions take about
// 10, six quotients per cell. (Negated: the reciprocal of -den makes both corrections plain multiply-adds.)
template <class D>
__device__ __forceinline__ float2 vnquot(float2 num, float2 den) {
  const float2 r0 = make_float2(rcp_approx(-den.x), rcp_approx(-den.y));
  if constexpr (std::is_same<D, FastDiv>::value) return vmul(num, r0);
  const float2 r = vfma(vfma(den, r0, vc<float2>(1)), r0, r0);
  const float2 q = vmul(num, r);
  return vfma(vfma(den, q, num), r, q);
}
template <class D>
__device__ __forceinline__ double2 vnquot(double2 num, double2 den) {
  return make_double2(-num.x / den.x, -num.y / den.y);
}

// One side of a face. With f at i-2..i+2 called a..e, first differences A = b-a .. Dd = e-d and
// second differences t0 = B-A, t1 = C-B, t2 = Dd-C, the reference's quantities are
//   4 beta_k = 13/3 t_k^2 + s_k^2,  s0 = t0 + 2B, s1 = B + C, s2 = t2 - 2C
//   q_k/6 = c + C/2 + { t0/3 - t1/2 | -t1/6 | -t2/6 }
// so the weighted mean of the q_k/6 is
//   c + C/2 - t1/6 - 1/2 [ (2/3) w0 (t1-t0) + 3 w2' (t2-t1)/3 ] / (w0 + w1 + w2),  w2 = 3 w2'
// A constant part and one quotient. b0..b2 are 4 (beta_k + eps); the weights are taken times 10 and
// times the common denominator. Against the form that weighs the three q_k this needs a quarter
// fewer operations, and its quotient only corrects the (exact in the mean) linear part, so the FP32
// rounding error of a face falls (rms 6.2e-8 -> 4.3e-8 on smooth data, 6.4e-8 -> 4.8e-8 on noise).
// Returns the negated quotient -[..]; d_a = t1-t0, d_b = t2-t1 (both negated give the quotient).
template <bool Z, class D, class V>
__device__ __forceinline__ V weno_nl(V b0, V b1, V b2, V d_a, V d_b) {
  const V p12 = vmul(b1, b2);
  V e0, e1, e2;
  if (Z) {  // alpha_k = d_k (1 + tau/b_k), times 10 b0 b1 b2: d_k (P + tau P/b_k), P = b0 b1 b2
    const V tau = vabs(vsub(b0, b2)), P = vmul(b0, p12);
    e0 = vfma(tau, p12, P);
    e1 = vfma(tau, vmul(b0, b2), P);
    e2 = vfma(tau, vmul(b0, b1), P);
  } else {  // alpha_k = d_k / b_k^2, times 10 (b0 b1 b2)^2
    const V p02 = vmul(b0, b2), p01 = vmul(b0, b1);
    e0 = vmul(p12, p12);
    e1 = vmul(p02, p02);
    e2 = vmul(p01, p01);
  }
  const V den = vfma(vc<V>(3), e2, vfma(vc<V>(6), e1, e0));
  const V num = vfma(e2, d_b, vmul(vc<V>(2.0 / 3.0), vmul(e0, d_a)));
  return vnquot<D>(num, den);
}

// 4 (beta + eps) from the second difference's share T = 13/3 t^2 + 4 eps and s.
template <class V>
__device__ __forceinline__ V weno_T(V t) {
  return vfma(vmul(vc<V>(13.0 / 3.0), t), t, vc<V>(4e-6));
}

// Side from a..e: lin = c (the caller adds C/2 and t1/6 of both sides together), C, t1, quotient.
template <bool Z, class D, class V>
__device__ __forceinline__ V weno_side2(V a, V b, V c, V d, V e, V& C, V& t1) {
  const V A = vsub(b, a), B = vsub(c, b), E = vsub(e, d);
  C = vsub(d, c);
  const V t0 = vsub(B, A), t2 = vsub(E, C);
  t1 = vsub(C, B);
  const V two = vc<V>(2);
  const V s0 = vfma(two, B, t0), s1 = vadd(B, C), s2 = vfma(vc<V>(-2), C, t2);
  return weno_nl<Z, D>(vfma(s0, s0, weno_T(t0)), vfma(s1, s1, weno_T(t1)), vfma(s2, s2, weno_T(t2)), vsub(t1, t0),
                       vsub(t2, t1));
}

// Two faces i+1/2: f+ at i-2..i+2 (p0..p4) and f- at i-1..i+3 (m0..m4) of each.
template <bool Z, class D, class V>
__device__ __forceinline__ V weno_face2(V p0, V p1, V p2, V p3, V p4, V m0, V m1, V m2, V m3, V m4) {
  V Cp, tp, Cm, tm;
  const V qp = weno_side2<Z, D>(p0, p1, p2, p3, p4, Cp, tp);
  const V qm = weno_side2<Z, D>(m4, m3, m2, m1, m0, Cm, tm);
  const V lin = vfma(vc<V>(-1.0 / 6.0), vadd(tp, tm), vfma(vc<V>(0.5), vadd(Cp, Cm), vadd(p2, m2)));
  return vfma(vc<V>(0.5), vadd(qp, qm), lin);
}

// WENO-Z of FP32 states in forward runs that an adjoint sweep follows (adv_burgers_forward). tau = |b0 - b2| has a
// kink, so a gradient jumps where the rounding of a state or of an indicator decides the sign of b0 - b2: two forms of
// the same run differ in single entries by up to 5e-3 of the gradient's rms at 24^3 .. 64^3, either of them as far from
// FP64. These runs and the adjoint take one form, and the same indicators: the candidates q_k/6 = c + t_k/12 +
// { s0/4 | s1/4 | -s2/4 } themselves, weighed (128^3: 1.8% of a gradient's 3860 us). Their sum of weights adds
// products that must not be fused into it; tests/test_gpu_burgers_gradient_form.py holds the states to the separately
// rounded operations. D: the quotient's kind.
template <class D>
struct Candidates {};
template <class D> struct IsCandidates : std::false_type {};
template <class D> struct IsCandidates<Candidates<D>> : std::true_type {};
// w_k = 4 (beta_k + eps) with t_k and s_k of a..e as above, and 13/3 t_k.
template <class V>
__device__ __forceinline__ void weno_indicators(V a, V b, V c, V d, V e, V (&t)[3], V (&s)[3], V (&k)[3], V (&w)[3]) {
  const V m2 = vc<V>(-2), m4 = vc<V>(-4), p3 = vc<V>(3), K = vc<V>(13.0 / 3.0), eps = vc<V>(4e-6);
  t[0] = vadd(vfma(m2, b, a), c); t[1] = vadd(vfma(m2, c, b), d); t[2] = vadd(vfma(m2, d, c), e);
  s[0] = vfma(p3, c, vfma(m4, b, a)); s[1] = vsub(d, b); s[2] = vfma(p3, c, vfma(m4, d, e));
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    k[i] = vmul(K, t[i]);
    w[i] = vfma(k[i], t[i], vfma(s[i], s[i], eps));
  }
}
// The negated side from a..e.
template <class D>
__device__ __forceinline__ float2 weno_side_mean(float2 a, float2 b, float2 c, float2 d, float2 e) {
  using V = float2;
  V t[3], s[3], k[3], w[3];
  weno_indicators(a, b, c, d, e, t, s, k, w);
  const V r12 = vc<V>(1.0 / 12.0), qt = vc<V>(0.25);
  const V q0 = vfma(qt, s[0], vfma(r12, t[0], c)), q1 = vfma(qt, s[1], vfma(r12, t[1], c)),
          q2 = vfma(vc<V>(-0.25), s[2], vfma(r12, t[2], c));
  const V tau = vabs(vsub(w[0], w[2])), p12 = vmul(w[1], w[2]), P = vmul(w[0], p12);
  const V w0 = vfma(tau, p12, P), w1 = vmul(vc<V>(6), vfma(tau, vmul(w[0], w[2]), P)),
          w2 = vmul(vc<V>(3), vfma(tau, vmul(w[0], w[1]), P));
  return vnquot<D>(vfma(w2, q2, vfma(w1, q1, vmul(w0, q0))), vadd(vadd(w0, w1), w2));
}
template <class D>
__device__ __forceinline__ float2 weno_face_mean(float2 p0, float2 p1, float2 p2, float2 p3, float2 p4, float2 m0,
                                                 float2 m1, float2 m2, float2 m3, float2 m4) {
  return vsub(vmul(vc<float2>(-1), weno_side_mean<D>(p0, p1, p2, p3, p4)), weno_side_mean<D>(m4, m3, m2, m1, m0));
}

// One split part along a line walked cell by cell: what neighbouring faces share (differences, the
// three indicators of a triple of cells) is computed once per cell. After push(f_n) the state holds
// f_n, D_n = f_n - f_{n-1}, t_{n-1} = D_n - D_{n-1}, d_{n-1} = t_{n-1} - t_{n-2}; of the triple
// around m = n-1 the central indicator, and the right-sided ones of n-1 and n-2. push returns the
// negated quotient of the side whose upwind cell is n-2 (PLUS: the face above it, f+) or of the side whose
// downwind cell is n-2 (the face below it, f-), and t_{n-2}.
template <class V>
struct WenoLine {
  V f, D, t, d, bc, br1, br2;
  __device__ __forceinline__ void clear() { f = D = t = d = bc = br1 = br2 = vc<V>(0); }
  // (want false: the state alone, while a segment's first planes fill it)
  template <bool Z, class DIV, bool PLUS>
  __device__ __forceinline__ V push(V fn, bool want, V& t_mid) {
    const V Dn = vsub(fn, f), tn = vsub(Dn, D), dn = vsub(tn, t), T = weno_T(tn);
    const V sl = vfma(vc<V>(-2), D, tn), sc = vadd(D, Dn), sr = vfma(vc<V>(2), Dn, tn);
    const V bl = vfma(sl, sl, T);
    t_mid = t;
    V q = vc<V>(0);
    if (want) q = PLUS ? weno_nl<Z, DIV>(br2, bc, bl, d, dn) : weno_nl<Z, DIV>(bl, bc, br2, dn, d);
    f = fn; D = Dn; t = tn; d = dn;
    bc = vfma(sc, sc, T);
    br2 = br1;
    br1 = vfma(sr, sr, T);
    return q;
  }
};

// ---------------------------------------------------------- reference literal form
// Operand order of kernels.cu:142-192 / :92-140 (and of the CPU oracle), every operation rounded on
// its own. Products by powers of two are exact (short of overflow; the quarter of C*C: weno_ref_beta), so
// they go into fused multiply-adds without changing a bit:
// 52 operations and four divisions per side instead of 66 and four. FP64 is bound by its pipe (two lanes
// per SM and cycle), so a stage's time follows this count.
// RECIP: the normalisation of SingleGPU/Burgers3d_WENO5_SharedMem/kernels.cu:51-198, which takes
// alphasum = 1/(a0 + a1 + a2) and multiplies by (1/6)*alphasum instead of dividing by 6*alphasum.

// The second difference's share of an indicator, 13/12 (a - 2b + c)^2: the same for the three sides
// that use the triple (a, b, c), always in ascending cell order.
template <class T>
__device__ __forceinline__ T weno_ref_k(T a, T b, T c) {
  const T A = add_rn(fma_rn_(T(-2), b, a), c);
  return mul_rn(mul_rn(T(13. / 12.), A), A);
}

// The three indicators K + C^2/4 from their triples' shares and first differences, (1/4 C) C rounded twice as
// written. FP64 fuses the exact quarter of C^2 instead (what a subnormal C^2 loses only ever meets eps = 1e-6 or a
// tau of the same size), except where C^2 overflows and a quarter of it need not.
__device__ __forceinline__ void weno_ref_beta(const float (&K)[3], const float (&C)[3], float (&B)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) B[i] = add_rn(K[i], mul_rn(mul_rn(0.25f, C[i]), C[i]));
}
__device__ __forceinline__ void weno_ref_beta(const double (&K)[3], const double (&C)[3], double (&B)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) B[i] = fma_rn_(0.25, mul_rn(C[i], C[i]), K[i]);
  if (max(max(__double2hiint(B[0]), __double2hiint(B[1])), __double2hiint(B[2])) >= 0x7ff00000) {
#pragma unroll
    for (int i = 0; i < 3; ++i) B[i] = add_rn(K[i], mul_rn(mul_rn(0.25, C[i]), C[i]));
  }
}

// A compiled FP64 division leaves its short form for a numerator of zero, and one such lane (a constant state,
// a tile's columns past the domain) takes its warp along: with it kept away, a stage of 121 x 101 x 97, whose
// last tiles hold seven such columns, took 1740 us instead of 2086 (1714 now), periodic 120^3 2510 instead of 3397,
// 128^3 2389 instead of 2447. Neither operation changes a result: beside an indicator of at least eps, a tau
// below 2^-100 leaves 1 + tau / (B + eps) at exactly 1 (unsigned: the NaN of two infinite indicators, which the
// absolute value may leave with its sign, is not below it) ...
__device__ __forceinline__ float weno_ref_tau(float t) { return t; }
__device__ __forceinline__ double weno_ref_tau(double t) {
  return (unsigned)__double2hiint(t) < (1023u - 100u) << 20 ? __hiloint2double((1023 - 100) << 20, 0) : t;
}
// ... and zero over a positive finite sum is the same zero. (Over any other it is not: from |u| of about 1e39 on
// every WENO5-JS weight underflows to 0, and 0/0 has to come out as NaN.)
__device__ __forceinline__ float weno_ref_quot(float n, float d) { return div_rn(n, d); }
__device__ __forceinline__ double weno_ref_quot(double n, double d) {
  const bool zero = ((__double2hiint(n) << 1) | __double2loint(n)) == 0 && (unsigned)__double2hiint(d) - 1u < 0x7fefffffu;
  const double q = div_rn(zero ? 1.0 : n, d);
  return zero ? n : q;
}

// One side from its five cells in ascending order and their three triples' shares. PLUS: f+ (weights
// 1/10, 6/10, 3/10), else f- on the mirrored candidates (3/10, 6/10, 1/10).
template <bool Z, class T, bool RECIP, bool PLUS>
__device__ __forceinline__ T weno_side_ref(T a, T b, T c, T d, T e, T K0, T K1, T K2) {
  const T eps = T(1e-6);
  const T c3 = mul_rn(T(3), c);
  const T C0 = add_rn(fma_rn_(T(-4), b, a), c3), C1 = sub_rn(b, d), C2 = add_rn(fma_rn_(T(-4), d, c3), e);
  T B[3];
  weno_ref_beta({K0, K1, K2}, {C0, C1, C2}, B);
  const T B0 = B[0], B1 = B[1], B2 = B[2];
  const T d0 = T(PLUS ? 1. / 10. : 3. / 10.), d1 = T(6. / 10.), d2 = T(PLUS ? 3. / 10. : 1. / 10.);
  T a0, a1, a2;
  if (Z) {
    const T tau5 = weno_ref_tau(fabs(sub_rn(B0, B2)));
    a0 = mul_rn(d0, add_rn(T(1), div_rn(tau5, add_rn(B0, eps))));
    a1 = mul_rn(d1, add_rn(T(1), div_rn(tau5, add_rn(B1, eps))));
    a2 = mul_rn(d2, add_rn(T(1), div_rn(tau5, add_rn(B2, eps))));
  } else {
    const T e0 = add_rn(eps, B0), e1 = add_rn(eps, B1), e2 = add_rn(eps, B2);
    a0 = div_rn(d0, mul_rn(e0, e0));
    a1 = div_rn(d1, mul_rn(e1, e1));
    a2 = div_rn(d2, mul_rn(e2, e2));
  }
  T q0, q1, q2;
  if (PLUS) {
    q0 = add_rn(fma_rn_(T(2), a, -mul_rn(T(7), b)), mul_rn(T(11), c));  // (2a - 7b) + 11c
    q1 = fma_rn_(T(2), d, add_rn(-b, mul_rn(T(5), c)));                 // (-b + 5c) + 2d
    q2 = sub_rn(fma_rn_(T(2), c, mul_rn(T(5), d)), e);                  // (2c + 5d) - e
  } else {
    q0 = fma_rn_(T(2), c, add_rn(-a, mul_rn(T(5), b)));                 // (-a + 5b) + 2c
    q1 = sub_rn(fma_rn_(T(2), b, mul_rn(T(5), c)), d);                  // (2b + 5c) - d
    q2 = fma_rn_(T(2), e, sub_rn(mul_rn(T(11), c), mul_rn(T(7), d)));   // (11c - 7d) + 2e
  }
  const T num = add_rn(add_rn(mul_rn(a0, q0), mul_rn(a1, q1)), mul_rn(a2, q2)), sum = add_rn(add_rn(a0, a1), a2);
  return RECIP ? mul_rn(num, mul_rn(T(1. / 6.), div_rn(T(1), sum))) : weno_ref_quot(num, mul_rn(T(6), sum));
}

template <bool Z, class T, bool RECIP = false>
__device__ __forceinline__ T weno_face_ref(T vmm, T vm, T v, T vp, T vpp, T umm, T um, T u, T up, T upp) {
  const T fm = weno_side_ref<Z, T, RECIP, true>(vmm, vm, v, vp, vpp, weno_ref_k(vmm, vm, v), weno_ref_k(vm, v, vp),
                                                weno_ref_k(v, vp, vpp));
  const T fp = weno_side_ref<Z, T, RECIP, false>(umm, um, u, up, upp, weno_ref_k(umm, um, u), weno_ref_k(um, u, up),
                                                 weno_ref_k(u, up, upp));
  return add_rn(fm, fp);
}

// The literal form along a line: the triples' shares are computed once per cell (K0, K1: of the two
// triples before the newest). push returns the side of the newest five cells.
template <bool Z, bool PLUS>
struct WenoRefLine {
  double2 f[4], K0, K1;  // the last four cells
  __device__ __forceinline__ void clear() {
    const double2 zero = make_double2(0.0, 0.0);
    K0 = K1 = f[0] = f[1] = f[2] = f[3] = zero;
  }
  __device__ __forceinline__ double2 push(double2 n, bool want) {
    const double2 K2 = make_double2(weno_ref_k(f[2].x, f[3].x, n.x), weno_ref_k(f[2].y, f[3].y, n.y));
    double2 r = make_double2(0.0, 0.0);
    if (want) {
      r.x = weno_side_ref<Z, double, false, PLUS>(f[0].x, f[1].x, f[2].x, f[3].x, n.x, K0.x, K1.x, K2.x);
      r.y = weno_side_ref<Z, double, false, PLUS>(f[0].y, f[1].y, f[2].y, f[3].y, n.y, K0.y, K1.y, K2.y);
    }
    K0 = K1;
    K1 = K2;
    f[0] = f[1]; f[1] = f[2]; f[2] = f[3]; f[3] = n;
    return r;
  }
};

}  // namespace adv
