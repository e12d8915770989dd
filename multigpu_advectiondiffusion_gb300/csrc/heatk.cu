// heatk.cu -- 3D heat with a spatially varying diffusivity k(x), its discrete adjoint, and the
// checkpointed forward/backward runs (adv_heatk_* in advdiff.h). No reference counterpart: the
// reference's diffusivity is one constant C (SingleGPU/Diffusion3d_baselineCode/main.cpp:58-61).
//
// Scheme (conservative 7-point form, arithmetic face averages), for an interior node i and each
// axis a with neighbours p (+1) and m (-1):
//   k_p = (k_i + k_p)/2, k_m = (k_i + k_m)/2,  F_a = k_p (u_p - u_i) - k_m (u_i - u_m)
//   u'_i = u_i + c_x F_x + c_y F_y + c_z F_z,   c_a = dt / h_a^2
// The outermost layer is frozen (held, or set to 0 with zero_boundary).
//
// Adjoint of one step (J depends on u' through lam' = dJ/du'): with the masked adjoint
// mu_j = [j interior] lam'_j and P_i = [i interior or not zero_boundary],
//   lam_i  = P_i lam'_i + sum_a c_a sum_{j in nb_a(i)} k_ij (mu_j - mu_i)
//   dJ/dk_i += 1/2 sum_a c_a sum_{j in nb_a(i)} (u_j - u_i)(mu_i - mu_j)
// (each face coefficient k_ij = (k_i + k_j)/2 feeds half its derivative to each end). Neighbours
// outside the domain contribute nothing.
//
// Kernels (heatk_step_kernel, heatk_adjoint_kernel): a thread owns VX nodes along x (one 16- or 8-byte
// vector where rows allow it, else one) by RY rows and marches through a chunk of z planes; loads run one
// plane ahead of their use. What a face needs -- its coefficient, the difference across it and one
// rounded product -- is computed once and serves both its ends: along z it is carried from plane to
// plane, along y and x between the thread's own nodes. x neighbours of a vector come from shuffles, y
// neighbours beyond the thread's rows from global loads that hit L1. No node tests any neighbour: mu is
// masked when it is loaded, absent neighbours are the centre's own values (the boundary's mu is 0, so
// their terms vanish as the formulas ask), and boundary nodes are fixed up afterwards in the warps that
// hold any. Every operation is an explicit correctly rounded add/mul/fma in the oracle's order, FP32 in
// pairs. Bound by the latency of the loads in flight (192^3 FP32: 12 B per node and step in 16.0 us,
// 5.3 TB/s out of HBM and L2 together; 24 B per adjoint step in 37.6 us, 4.5 TB/s). The form before this,
// one thread per column with its neighbours' tests and products per node, was issue bound in its selects:
// 59 and 171 instructions per node, 20.8 and 48.5 us (191^3, scalar rows: 26.6 -> 20.2 and 78 -> 40.2).
#include <algorithm>
#include <cstring>
#include <initializer_list>

#include "adv_device.cuh"
#include "adv_internal.h"
#include "adv_math.cuh"
#include "heatk_rows.h"
#include "nvtx_range.h"

namespace adv {

namespace {

template <class T>
struct HeatKArgs {
  const T* k;
  const T* u;    // forward: u^n; adjoint: u^n (the step's input)
  const T* lam;  // adjoint: lam^{n+1}
  T* out;        // forward: u^{n+1}; adjoint: lam^n
  T* grad;       // adjoint: dJ/dk accumulator
  int nx, ny, nz, zero_boundary;
  int zc;  // z planes per CTA
  T cx, cy, cz;
  int* status;
};

// Resident 256-thread CTAs the register budget is sized for. FP32 adjoint on vectors: two (126
// registers; three spill and run 81 us at 192^3 against 38).
template <class T, int VX, bool ADJOINT>
constexpr int heatk_min_ctas() {
  return ADJOINT ? (sizeof(T) == 4 && VX == 1 ? 3 : 2) : (sizeof(T) == 4 ? 4 : 3);
}
// N values; elementwise operations, FP32 two at a time in paired instructions (each lane rounded like
// the scalar operation).
template <class T, int N> struct VN { T v[N]; };
template <class T, int N, class F2, class F1>
__device__ __forceinline__ void each(F2 f2, F1 f1) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i + 1 < N; i += 2) f2(i);
    if constexpr (N % 2) f1(N - 1);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) f1(i);
  }
}
template <class T, int N> __device__ __forceinline__ float2 pr(const VN<T, N>& a, int i) { return make_float2(a.v[i], a.v[i + 1]); }
#define ADV_VN_PUT(r, i, w) do { const float2 w_ = (w); r.v[i] = w_.x; r.v[(i) + 1] = w_.y; } while (0)
template <class T, int N>
__device__ __forceinline__ VN<T, N> vadd(const VN<T, N>& a, const VN<T, N>& b) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, add_rn(pr(a, i), pr(b, i))); }, [&](int i) { r.v[i] = add_rn(a.v[i], b.v[i]); });
  return r;
}
template <class T, int N>
__device__ __forceinline__ VN<T, N> vsub(const VN<T, N>& a, const VN<T, N>& b) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, sub_rn(pr(a, i), pr(b, i))); }, [&](int i) { r.v[i] = sub_rn(a.v[i], b.v[i]); });
  return r;
}
template <class T, int N>
__device__ __forceinline__ VN<T, N> vmul(const VN<T, N>& a, const VN<T, N>& b) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, mul_rn(pr(a, i), pr(b, i))); }, [&](int i) { r.v[i] = mul_rn(a.v[i], b.v[i]); });
  return r;
}
template <class T, int N>
__device__ __forceinline__ VN<T, N> vscale(T s, const VN<T, N>& a) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, mul_rn(make_float2(s, s), pr(a, i))); }, [&](int i) { r.v[i] = mul_rn(s, a.v[i]); });
  return r;
}
template <class T, int N>
__device__ __forceinline__ VN<T, N> vfma(const VN<T, N>& a, const VN<T, N>& b, const VN<T, N>& c) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, __ffma2_rn(pr(a, i), pr(b, i), pr(c, i))); },
             [&](int i) { r.v[i] = fma_rn_(a.v[i], b.v[i], c.v[i]); });
  return r;
}
template <class T, int N>
__device__ __forceinline__ VN<T, N> vaxpy(T s, const VN<T, N>& a, const VN<T, N>& c) {
  VN<T, N> r;
  each<T, N>([&](int i) { ADV_VN_PUT(r, i, __ffma2_rn(make_float2(s, s), pr(a, i), pr(c, i))); },
             [&](int i) { r.v[i] = fma_rn_(s, a.v[i], c.v[i]); });
  return r;
}
#undef ADV_VN_PUT

// VX nodes in one access (VX * sizeof(T) = 16 or 8 bytes, or one node).
template <class T, int N> struct VecN { using type = T; };
template <> struct VecN<float, 4> { using type = float4; };
template <> struct VecN<float, 2> { using type = float2; };
template <> struct VecN<double, 2> { using type = double2; };
template <class T, int N>
__device__ __forceinline__ VN<T, N> ldv(const T* p) {
  const typename VecN<T, N>::type w = *reinterpret_cast<const typename VecN<T, N>::type*>(p);
  VN<T, N> r;
#pragma unroll
  for (int e = 0; e < N; ++e) r.v[e] = reinterpret_cast<const T*>(&w)[e];
  return r;
}
template <class T, int N>
__device__ __forceinline__ void stv(T* p, const VN<T, N>& v) {
  typename VecN<T, N>::type w;
#pragma unroll
  for (int e = 0; e < N; ++e) reinterpret_cast<T*>(&w)[e] = v.v[e];
  *reinterpret_cast<typename VecN<T, N>::type*>(p) = w;
}

// A thread's nodes and what its neighbours are. LX: threads per block row.
template <class T, int VX, int RY, int LX>
struct HeatKThread : HeatKRows<RY> {
  using HeatKRows<RY>::dr;
  static constexpr int N = RY * VX;
  int x, y, z0, z1;
  int nx, ny, nz;
  int64_t sz;
  int64_t first;     // offset of its first node in the grid's first plane (clamped to the grid)
  bool ok[RY];       // the row is on the grid (and so are all VX nodes)
  int left, right;   // offsets of the nodes x-1 and x+VX (clamped)
  int tx;
  __device__ __forceinline__ bool init(int gnx, int gny, int gnz, int zc) {
    tx = threadIdx.x;
    nx = gnx; ny = gny; nz = gnz;
    x = (blockIdx.x * LX + tx) * VX;
    y = (blockIdx.y * blockDim.y + threadIdx.y) * RY;
    z0 = blockIdx.z * zc;
    z1 = min(nz, z0 + zc);
    sz = (int64_t)nx * ny;
    const bool any = x < nx && y < ny;
    const int xc = min(x, nx - VX), yc = min(y, ny - 1);  // threads past the grid read its last nodes (shuffles)
    first = (int64_t)yc * nx + xc;
#pragma unroll
    for (int r = 0; r < RY; ++r) ok[r] = any && y + r < ny;
    this->set(yc, nx, ny);
    left = xc > 0 ? -1 : 0;
    right = xc + VX < nx ? VX : VX - 1;
    return any;
  }
  // a field's pointer at this thread's first node of plane z (at most the last plane)
  __device__ __forceinline__ const T* at(const T* f, int z) const { return f + (int64_t)min(z, nz - 1) * sz + first; }
  __device__ __forceinline__ VN<T, N> plane(const T* p) const {  // its nodes of a plane
    VN<T, N> a;
#pragma unroll
    for (int r = 0; r < RY; ++r) {
      const VN<T, VX> w = ldv<T, VX>(p + dr[r]);
#pragma unroll
      for (int e = 0; e < VX; ++e) a.v[r * VX + e] = w.v[e];
    }
    return a;
  }
  // the values left and right of each of its rows (at the ends of the grid: its own end nodes)
  __device__ __forceinline__ void sides(const T* p, const VN<T, N>& c, T (&l)[RY], T (&r)[RY]) const {
#pragma unroll
    for (int j = 0; j < RY; ++j) {
      if constexpr (VX == 1) {
        l[j] = p[dr[j] + left];
        r[j] = p[dr[j] + right];
      } else {
        l[j] = __shfl_up_sync(0xffffffffu, c.v[j * VX + VX - 1], 1, LX);
        r[j] = __shfl_down_sync(0xffffffffu, c.v[j * VX], 1, LX);
        if (tx == 0) l[j] = p[dr[j] + left];
        if (tx == LX - 1) r[j] = p[dr[j] + right];
      }
    }
  }
};

template <class T, int VX, int RY, int LX>
__global__ void __launch_bounds__(256, heatk_min_ctas<T, VX, false>()) heatk_step_kernel(const __grid_constant__ HeatKArgs<T> a) {
  using Th = HeatKThread<T, VX, RY, LX>;
  constexpr int N = Th::N;
  using V = VN<T, N>;
  Th t;
  const bool any = t.init(a.nx, a.ny, a.nz, a.zc);
  const T h = T(0.5);
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  bool fixed = false;  // some node of this thread on the x or y boundary
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int gx = t.x + i % VX, gy = t.y + i / VX;
    fixed |= gx <= 0 || gx >= nx - 1 || gy <= 0 || gy >= ny - 1;
  }
  const bool warp_fixed = __any_sync(0xffffffffu, fixed);
  const T* pu = t.at(a.u, t.z0);  // plane z, and two planes ahead
  const T* pk = t.at(a.k, t.z0);
  const T* pu2 = t.at(a.u, t.z0 + 2);
  const T* pk2 = t.at(a.k, t.z0 + 2);
  T* po = a.out + (pu - a.u);
  V uc = t.plane(pu), kc = t.plane(pk);
  V up = t.plane(t.at(a.u, t.z0 + 1)), kp = t.plane(t.at(a.k, t.z0 + 1));
  V npz;  // negated rounded product of the face below the plane
  {
    const int zm = max(t.z0 - 1, 0);
    const V um = t.plane(t.at(a.u, zm)), km = t.plane(t.at(a.k, zm));
    npz = vmul(vscale(h, vadd(kc, km)), vsub(um, uc));
  }
  for (int z = t.z0; z < t.z1; ++z) {
    const V un = t.plane(pu2), kn = t.plane(pk2);  // used by the next plane
    const VN<T, VX> ua = ldv<T, VX>(pu + t.above), ub = ldv<T, VX>(pu + t.below);
    const VN<T, VX> ka = ldv<T, VX>(pk + t.above), kb = ldv<T, VX>(pk + t.below);
    T ul[RY], ur[RY], kl[RY], kr[RY];
    t.sides(pu, uc, ul, ur);
    t.sides(pk, kc, kl, kr);
    // per axis F = kf_p (u_p - u) - rn(kf_m (u - u_m)), the second term negated as kf_m (u_m - u)
    V Fx, Fy, Fz;
    {
      const V kf = vscale(h, vadd(kc, kp));
      Fz = vfma(kf, vsub(up, uc), npz);
      npz = vmul(kf, vsub(uc, up));
    }
    if constexpr (VX == 1) {
      V L, R, KL, KR;
#pragma unroll
      for (int j = 0; j < RY; ++j) { L.v[j] = ul[j]; R.v[j] = ur[j]; KL.v[j] = kl[j]; KR.v[j] = kr[j]; }
      Fx = vfma(vscale(h, vadd(kc, KR)), vsub(R, uc), vmul(vscale(h, vadd(kc, KL)), vsub(L, uc)));
    } else {
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        T np = mul_rn(mul_rn(h, add_rn(kc.v[j * VX], kl[j])), sub_rn(ul[j], uc.v[j * VX]));
#pragma unroll
        for (int e = 0; e < VX; ++e) {
          const int i = j * VX + e;
          const T u1 = e + 1 < VX ? uc.v[e + 1 < VX ? i + 1 : i] : ur[j], k1 = e + 1 < VX ? kc.v[e + 1 < VX ? i + 1 : i] : kr[j];
          const T kf = mul_rn(h, add_rn(kc.v[i], k1)), d = sub_rn(u1, uc.v[i]);
          Fx.v[i] = fma_rn_(kf, d, np);
          np = mul_rn(kf, -d);
        }
      }
    }
    {
      VN<T, VX> u0, k0;  // the row above
      auto rowv = [&](const V& f, int j) {
        VN<T, VX> w;
#pragma unroll
        for (int e = 0; e < VX; ++e) w.v[e] = f.v[j * VX + e];
        return w;
      };
      u0 = rowv(uc, 0); k0 = rowv(kc, 0);
      VN<T, VX> np = vmul(vscale(h, vadd(k0, ka)), vsub(ua, u0));
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        const VN<T, VX> u1 = j + 1 < RY ? rowv(uc, j + 1 < RY ? j + 1 : j) : ub, k1 = j + 1 < RY ? rowv(kc, j + 1 < RY ? j + 1 : j) : kb;
        const VN<T, VX> kf = vscale(h, vadd(k0, k1));
        const VN<T, VX> F = vfma(kf, vsub(u1, u0), np);
        np = vmul(kf, vsub(u0, u1));
#pragma unroll
        for (int e = 0; e < VX; ++e) Fy.v[j * VX + e] = F.v[e];
        u0 = u1; k0 = k1;
      }
    }
    V res = vadd(uc, vaxpy(a.cz, Fz, vaxpy(a.cy, Fy, vscale(a.cx, Fx))));
    const bool zfix = z == 0 || z == nz - 1;
    if (warp_fixed || zfix) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int gx = t.x + i % VX, gy = t.y + i / VX;
        if (zfix || gx <= 0 || gx >= nx - 1 || gy <= 0 || gy >= ny - 1) res.v[i] = a.zero_boundary ? T(0) : uc.v[i];
      }
    }
    if (any) {
#pragma unroll
      for (int j = 0; j < RY; ++j)
        if (t.ok[j]) {
          VN<T, VX> w;
#pragma unroll
          for (int e = 0; e < VX; ++e) w.v[e] = res.v[j * VX + e];
          if (ADV_IN_RANGE(po - a.out + t.dr[j] + VX - 1, t.sz * nz, a.status)) stv<T, VX>(po + t.dr[j], w);
        }
    }
    uc = up; up = un; kc = kp; kp = kn;
    pu += t.sz; pk += t.sz; po += t.sz;
    if (z + 3 < nz) { pu2 += t.sz; pk2 += t.sz; }
  }
}

template <class T, int VX, int RY, int LX>
__global__ void __launch_bounds__(256, heatk_min_ctas<T, VX, true>()) heatk_adjoint_kernel(const __grid_constant__ HeatKArgs<T> a) {
  using Th = HeatKThread<T, VX, RY, LX>;
  constexpr int N = Th::N;
  using V = VN<T, N>;
  Th t;
  const bool any = t.init(a.nx, a.ny, a.nz, a.zc);
  const T h = T(0.5);
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  auto in1 = [](int i, int n) { return i > 0 && i < n - 1; };
  // which nodes of this thread (bit i), of the rows beside it and of the columns beside it lie off the
  // x and y boundary; warps without a boundary node anywhere near need no masks
  unsigned inb = 0, ina = 0, inl = 0, inr = 0, inbl = 0;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (in1(t.x + i % VX, nx) && in1(t.y + i / VX, ny)) inb |= 1u << i;
#pragma unroll
  for (int e = 0; e < VX; ++e) {
    if (in1(t.x + e, nx) && in1(t.y - 1, ny)) ina |= 1u << e;
    if (in1(t.x + e, nx) && in1(t.y + RY, ny)) inbl |= 1u << e;
  }
#pragma unroll
  for (int j = 0; j < RY; ++j) {
    if (in1(t.x - 1, nx) && in1(t.y + j, ny)) inl |= 1u << j;
    if (in1(t.x + VX, nx) && in1(t.y + j, ny)) inr |= 1u << j;
  }
  constexpr unsigned ALL = (1u << N) - 1u, ROW = (1u << VX) - 1u, COL = (1u << RY) - 1u;
  const bool warp_masked = __any_sync(0xffffffffu, inb != ALL || ina != ROW || inbl != ROW || inl != COL || inr != COL);
  auto mask = [&](V m, int z) {  // lam of plane z -> mu
    if (warp_masked || !in1(z, nz)) {
      const unsigned b = in1(z, nz) ? inb : 0u;
#pragma unroll
      for (int i = 0; i < N; ++i) m.v[i] = (b >> i) & 1u ? m.v[i] : T(0);
    }
    return m;
  };
  const T* pu = t.at(a.u, t.z0);  // plane z, and two planes ahead
  const T* pk = t.at(a.k, t.z0);
  const T* pl = t.at(a.lam, t.z0);
  const T* pu2 = t.at(a.u, t.z0 + 2);
  const T* pk2 = t.at(a.k, t.z0 + 2);
  const T* pl2 = t.at(a.lam, t.z0 + 2);
  T* po = a.out + (pu - a.u);
  T* pg = a.grad + (pu - a.u);
  V uc = t.plane(pu), kc = t.plane(pk), mc = mask(t.plane(pl), t.z0);
  V kfz, dmz, duz;  // the face below the plane: coefficient, mu and u differences (upper - lower)
  {
    const int zm = max(t.z0 - 1, 0);
    const V um = t.plane(t.at(a.u, zm)), km = t.plane(t.at(a.k, zm));
    const V mm = t.z0 > 0 ? mask(t.plane(t.at(a.lam, zm)), zm) : mc;
    kfz = vscale(h, vadd(kc, km));
    dmz = vsub(mc, mm);
    duz = vsub(uc, um);
  }
  V up, kp, mp;
  {
    const int zp = min(t.z0 + 1, nz - 1);
    up = t.plane(t.at(a.u, zp)); kp = t.plane(t.at(a.k, zp));
    mp = mask(t.plane(t.at(a.lam, zp)), zp);
  }
  for (int z = t.z0; z < t.z1; ++z) {
    const int z2 = min(z + 2, nz - 1);
    const V un = t.plane(pu2), kn = t.plane(pk2), ln = t.plane(pl2);  // used by the next plane
    const V g = t.plane(pg);
    const VN<T, VX> ua = ldv<T, VX>(pu + t.above), ub = ldv<T, VX>(pu + t.below);
    const VN<T, VX> ka = ldv<T, VX>(pk + t.above), kb = ldv<T, VX>(pk + t.below);
    VN<T, VX> ma = ldv<T, VX>(pl + t.above), mb = ldv<T, VX>(pl + t.below);
    T ul[RY], ur[RY], kl[RY], kr[RY], ml[RY], mr[RY];
    t.sides(pu, uc, ul, ur);
    t.sides(pk, kc, kl, kr);
    t.sides(pl, mc, ml, mr);
    const bool zin = in1(z, nz);
    if (warp_masked || !zin) {
#pragma unroll
      for (int e = 0; e < VX; ++e) {
        if (!zin || !((ina >> e) & 1u)) ma.v[e] = T(0);
        if (!zin || !((inbl >> e) & 1u)) mb.v[e] = T(0);
      }
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        if (!zin || !((inl >> j) & 1u)) ml[j] = T(0);
        if (!zin || !((inr >> j) & 1u)) mr[j] = T(0);
      }
    }
    // Per axis S = kf_m (mu_m - mu) + rn(kf_p (mu_p - mu)), G = (u_m - u) (mu - mu_m) + rn((u_p - u)(mu - mu_p)):
    // a face with differences dm, du (upper - lower) gives its lower end rn(kf dm) and rn(du (-dm)),
    // its upper end kf (-dm) and (-du) dm, all in the signs of the formulas.
    V Sx, Gx, Sy, Gy, Sz, Gz;
    auto ends = [&](auto kf0, auto dm0, auto du0, auto kf1, auto dm1, auto du1, auto& S, auto& G) {
      auto neg = [](auto v) {
#pragma unroll
        for (auto& e : v.v) e = -e;
        return v;
      };
      S = vfma(kf0, neg(dm0), vmul(kf1, dm1));
      G = vfma(neg(du0), dm0, vmul(du1, neg(dm1)));
    };
    {
      const V kf = vscale(h, vadd(kc, kp)), dm = vsub(mp, mc), du = vsub(up, uc);
      ends(kfz, dmz, duz, kf, dm, du, Sz, Gz);
      kfz = kf; dmz = dm; duz = du;
    }
    if constexpr (VX == 1) {
      V L, R, KL, KR, ML, MR;
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        L.v[j] = ul[j]; R.v[j] = ur[j]; KL.v[j] = kl[j]; KR.v[j] = kr[j]; ML.v[j] = ml[j]; MR.v[j] = mr[j];
      }
      ends(vscale(h, vadd(kc, KL)), vsub(mc, ML), vsub(uc, L), vscale(h, vadd(kc, KR)), vsub(MR, mc), vsub(R, uc), Sx, Gx);
    } else {
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        const int i0 = j * VX;
        T kf0 = mul_rn(h, add_rn(kc.v[i0], kl[j])), dm0 = sub_rn(mc.v[i0], ml[j]), du0 = sub_rn(uc.v[i0], ul[j]);
#pragma unroll
        for (int e = 0; e < VX; ++e) {
          const int i = i0 + e, n = e + 1 < VX ? i + 1 : i;
          const T u1 = e + 1 < VX ? uc.v[n] : ur[j], k1 = e + 1 < VX ? kc.v[n] : kr[j], m1 = e + 1 < VX ? mc.v[n] : mr[j];
          const T kf = mul_rn(h, add_rn(kc.v[i], k1)), dm = sub_rn(m1, mc.v[i]), du = sub_rn(u1, uc.v[i]);
          Sx.v[i] = fma_rn_(kf0, -dm0, mul_rn(kf, dm));
          Gx.v[i] = fma_rn_(-du0, dm0, mul_rn(du, -dm));
          kf0 = kf; dm0 = dm; du0 = du;
        }
      }
    }
    {
      auto rowv = [&](const V& f, int j) {
        VN<T, VX> w;
#pragma unroll
        for (int e = 0; e < VX; ++e) w.v[e] = f.v[j * VX + e];
        return w;
      };
      VN<T, VX> u0 = rowv(uc, 0), k0 = rowv(kc, 0), m0 = rowv(mc, 0);
      VN<T, VX> kf0 = vscale(h, vadd(k0, ka)), dm0 = vsub(m0, ma), du0 = vsub(u0, ua);
#pragma unroll
      for (int j = 0; j < RY; ++j) {
        const int n = j + 1 < RY ? j + 1 : j;
        const VN<T, VX> u1 = j + 1 < RY ? rowv(uc, n) : ub, k1 = j + 1 < RY ? rowv(kc, n) : kb, m1 = j + 1 < RY ? rowv(mc, n) : mb;
        const VN<T, VX> kf = vscale(h, vadd(k0, k1)), dm = vsub(m1, m0), du = vsub(u1, u0);
        VN<T, VX> S, G;
        ends(kf0, dm0, du0, kf, dm, du, S, G);
#pragma unroll
        for (int e = 0; e < VX; ++e) { Sy.v[j * VX + e] = S.v[e]; Gy.v[j * VX + e] = G.v[e]; }
        u0 = u1; k0 = k1; m0 = m1; kf0 = kf; dm0 = dm; du0 = du;
      }
    }
    V keep = mc;
    if (!a.zero_boundary && (warp_masked || !zin)) {
      const V l = t.plane(pl);
#pragma unroll
      for (int i = 0; i < N; ++i) keep.v[i] = l.v[i];
    }
    const V out = vadd(keep, vaxpy(a.cz, Sz, vaxpy(a.cy, Sy, vscale(a.cx, Sx))));
    const V gn = vaxpy(h, vaxpy(a.cz, Gz, vaxpy(a.cy, Gy, vscale(a.cx, Gx))), g);
    if (any) {
#pragma unroll
      for (int j = 0; j < RY; ++j)
        if (t.ok[j]) {
          VN<T, VX> w, q;
#pragma unroll
          for (int e = 0; e < VX; ++e) { w.v[e] = out.v[j * VX + e]; q.v[e] = gn.v[j * VX + e]; }
          if (ADV_IN_RANGE(po - a.out + t.dr[j] + VX - 1, t.sz * nz, a.status)) {
            stv<T, VX>(po + t.dr[j], w);
            stv<T, VX>(pg + t.dr[j], q);
          }
        }
    }
    uc = up; up = un; kc = kp; kp = kn; mc = mp;
    mp = mask(ln, z2);
    pu += t.sz; pk += t.sz; pl += t.sz; po += t.sz; pg += t.sz;
    if (z + 3 < nz) { pu2 += t.sz; pk2 += t.sz; pl2 += t.sz; }
  }
}

// Launch forms: rows of whole vectors in aligned arrays, or one node per thread along x.
template <class T> struct HeatKForm;
template <> struct HeatKForm<float> {
  static constexpr int STEP_VX = 4, STEP_RY = 1, ADJ_VX = 2, ADJ_RY = 2;
};
template <> struct HeatKForm<double> {
  static constexpr int STEP_VX = 2, STEP_RY = 1, ADJ_VX = 2, ADJ_RY = 1;
};
constexpr int kLxVec = 16, kLxOne = 32;  // threads per block row
constexpr int kRyOne = 2;                // rows per thread, one node along x

adv_status heatk_validate(const adv_heatk_desc* d) {
  if (!d) return set_error(ADV_ERR_INVALID_ARG, "heatk: null descriptor");
  if (d->dtype != ADV_F32 && d->dtype != ADV_F64) return set_error(ADV_ERR_INVALID_ARG, "heatk: bad dtype");
  if (d->nx < 1 || d->ny < 1 || d->nz < 1) return set_error(ADV_ERR_INVALID_ARG, "heatk: empty grid");
  if ((int64_t)d->nx * d->ny * d->nz > ((int64_t)1 << 40) || d->nx > (1 << 30) || d->ny > (1 << 30) ||
      d->nz > (1 << 30))
    return set_error(ADV_ERR_INVALID_ARG, "heatk: grid too large");
  return ADV_OK;
}

template <class T>
HeatKArgs<T> make_args(const adv_heatk_desc& d, const void* k, const void* u, const void* lam, void* out, void* grad) {
  HeatKArgs<T> a;
  a.k = static_cast<const T*>(k);
  a.u = static_cast<const T*>(u);
  a.lam = static_cast<const T*>(lam);
  a.out = static_cast<T*>(out);
  a.grad = static_cast<T*>(grad);
  a.nx = d.nx; a.ny = d.ny; a.nz = d.nz;
  a.zero_boundary = d.zero_boundary;
  a.cx = (T)d.cx; a.cy = (T)d.cy; a.cz = (T)d.cz;
  a.status = device_status_ptr();
  return a;
}

// The vector kernels need whole 16-byte vectors per row and 16-byte aligned arrays.
bool vec_ok(const adv_heatk_desc& d, std::initializer_list<const void*> ptrs) {
  const int vx = d.dtype == ADV_F32 ? 4 : 2;
  if (d.nx % vx != 0) return false;
  for (const void* p : ptrs)
    if ((uintptr_t)p % 16 != 0) return false;
  return true;
}

// Block height and z planes per CTA: the autotuner's choice for this problem, else (its default
// candidate, 8 and 16, included) 8 and what gives one wave of CTAs: a chunk's two extra planes are cheap
// against idle SMs (16 planes left a 64^3 grid 2 CTAs per SM at 12.6 us per step, one wave runs 2.5) and
// against a second, nearly empty wave (192^3 step: 16.0 us; 8 planes, 1.1 waves: 21). bx, by: nodes per
// CTA at height 8.
void heatk_shape(const adv_heatk_desc& d, int kind, const void* kernel, int lx, int bx, int by, int* ky, int* zc) {
  const TuneParams tp = tune_lookup(kind, d.dtype, d.nx, d.ny, d.nz);
  if (tp.set && !(tp.a == 8 && tp.b == 16)) {
    *ky = tp.a;
    *zc = tp.b;
    return;
  }
  *ky = 8;
  DeviceInfo di;
  const int sms = device_info(&di) == ADV_OK ? di.sms : 152;
  int occ = 0;
  if (kernel_setup(kernel, lx * 8, 0, &occ) != ADV_OK) occ = 4;
  const int64_t tiles = (int64_t)((d.nx + bx - 1) / bx) * ((d.ny + by - 1) / by);
  const int64_t chunks = std::max<int64_t>(1, std::min<int64_t>(d.nz, (int64_t)sms * occ / tiles));
  *zc = (int)((d.nz + chunks - 1) / chunks);
}

// Grid of a kernel with vx x ry nodes per thread and lx threads per block row.
dim3 heatk_grid(const adv_heatk_desc& d, int vx, int ry, int lx, int ky, int zc) {
  const int bx = vx * lx, by = ry * ky;
  return dim3((unsigned)((d.nx + bx - 1) / bx), (unsigned)((d.ny + by - 1) / by), (unsigned)((d.nz + zc - 1) / zc));
}

template <class T, int VX, int RY, int LX>
adv_status heatk_step_t(const adv_heatk_desc& d, const void* k, const void* u_in, void* u_out, cudaStream_t s) {
  int ky, zc;
  const auto kernel = &heatk_step_kernel<T, VX, RY, LX>;
  heatk_shape(d, TUNE_HEATK_STEP, reinterpret_cast<const void*>(kernel), LX, VX * LX, RY * 8, &ky, &zc);
  if (LX > 16) ky = std::min(ky, 8);  // 256 threads at most
  HeatKArgs<T> a = make_args<T>(d, k, u_in, nullptr, u_out, nullptr);
  a.zc = zc;
  kernel<<<heatk_grid(d, VX, RY, LX, ky, zc), dim3(LX, ky), 0, s>>>(a);
  ADV_CUDA_TRY(cudaGetLastError());
  count_launches(1);
  return ADV_OK;
}

template <class T, int VX, int RY, int LX>
adv_status heatk_adjoint_t(const adv_heatk_desc& d, const void* k, const void* u_n, const void* lam_next, void* lam_out,
                           void* grad_k, cudaStream_t s) {
  int ky, zc;
  const auto kernel = &heatk_adjoint_kernel<T, VX, RY, LX>;
  heatk_shape(d, TUNE_HEATK_ADJ, reinterpret_cast<const void*>(kernel), LX, VX * LX, RY * 8, &ky, &zc);
  if (LX > 16) ky = std::min(ky, 8);
  HeatKArgs<T> a = make_args<T>(d, k, u_n, lam_next, lam_out, grad_k);
  a.zc = zc;
  kernel<<<heatk_grid(d, VX, RY, LX, ky, zc), dim3(LX, ky), 0, s>>>(a);
  ADV_CUDA_TRY(cudaGetLastError());
  count_launches(1);
  return ADV_OK;
}

template <class T>
adv_status heatk_step_any(const adv_heatk_desc& d, const void* k, const void* u_in, void* u_out, cudaStream_t s) {
  using Fm = HeatKForm<T>;
  return vec_ok(d, {k, u_in, u_out}) ? heatk_step_t<T, Fm::STEP_VX, Fm::STEP_RY, kLxVec>(d, k, u_in, u_out, s)
                                     : heatk_step_t<T, 1, kRyOne, kLxOne>(d, k, u_in, u_out, s);
}

template <class T>
adv_status heatk_adjoint_any(const adv_heatk_desc& d, const void* k, const void* u_n, const void* lam_next, void* lam_out,
                             void* grad_k, cudaStream_t s) {
  using Fm = HeatKForm<T>;
  return vec_ok(d, {k, u_n, lam_next, lam_out, grad_k})
             ? heatk_adjoint_t<T, Fm::ADJ_VX, Fm::ADJ_RY, kLxVec>(d, k, u_n, lam_next, lam_out, grad_k, s)
             : heatk_adjoint_t<T, 1, kRyOne, kLxOne>(d, k, u_n, lam_next, lam_out, grad_k, s);
}

adv_status heatk_step_launch(const adv_heatk_desc& d, const void* k, const void* u_in, void* u_out, cudaStream_t s) {
  return d.dtype == ADV_F32 ? heatk_step_any<float>(d, k, u_in, u_out, s) : heatk_step_any<double>(d, k, u_in, u_out, s);
}

adv_status heatk_adjoint_launch(const adv_heatk_desc& d, const void* k, const void* u_n, const void* lam_next,
                                void* lam_out, void* grad_k, cudaStream_t s) {
  return d.dtype == ADV_F32 ? heatk_adjoint_any<float>(d, k, u_n, lam_next, lam_out, grad_k, s)
                            : heatk_adjoint_any<double>(d, k, u_n, lam_next, lam_out, grad_k, s);
}

size_t array_bytes(const adv_heatk_desc& d) {
  const size_t n = (size_t)d.nx * d.ny * d.nz * (d.dtype == ADV_F32 ? 4 : 8);
  return (n + 255) / 256 * 256;
}

}  // namespace

// for the autotuner
adv_status heatk_validate_desc(const adv_heatk_desc* d) { return heatk_validate(d); }
adv_status heatk_step_run(const adv_heatk_desc& d, const void* k, const void* u_in, void* u_out, cudaStream_t s) {
  return heatk_step_launch(d, k, u_in, u_out, s);
}
adv_status heatk_adjoint_run(const adv_heatk_desc& d, const void* k, const void* u_n, const void* lam_next,
                             void* lam_out, void* grad_k, cudaStream_t s) {
  return heatk_adjoint_launch(d, k, u_n, lam_next, lam_out, grad_k, s);
}

}  // namespace adv

using namespace adv;

extern "C" {

adv_status adv_heatk_step(const adv_heatk_desc* d, const void* k, const void* u_in, void* u_out, void* stream) {
  ADV_NVTX_RANGE("adv_heatk_step");
  adv_status st = heatk_validate(d);
  if (st != ADV_OK) return st;
  if (!k || !u_in || !u_out) return set_error(ADV_ERR_INVALID_ARG, "heatk: null buffer");
  if (u_in == u_out) return set_error(ADV_ERR_INVALID_ARG, "heatk: u_in and u_out must not alias");
  return heatk_step_launch(*d, k, u_in, u_out, static_cast<cudaStream_t>(stream));
}

adv_status adv_heatk_adjoint_step(const adv_heatk_desc* d, const void* k, const void* u_n, const void* lam_next,
                                  void* lam_out, void* grad_k, void* stream) {
  ADV_NVTX_RANGE("adv_heatk_adjoint_step");
  adv_status st = heatk_validate(d);
  if (st != ADV_OK) return st;
  if (!k || !u_n || !lam_next || !lam_out || !grad_k) return set_error(ADV_ERR_INVALID_ARG, "heatk: null buffer");
  if (lam_next == lam_out) return set_error(ADV_ERR_INVALID_ARG, "heatk: lam_next and lam_out must not alias");
  return heatk_adjoint_launch(*d, k, u_n, lam_next, lam_out, grad_k, static_cast<cudaStream_t>(stream));
}

adv_status adv_heatk_checkpoint_bytes(const adv_heatk_desc* d, int64_t nsteps, int64_t interval, size_t* ckpt_bytes,
                                      size_t* work_bytes) {
  adv_status st = heatk_validate(d);
  if (st != ADV_OK) return st;
  if (nsteps < 0 || interval < 1) return set_error(ADV_ERR_INVALID_ARG, "heatk: bad nsteps/interval");
  const size_t one = array_bytes(*d);
  const int64_t m = (nsteps + interval - 1) / interval;
  if (ckpt_bytes) *ckpt_bytes = (size_t)std::max<int64_t>(m, 1) * one;
  // forward: one ping-pong array; backward: the segment's states (interval - 1 beyond the
  // checkpoint) and one adjoint ping-pong array
  if (work_bytes) *work_bytes = (size_t)std::max<int64_t>(interval, 1) * one;
  return ADV_OK;
}

adv_status adv_heatk_forward(const adv_heatk_desc* d, const void* k, void* u, int64_t nsteps, int64_t interval,
                             void* ckpt, void* work, void* stream) {
  ADV_NVTX_RANGE("adv_heatk_forward");
  adv_status st = heatk_validate(d);
  if (st != ADV_OK) return st;
  if (!k || !u || !work) return set_error(ADV_ERR_INVALID_ARG, "heatk: null buffer");
  if (nsteps < 0 || interval < 1) return set_error(ADV_ERR_INVALID_ARG, "heatk: bad nsteps/interval");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t one = array_bytes(*d);
  const size_t nb = (size_t)d->nx * d->ny * d->nz * (d->dtype == ADV_F32 ? 4 : 8);
  char* const ub = static_cast<char*>(u);
  char* const wb = static_cast<char*>(work);
  char* const cb = static_cast<char*>(ckpt);
  // A step whose result is a checkpoint writes it into its slot (only u^0 is copied), so storing
  // checkpoints costs no traffic beyond the steps themselves; with interval 1 every state is kept
  // and the backward run recomputes nothing. The last interval runs from its checkpoint through
  // work's slots (the states u^{n0+1} .. u^{nsteps-1}, where adv_heatk_backward would recompute
  // them) into u.
  const int64_t m = (nsteps + interval - 1) / interval;
  const int64_t n_last = ckpt && nsteps > 0 ? (m - 1) * interval : nsteps;
  const char* src = ub;
  if (ckpt && nsteps > 0) ADV_CUDA_TRY(cudaMemcpyAsync(cb, ub, nb, cudaMemcpyDeviceToDevice, s));
  for (int64_t n = 0; n < n_last; ++n) {
    char* dst = ckpt && (n + 1) % interval == 0 ? cb + ((n + 1) / interval) * one : (src == ub ? wb : ub);
    if ((st = heatk_step_launch(*d, k, src, dst, s)) != ADV_OK) return st;
    src = dst;
  }
  if (n_last < nsteps) {
    src = cb + (m - 1) * one;  // u^{n_last}: the copy of u^0 or the step that wrote it there
    for (int64_t n = n_last; n < nsteps; ++n) {
      char* dst = n + 1 < nsteps ? wb + (n - n_last) * one : ub;
      if ((st = heatk_step_launch(*d, k, src, dst, s)) != ADV_OK) return st;
      src = dst;
    }
  } else if (src != ub) {
    ADV_CUDA_TRY(cudaMemcpyAsync(ub, src, nb, cudaMemcpyDeviceToDevice, s));
  }
  return ADV_OK;
}

adv_status adv_heatk_backward(const adv_heatk_desc* d, const void* k, int64_t nsteps, int64_t interval,
                              const void* ckpt, void* lam, void* grad_k, void* work, int flags, void* stream) {
  ADV_NVTX_RANGE("adv_heatk_backward");
  adv_status st = heatk_validate(d);
  if (st != ADV_OK) return st;
  if (!k || !ckpt || !lam || !grad_k || !work) return set_error(ADV_ERR_INVALID_ARG, "heatk: null buffer");
  if (nsteps < 0 || interval < 1) return set_error(ADV_ERR_INVALID_ARG, "heatk: bad nsteps/interval");
  if (flags & ~ADV_HEATK_LAST_INTERVAL_IN_WORK) return set_error(ADV_ERR_INVALID_ARG, "heatk: unknown flags");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t one = array_bytes(*d);
  const size_t nb = (size_t)d->nx * d->ny * d->nz * (d->dtype == ADV_F32 ? 4 : 8);
  char* states = static_cast<char*>(work);              // u^{n0+1} .. u^{n0+interval-1}
  char* lam_b = states + (size_t)(interval - 1) * one;  // adjoint ping-pong
  char* la = static_cast<char*>(lam);
  char* lb = lam_b;
  const int64_t m = (nsteps + interval - 1) / interval;
  for (int64_t seg = m - 1; seg >= 0; --seg) {
    const int64_t n0 = seg * interval, n1 = std::min(nsteps, n0 + interval);
    const char* base = static_cast<const char*>(ckpt) + seg * one;
    auto state = [&](int64_t n) -> const char* { return n == n0 ? base : states + (n - n0 - 1) * one; };
    const bool kept = seg == m - 1 && (flags & ADV_HEATK_LAST_INTERVAL_IN_WORK);
    for (int64_t n = n0; !kept && n + 1 < n1; ++n)
      if ((st = heatk_step_launch(*d, k, state(n), states + (n - n0) * one, s)) != ADV_OK) return st;
    for (int64_t n = n1 - 1; n >= n0; --n) {
      if ((st = heatk_adjoint_launch(*d, k, state(n), la, lb, grad_k, s)) != ADV_OK) return st;
      std::swap(la, lb);
    }
  }
  if (la != static_cast<char*>(lam)) ADV_CUDA_TRY(cudaMemcpyAsync(lam, la, nb, cudaMemcpyDeviceToDevice, s));
  return ADV_OK;
}

}  // extern "C"
