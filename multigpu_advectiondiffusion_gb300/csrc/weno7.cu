// weno7.cu -- the seventh-order WENO Burgers solver of the reference's MATLAB prototypes on the GPU
// (Matlab_Prototipes/InviscidBurgersNd/WENO7resAdv_{X,Y,Z}.m, LFWENO7FDM{2,3}d.m:65-104).
//
// Scheme (per axis, on every line of the grid):
//   * local Lax-Friedrichs split f+- = (f +- |u| u)/2 of f = u^2/2 at every node;
//   * the line extended past its ends by copies of its end values (a clamped index), faces at
//     i+1/2 for i = 0..N-1, the face left of node 0 taken as 0;
//   * the seven-point WENO of Balsara & Shu (J. Comput. Phys. 160 (2000) 405-452): four cubic
//     candidates, linear weights 1/35, 12/35, 18/35, 4/35, weights d_k / (eps + beta_k)^2,
//     eps = 1e-6, the prototype's integer quadratic-form smoothness indicators
//     (WENO7resAdv_X.m:75-82);
//   * res_i = (((hp_{i+1/2} + hn_{i+1/2}) - hp_{i-1/2}) - hn_{i-1/2}) / h, summed over the axes in
//     axis order;
//   * time: dt = CFL dx / max|u| trimmed to land on tEnd, the five-stage fourth-order 2N-storage
//     Runge-Kutta scheme of Carpenter & Kennedy (NASA TM-109112, 1994): r = A_s r + dt R(u),
//     u = u - B_s r.
// For the FP64 state every operation is evaluated in the prototypes' operand order with correctly
// rounded intrinsics (no contraction), so its results are those of the prototypes -- and of the
// CPU oracle that restates them -- bit for bit; the FP32 state evaluates the same scheme in a fused
// kernel of its own (weno7_fused_kernel below).
//
// Kernels. FP64, per stage and axis: a face kernel (one thread per face i+1/2, the two split parts'
// reconstructions hp and hn into two face arrays) and a residual kernel (one thread per node,
// accumulating the axis's residual into the stage's right-hand side); the last axis's residual
// kernel also applies the Runge-Kutta update in place and, at the last stage, reduces max|u| for
// the next step's dt. Threads run along x, so every access of every axis is coalesced. FP32: one launch
// per stage, the state going u -> a -> b -> a -> b -> u through two work arrays. The time loop is one
// CUDA graph with a device-driven while node (the step-start kernel of the Burgers loop: dt rule, trim,
// t in FP64); a run of a few steps at most is launched directly, each step predicated on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>

#include "adv_device.cuh"
#include "adv_internal.h"
#include "adv_math.cuh"
#include "nvtx_range.h"
#include "weno.cuh"

namespace adv {
namespace {

// Smoothness indicator of WENO7 candidate k over its cells x0..x3, in the prototype's order:
//   x2 (k0 x2 + k1 x3) + x0 (((k2 xb + k3 xc) + k4 xd) + k5 x3) + k6 x3 x3 + x1 ((k7 xs + k8 xt) + k9 x3)
// (the same table as the oracle's kW7Beta).
struct W7B {
  int b, c, d, s, t;
  double k[10];
};
__device__ constexpr W7B kBeta[4] = {
    {2, 1, 0, 2, 1, {134241, -114894, 56694, -47214, 6649, -22778, 25729, -210282, 85641, 86214}},
    {1, 0, 2, 1, 2, {41001, -30414, -19374, 3169, 19014, -5978, 6649, 33441, -70602, 23094}},
    {0, 1, 2, 1, 2, {33441, -19374, 6649, -30414, 23094, -5978, 3169, 41001, -70602, 19014}},
    {0, 1, 2, 1, 2, {85641, -47214, 25729, -114894, 86214, -22778, 6649, 134241, -210282, 56694}},
};
// candidates (c0 x0 + c1 x1 + c2 x2 + c3 x3)/12: the part moving towards +x (cells i-3+k .. i+k)
// and towards -x (cells i-2+k .. i+1+k); linear weights of each
__device__ constexpr double kPolyP[4][4] = {{-3, 13, -23, 25}, {1, -5, 13, 3}, {-1, 7, 7, -1}, {3, 13, -5, 1}};
__device__ constexpr double kPolyM[4][4] = {{1, -5, 13, 3}, {-1, 7, 7, -1}, {3, 13, -5, 1}, {25, -23, 13, -3}};
__device__ constexpr double kLinP[4] = {1. / 35., 12. / 35., 18. / 35., 4. / 35.};
__device__ constexpr double kLinM[4] = {4. / 35., 18. / 35., 12. / 35., 1. / 35.};

// Carpenter & Kennedy LSRK(5,4) coefficients (the published rational values).
__device__ constexpr double kA[5] = {0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
                                     -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0};
__device__ constexpr double kB[5] = {1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
                                     1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
                                     2277821191437.0 / 14882151754819.0};

// One split part's face value from its seven cells f[0..6] (candidate k uses f[k..k+3]).
template <class T, bool PLUS>
__device__ __forceinline__ T weno7_part(const T (&f)[7]) {
  const T eps = T(1e-6);
  T a[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T* x = f + k;
    const W7B& B = kBeta[k];
    const T t1 = mul_rn(x[2], add_rn(mul_rn(T(B.k[0]), x[2]), mul_rn(T(B.k[1]), x[3])));
    const T t2 = mul_rn(x[0], add_rn(add_rn(add_rn(mul_rn(T(B.k[2]), x[B.b]), mul_rn(T(B.k[3]), x[B.c])),
                                            mul_rn(T(B.k[4]), x[B.d])),
                                     mul_rn(T(B.k[5]), x[3])));
    const T t3 = mul_rn(T(B.k[6]), mul_rn(x[3], x[3]));
    const T t4 = mul_rn(x[1], add_rn(add_rn(mul_rn(T(B.k[7]), x[B.s]), mul_rn(T(B.k[8]), x[B.t])),
                                     mul_rn(T(B.k[9]), x[3])));
    const T beta = add_rn(add_rn(add_rn(t1, t2), t3), t4);
    const T e = add_rn(eps, beta);
    a[k] = div_rn(T(PLUS ? kLinP[k] : kLinM[k]), mul_rn(e, e));
  }
  const T sum = add_rn(add_rn(add_rn(a[0], a[1]), a[2]), a[3]);
  T h = T(0);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const T* x = f + k;
    const double* c = PLUS ? kPolyP[k] : kPolyM[k];
    const T cand = add_rn(add_rn(add_rn(mul_rn(T(c[0]), x[0]), mul_rn(T(c[1]), x[1])), mul_rn(T(c[2]), x[2])),
                          mul_rn(T(c[3]), x[3]));
    const T term = div_rn(mul_rn(div_rn(a[k], sum), cand), T(12));
    h = k == 0 ? term : add_rn(h, term);
  }
  return h;
}

// f+- of one node value (WENO7resAdv_X.m's split with a = |u|).
template <class T>
__device__ __forceinline__ void split(T v, T& fp, T& fm) {
  const T f = div_rn(mul_rn(v, v), T(2));
  const T av = mul_rn(fabs(v), v);
  fp = mul_rn(T(0.5), add_rn(f, av));
  fm = mul_rn(T(0.5), sub_rn(f, av));
}

struct W7Geom {
  int nx, ny, nz;
  int64_t n;
};

// Face kernel of axis AX: for every node (the face i+1/2 on its right along AX) the two parts'
// reconstructions into hp / hn. active (may be null): 0 in a step past the run's end, which computes nothing.
template <class T, int AX>
__global__ void __launch_bounds__(256) weno7_face_kernel(const T* __restrict__ u, T* __restrict__ hp,
                                                         T* __restrict__ hn, W7Geom g, const int* active) {
  if (active && *active == 0) return;
  const int64_t stride = AX == 0 ? 1 : AX == 1 ? (int64_t)g.nx : (int64_t)g.nx * g.ny;
  const int N = AX == 0 ? g.nx : AX == 1 ? g.ny : g.nz;
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < g.n; o += (int64_t)gridDim.x * blockDim.x) {
    const int64_t line_pos = AX == 0 ? o % g.nx : AX == 1 ? (o / g.nx) % g.ny : o / ((int64_t)g.nx * g.ny);
    const int i = (int)line_pos;
    const T* line = u + (o - (int64_t)i * stride);
    T fp[8], fm[8];  // cells i-3 .. i+4 (clamped)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int c = min(max(i + j - 3, 0), N - 1);
      split<T>(line[(int64_t)c * stride], fp[j], fm[j]);
    }
    T p[7], m[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      p[j] = fp[j];      // cells i-3 .. i+3
      m[j] = fm[j + 1];  // cells i-2 .. i+4
    }
    hn[o] = weno7_part<T, true>(p);
    hp[o] = weno7_part<T, false>(m);
  }
}

// ------------------------------------------------------------------ FP32 fused stage
// One launch per Runge-Kutta stage: R(u) of all axes, then r = A r + dt R, u_out = u - B r (or R alone for
// adv_weno7_rhs). 16 bytes per cell and stage (u, r read; r, u_out written) where separate face and
// residual kernels moved 92.
//
// The scheme in differences. With f at i-3 .. i+3, D2_j the second difference at j, c3_k the third
// difference of candidate k's cells (k = 0: i-3..i, .., 3: i..i+3) and s_j = f_{j+1} - f_{j-1}, the
// prototype's integer indicators are, for every candidate, the same form of its cubic's derivatives
// at i:
//   beta_k / 720 = G_k^2 + 13/3 C_k^2 + 781/180 c3_k^2
//   G_1 = s_i - c3_1/4, G_2 = s_i - c3_2/4, C_1 = C_2 = D2_i
//   G_0 = s_{i-1} + 2 D2_{i-1} + 3/4 c3_0, C_0 = D2_{i-1} + c3_0
//   G_3 = s_{i+1} - 2 D2_{i+1} + 3/4 c3_3, C_3 = D2_{i+1} - c3_3
// (expanded, the sixteen coefficients of kBeta), and the candidates' face values differ by fourth
// differences D4: v_1 - v_2 = D4_i/12, v_0 - v_1 = -D4_{i-1}/4, v_3 - v_2 = D4_{i+1}/12. So a side is
// the symmetric candidate v_2 plus one quotient; both sides' v_2 add up to (7 (w_i + w_{i+1}) -
// (w_{i-1} + w_{i+2}))/12 with w = f+ + f- = u^2/2. Weights d_k/(eps + beta_k)^2 come from r_k = e_min/e_k
// (e_k = (eps + beta_k)/720, e_min the smallest): alpha_k = d_k r_k^2 lies in (0, d_k] and the largest is at
// least d_min, so no product overflows, underflows or leaves a zero sum. Reciprocals are the
// approximation (1 ulp). No term cancels to less than its own rounding, unlike the integer forms.
//
// Layout as the WENO5 stage (burgers_kernels.cuh): 32 x 16 columns per CTA, two adjacent in x per
// thread; planes with a halo of 4 stream through an 8-slot ring (cp.async from a list of the clamped
// in-plane offsets); f+- of the output plane go to shared memory in pairs of rows (x-faces) and of
// columns (y-faces); z-faces come from register windows; three barriers per plane (copies landed, parts split, faces done). Bound by the FMA pipe
// and the barriers (pipe 54% busy, 459 paired FP32 instructions of 922 per pair of cells): right-hand side
// 256^3 383 us with two CTAs per SM, 371 with three; a run of 3 steps at 160^3 2556 -> 1743 us against
// six face and residual launches per stage.
struct W7Tile {
  static constexpr int BX = 32, BY = 16, NT = 256, PX = BX / 2, R = 4;
  static constexpr int SW = BX + 2 * R, SH = BY + 2 * R, PLANE = SW * SH;
  static constexpr int NS = 8, P = 3;
  static constexpr int XS = SW;                            // x-face operands per pair of rows
  static constexpr int PART = BY / 2 * XS + SH * PX;       // pairs of one split part
  static constexpr int XF = BX + 2;
  static constexpr size_t SMEM = (size_t)NS * PLANE * 4 + (size_t)(2 * PART + (BY + 1) * PX) * 8 + (size_t)BY * XF * 4 +
                                 (size_t)PLANE * 8;
};

struct W7Params {
  const float* u;
  float* out;  // the new state, or R(u)
  float* r;    // 2N-storage register; null: R(u) alone
  int nx, ny, nz, tiles_x, tiles_y;
  WorkSplit split;  // of the (tile, plane) pairs over the CTAs
  int stage;
  int vec_ok;  // out and r: pairs of nodes aligned for one access
  float rhx, rhy, rhz;
  const double* dt_dev;
  unsigned* maxkey;
  const int* active;
  int* status;
};

// The nonlinear part of one side for two faces, times 12: 12 (side - v_2); cells i-3 .. i+3.
__device__ __forceinline__ float2 w7_side2(const float2 (&f)[7]) {
  auto c = [](double v) { return vc<float2>(v); };
  float2 D1[6], D2[5], D3[4];
#pragma unroll
  for (int j = 0; j < 6; ++j) D1[j] = vsub(f[j + 1], f[j]);
#pragma unroll
  for (int j = 0; j < 5; ++j) D2[j] = vsub(D1[j + 1], D1[j]);  // at cells i-2 .. i+2
#pragma unroll
  for (int j = 0; j < 4; ++j) D3[j] = vsub(D2[j + 1], D2[j]);
  const float2 s0 = vadd(D1[1], D1[2]), s1 = vadd(D1[2], D1[3]), s2 = vadd(D1[3], D1[4]);
  float2 T[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) T[j] = vfma(vmul(c(781.0 / 180.0), D3[j]), D3[j], c(1e-6 / 720.0));
  const float2 K = vmul(vmul(c(13.0 / 3.0), D2[2]), D2[2]);
  const float2 C0 = vadd(D2[1], D3[0]), C3 = vsub(D2[3], D3[3]);
  const float2 G1 = vfma(c(-0.25), D3[1], s1), G2 = vfma(c(-0.25), D3[2], s1);
  const float2 G0 = vfma(c(0.75), D3[0], vfma(c(2), D2[1], s0)), G3 = vfma(c(0.75), D3[3], vfma(c(-2), D2[3], s2));
  const float2 e0 = vfma(G0, G0, vfma(vmul(c(13.0 / 3.0), C0), C0, T[0])), e1 = vfma(G1, G1, vadd(K, T[1]));
  const float2 e2 = vfma(G2, G2, vadd(K, T[2])), e3 = vfma(G3, G3, vfma(vmul(c(13.0 / 3.0), C3), C3, T[3]));
  const float2 em = make_float2(fminf(fminf(e0.x, e1.x), fminf(e2.x, e3.x)), fminf(fminf(e0.y, e1.y), fminf(e2.y, e3.y)));
  auto sq = [&](float2 e) {
    const float2 r = vmul(em, make_float2(rcp_approx(e.x), rcp_approx(e.y)));
    return vmul(r, r);
  };
  const float2 a0 = sq(e0), a1 = sq(e1), a2 = sq(e2), a3 = sq(e3);  // x 1, 12, 18, 4
  const float2 den = vfma(c(18), a2, vfma(c(12), a1, vfma(c(4), a3, a0)));
  const float2 q0 = vsub(D3[1], D3[0]), q1 = vsub(D3[2], D3[1]), q2 = vsub(D3[3], D3[2]);  // D4 at i-1, i, i+1
  const float2 num = vfma(vmul(c(12), a1), q1, vfma(vmul(c(4), a3), q2, vmul(a0, vfma(c(-3), q0, q1))));
  return vmul(num, make_float2(rcp_approx(den.x), rcp_approx(den.y)));
}

__device__ __forceinline__ void w7_split2(float2 u, float2& fp, float2& fm) { lf_split2(u, vabs(u), fp, fm); }

__global__ void __launch_bounds__(256, 3) weno7_fused_kernel(const __grid_constant__ W7Params p) {
  using TL = W7Tile;
  constexpr int R = TL::R, SW = TL::SW, PX = TL::PX, XS = TL::XS, PART = TL::PART, YP = TL::BY / 2 * XS;
  if (p.active && *p.active == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* const ring = reinterpret_cast<float*>(smem_raw);
  float2* const part = reinterpret_cast<float2*>(ring + TL::NS * TL::PLANE);  // f+; f- PART pairs later
  float2* const fyS = part + 2 * PART;                                        // y-faces [BY+1][PX]
  float* const fxS = reinterpret_cast<float*>(fyS + (TL::BY + 1) * PX);       // x-faces [BY][XF]
  int64_t* const src = reinterpret_cast<int64_t*>(fxS + TL::BY * TL::XF);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cp = tid & (PX - 1), row = tid / PX;
  const int own = (row + R) * SW + R + 2 * cp;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const size_t sxy = (size_t)nx * ny;
  const bool twod = nz == 1;
  const int lag = twod ? 0 : R;
  const float A = (float)kA[p.stage], B = (float)kB[p.stage];
  const float dt = p.r ? (float)*p.dt_dev : 0.f;
  unsigned kmax = 0;
  // halo splits, two values each: threads [0, 128) the eight halo rows, [128, 192) the eight halo columns
  const bool halo = tid < 8 * PX + 8 * (TL::BY / 2);
  int h_src, h_step;
  float2* h_dst;
  if (tid < 8 * PX) {
    const int h = tid / PX, r = h < R ? h : h + TL::BY;
    h_src = r * SW + R + 2 * cp;
    h_step = 1;
    h_dst = part + YP + r * PX + cp;
  } else {
    const int i = tid - 8 * PX, rp = (i / 8) % (TL::BY / 2), h = i % 8, c = h < R ? h : h + TL::BX;
    h_src = (2 * rp + R) * SW + c;
    h_step = SW;
    h_dst = part + rp * XS + c;
  }
  // the last x-face of each row pair (lanes [0, 8)) and the top row of y-faces (lanes [8, 24))
  const bool l_x = lane < TL::BY / 2;
  const int l_st = l_x ? 1 : PX;
  const int l_src = l_x ? lane * XS + TL::BX : YP + TL::BY * PX + (lane - TL::BY / 2);
  unsigned n = 0;  // stream entries so far (slot n % NS)

  int64_t seg_a, seg_b;
  split_range(p.split, blockIdx.x, nz, &seg_a, &seg_b);
  for (int64_t pos = seg_a; pos < seg_b;) {
    const int64_t tile = div_units(pos, nz);
    const int zs = (int)(pos - tile * nz);
    const int ze = (int)min((int64_t)nz, zs + (seg_b - pos));
    pos += ze - zs;
    const int64_t ty = div_units(tile, p.tiles_x);
    const int x0 = (int)(tile - ty * p.tiles_x) * TL::BX, y0 = (int)ty * TL::BY;
    const int Q = (ze - zs) + 2 * lag;
    for (int e = tid; e < TL::PLANE; e += TL::NT) {  // (each thread reads back only what it wrote)
      const int r = e / SW, c = e - r * SW;
      src[e] = (int64_t)min(max(y0 - R + r, 0), ny - 1) * nx + min(max(x0 - R + c, 0), nx - 1);
    }
    auto slot = [&](int q) { return ring + ((n + (unsigned)q) % TL::NS) * TL::PLANE; };
    auto issue = [&](int q) {
      if (q < Q) {
        float* const dst = slot(q);
        const float* const plane = p.u + (size_t)min(max(zs - lag + q, 0), nz - 1) * sxy;
        for (int e = tid; e < TL::PLANE; e += TL::NT)
          cp_async_zfill<4>(dst + e, plane + src[e], ADV_IN_RANGE(plane + src[e] - p.u, sxy * nz, p.status));
      }
      cp_async_commit();
    };
    for (int q = 0; q <= TL::P; ++q) issue(q);

    const int x = x0 + 2 * cp, y = y0 + row;
    const bool in0 = x < nx && y < ny, in1 = x + 1 < nx && y < ny;
    const bool vec = p.vec_ok && in1;
    size_t gi = (size_t)zs * sxy + (size_t)y * nx + x;
    float2 fp[7], fm[7], fp_new = vc<float2>(0);  // f+ at q-7 .. q-1, f- at q-6 .. q
#pragma unroll
    for (int k = 0; k < 7; ++k) fp[k] = fm[k] = vc<float2>(0);
    float2 w1 = vc<float2>(0), w2 = w1, w3 = w1;  // u^2 at planes q-3, q-4, q-5
    float2 fz_prev = vc<float2>(0);
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const float* const plq = slot(q);
      const float* const plc = slot(q - lag);  // the output plane
      cp_async_wait<TL::P>();
      __syncthreads();  // plane q visible
      const bool out = q >= 2 * lag;
      const float2 uc = *reinterpret_cast<const float2*>(plc + own);
      if (out) {
        float2 a, b;
        w7_split2(uc, a, b);
        float2* const yw = part + YP + R * PX + tid;
        yw[0] = a;
        yw[PART] = b;
        float* const xw = reinterpret_cast<float*>(part + warp * XS + 2 * cp + R) + (row & 1);
        xw[0] = a.x; xw[2] = a.y;
        xw[2 * PART] = b.x; xw[2 * PART + 2] = b.y;
        if (halo) {
          w7_split2(make_float2(plc[h_src], plc[h_src + h_step]), a, b);
          h_dst[0] = a;
          h_dst[PART] = b;
        }
      }
      // ---- the z-face between planes q-4 and q-3
      float2 fz = vc<float2>(0);
      if (!twod) {
        float2 a, b;
        w7_split2(*reinterpret_cast<const float2*>(plq + own), a, b);
        const float2 u2 = *reinterpret_cast<const float2*>(slot(q - 2) + own);  // (before plane 2: stale, not used)
        const float2 w0 = vmul(u2, u2);
#pragma unroll
        for (int k = 0; k < 6; ++k) { fp[k] = fp[k + 1]; fm[k] = fm[k + 1]; }
        fp[6] = fp_new;
        fp_new = a;
        fm[6] = b;
        if (q >= 2 * R - 1 && zs - 2 * R + q >= 0) {  // (the face below plane 0 is 0)
          const float2 qp = w7_side2(fp);
          const float2 m[7] = {fm[6], fm[5], fm[4], fm[3], fm[2], fm[1], fm[0]};
          const float2 lin = vfma(vc<float2>(3.5), vadd(w1, w2), vmul(vc<float2>(-0.5), vadd(w0, w3)));
          fz = vmul(vc<float2>(1.0 / 12.0), vadd(lin, vadd(qp, w7_side2(m))));
        }
        w3 = w2; w2 = w1; w1 = w0;
      }
      __syncthreads();  // f+- in place; every read of the output plane's slot is done
      issue(q + TL::P + 1);
      if (out) {
        float2 rr = vc<float2>(0);
        if (p.r && p.stage > 0) {  // requested before the faces, used after them (stage 0: A = 0)
          if (vec) {
            if (ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) rr = *reinterpret_cast<const float2*>(p.r + gi);
          } else {
            if (in0 && ADV_IN_RANGE(gi, sxy * nz, p.status)) rr.x = p.r[gi];
            if (in1 && ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) rr.y = p.r[gi + 1];
          }
        }
        auto face = [](const float2* a, int st) {
          const float2* const b = a + PART;
          const float2 f[7] = {a[0], a[st], a[2 * st], a[3 * st], a[4 * st], a[5 * st], a[6 * st]};
          const float2 m[7] = {b[7 * st], b[6 * st], b[5 * st], b[4 * st], b[3 * st], b[2 * st], b[st]};
          // cells i-1, i, i+1, i+2: f[2..5] and m[5..2]
          const float2 in = vadd(vadd(f[3], m[4]), vadd(f[4], m[3])), ex = vadd(vadd(f[2], m[5]), vadd(f[5], m[2]));
          const float2 lin = vfma(vc<float2>(7), in, vmul(vc<float2>(-1), ex));
          return vmul(vc<float2>(1.0 / 12.0), vadd(lin, vadd(w7_side2(f), w7_side2(m))));
        };
        float2 fx = face(part + warp * XS + lane, 1);
        if (x0 + lane == 0) fx = vc<float2>(0);  // the face left of the first node
        fxS[(2 * warp) * TL::XF + lane] = fx.x;
        fxS[(2 * warp + 1) * TL::XF + lane] = fx.y;
        float2 fym = face(part + YP + tid, PX);
        if (y == 0) fym = vc<float2>(0);
        fyS[tid] = fym;
        if (warp == (q & 7) && lane < TL::BY / 2 + PX) {
          const float2 f = face(part + l_src, l_st);
          if (l_x) {
            fxS[(2 * lane) * TL::XF + TL::BX] = f.x;
            fxS[(2 * lane + 1) * TL::XF + TL::BX] = f.y;
          } else {
            fyS[TL::BY * PX + lane - TL::BY / 2] = f;
          }
        }
        __syncthreads();
        const float2 fx0 = *reinterpret_cast<const float2*>(fxS + row * TL::XF + 2 * cp);
        const float2 fx1 = make_float2(fx0.y, fxS[row * TL::XF + 2 * cp + 2]);
        const float2 fyp = fyS[tid + PX];
        const float2 L = vfma(vsub(fz, fz_prev), make_float2(p.rhz, p.rhz),
                              vfma(vsub(fyp, fym), make_float2(p.rhy, p.rhy), vmul(vsub(fx1, fx0), make_float2(p.rhx, p.rhx))));
        float2 res = L;
        if (p.r) {
          rr = vfma(make_float2(A, A), rr, vmul(make_float2(dt, dt), L));
          res = vfma(make_float2(-B, -B), rr, uc);
          const unsigned k0 = in0 ? abs_key(res.x) : 0u, k1 = in1 ? abs_key(res.y) : 0u;
          kmax = max(kmax, max(k0, k1));
        }
        auto put = [&](float* dst, float2 v) {
          if (vec) {
            if (ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) *reinterpret_cast<float2*>(dst + gi) = v;
          } else {
            if (in0 && ADV_IN_RANGE(gi, sxy * nz, p.status)) dst[gi] = v.x;
            if (in1 && ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) dst[gi + 1] = v.y;
          }
        };
        put(p.out, res);
        if (p.r) put(p.r, rr);
        gi += sxy;
      }
      fz_prev = fz;
    }
    n += (unsigned)Q;
  }
  if (p.maxkey) {
    kmax = warp_max(kmax);
    if (lane == 0 && kmax) atomicMax(p.maxkey, kmax);
  }
}

template <class T, int AX>
void weno7_face_launch(const T* u, T* hp, T* hn, const W7Geom& g, const int* active, int grid, cudaStream_t s) {
  weno7_face_kernel<T, AX><<<grid, 256, 0, s>>>(u, hp, hn, g, active);
}

// Residual kernel of axis AX: res_i = (((hp_i + hn_i) - hp_{i-1}) - hn_{i-1}) / h (0 for the face
// left of node 0), accumulated into acc (FIRST: acc = res). LAST: then the Runge-Kutta update
// r = A r + dt acc, u = u - B r in place, and (REDUCE) max|u_new| into *maxkey.
constexpr int kW7ResZ = 16;  // z planes per thread of the tiled residual kernel

// TILED: a 3D grid of 32 x 8 (x, y) tiles, each thread walking kW7ResZ z planes of its column,
// so a node's line position comes from its coordinates; otherwise a grid-stride loop over the
// flat index (whose line position takes an integer division).
template <class T, int AX, bool FIRST, bool LAST, bool TILED>
__global__ void __launch_bounds__(256) weno7_residual_kernel(const T* __restrict__ hp, const T* __restrict__ hn,
                                                             T* __restrict__ acc, T* __restrict__ r, T* __restrict__ u,
                                                             W7Geom g, T h, int stage, const double* dt_dev,
                                                             typename KeyOf<T>::type* maxkey, const int* active) {
  using K = typename KeyOf<T>::type;
  if (active && *active == 0) return;
  const int64_t stride = AX == 0 ? 1 : AX == 1 ? (int64_t)g.nx : (int64_t)g.nx * g.ny;
  const T A = T(kA[stage]), B = T(kB[stage]);
  const T dt = LAST ? T(*dt_dev) : T(0);
  K kmax = 0;
  int64_t o, o_end, o_step;
  int64_t i = 0;
  if (TILED) {
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    const int z0 = blockIdx.z * kW7ResZ, z1 = min(g.nz, z0 + kW7ResZ);
    const bool in = x < g.nx && y < g.ny;
    o_step = (int64_t)g.nx * g.ny;
    o = (int64_t)z0 * o_step + (int64_t)y * g.nx + x;
    o_end = in ? o + (int64_t)(z1 - z0) * o_step : o;
    i = AX == 0 ? x : AX == 1 ? y : z0;
  } else {
    o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    o_end = g.n;
    o_step = (int64_t)gridDim.x * blockDim.x;
  }
  for (; o < o_end; o += o_step, i += (TILED && AX == 2) ? 1 : 0) {
    if (!TILED) i = AX == 0 ? o % g.nx : AX == 1 ? (o / g.nx) % g.ny : o / ((int64_t)g.nx * g.ny);
    const T hp0 = i > 0 ? hp[o - stride] : T(0), hn0 = i > 0 ? hn[o - stride] : T(0);
    const T res = div_rn(sub_rn(sub_rn(add_rn(hp[o], hn[o]), hp0), hn0), h);
    const T L = FIRST ? res : add_rn(acc[o], res);
    if (!LAST) {
      acc[o] = L;
    } else {
      const T rn = add_rn(mul_rn(A, r[o]), mul_rn(dt, L));
      r[o] = rn;
      const T un = sub_rn(u[o], mul_rn(B, rn));
      u[o] = un;
      if (maxkey) {
        const K k = abs_key(un);
        kmax = k > kmax ? k : kmax;
      }
    }
  }
  if (LAST && maxkey) {
    kmax = warp_max(kmax);
    if ((threadIdx.x & 31) == 0 && kmax) atomicMax(maxkey, kmax);
  }
}

// Residual launch of axis AX: the tiled kernel where its grid fits, else the grid-stride one.
template <class T, int AX, bool FIRST, bool LAST>
void weno7_residual_launch(const T* hp, const T* hn, T* acc, T* r, T* u, const W7Geom& g, T h, int stage,
                           const double* dt_dev, typename KeyOf<T>::type* maxkey, const int* active, int grid,
                           cudaStream_t s) {
  const int64_t gx = (g.nx + 31) / 32, gy = (g.ny + 7) / 8, gz = (g.nz + kW7ResZ - 1) / kW7ResZ;
  if (gx <= 0x7fffffff && gy <= 65535 && gz <= 65535)
    weno7_residual_kernel<T, AX, FIRST, LAST, true><<<dim3((unsigned)gx, (unsigned)gy, (unsigned)gz), 256, 0, s>>>(
        hp, hn, acc, r, u, g, h, stage, dt_dev, maxkey, active);
  else
    weno7_residual_kernel<T, AX, FIRST, LAST, false><<<grid, 256, 0, s>>>(hp, hn, acc, r, u, g, h, stage, dt_dev,
                                                                          maxkey, active);
}

adv_status weno7_validate(const adv_weno7_desc* d) {
  if (!d) return set_error(ADV_ERR_INVALID_ARG, "weno7: null descriptor");
  if (d->dtype != ADV_F32 && d->dtype != ADV_F64) return set_error(ADV_ERR_INVALID_ARG, "weno7: bad dtype");
  if (d->nx < 1 || d->ny < 1 || d->nz < 1) return set_error(ADV_ERR_INVALID_ARG, "weno7: empty grid");
  if (d->ny < 2) return set_error(ADV_ERR_UNSUPPORTED, "weno7: 2D and 3D grids only (ny >= 2)");
  if ((int64_t)d->nx * d->ny * d->nz > ((int64_t)1 << 36)) return set_error(ADV_ERR_INVALID_ARG, "weno7: grid too large");
  if (!(d->dx > 0) || !(d->dy > 0) || !(d->dz > 0)) return set_error(ADV_ERR_INVALID_ARG, "weno7: spacing must be > 0");
  return ADV_OK;
}

size_t weno7_array_bytes(const adv_weno7_desc& d) {
  const size_t n = (size_t)d.nx * d.ny * d.nz;
  return (n * (d.dtype == ADV_F32 ? 4 : 8) + 255) / 256 * 256;
}

int weno7_ndim(const adv_weno7_desc& d) { return d.nz > 1 ? 3 : 2; }

// Workspace: hp, hn, acc, r, then the loop state.
struct W7Work {
  char *hp, *hn, *acc, *r;
  BurgersLoopState* st;
};
W7Work weno7_work(const adv_weno7_desc& d, void* ws) {
  const size_t one = weno7_array_bytes(d);
  char* b = static_cast<char*>(ws);
  return W7Work{b, b + one, b + 2 * one, b + 3 * one, reinterpret_cast<BurgersLoopState*>(b + 4 * one)};
}

int weno7_grid(const adv_weno7_desc& d) {
  DeviceInfo di;
  const int sms = device_info(&di) == ADV_OK ? di.sms : 152;
  const int64_t n = (int64_t)d.nx * d.ny * d.nz;
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sms * 16));
}

// One FP32 stage (out: the new state; r: the 2N-storage register) or, with r null, R(u) alone.
adv_status weno7_fused(const adv_weno7_desc& d, const float* u, float* out, float* r, int stage, const double* dt_dev,
                       void* maxkey, const int* active, bool count, cudaStream_t s) {
  DeviceInfo di;
  adv_status st = device_info(&di);
  if (st != ADV_OK) return st;
  W7Params p;
  p.u = u;
  p.out = out;
  p.r = r;
  p.nx = d.nx; p.ny = d.ny; p.nz = d.nz;
  p.tiles_x = (d.nx + W7Tile::BX - 1) / W7Tile::BX;
  p.tiles_y = (d.ny + W7Tile::BY - 1) / W7Tile::BY;
  p.stage = stage;
  p.vec_ok = d.nx % 2 == 0 && (uintptr_t)out % 8 == 0 && (uintptr_t)r % 8 == 0 ? 1 : 0;
  p.rhx = (float)(1.0 / d.dx); p.rhy = (float)(1.0 / d.dy); p.rhz = (float)(1.0 / d.dz);
  p.dt_dev = dt_dev;
  p.maxkey = static_cast<unsigned*>(maxkey);
  p.active = active;
  p.status = device_status_ptr();
  int occ = 0;
  if ((st = kernel_setup(reinterpret_cast<const void*>(&weno7_fused_kernel), W7Tile::NT, W7Tile::SMEM, &occ)) != ADV_OK) return st;
  // one wave of equal shares, at least two planes each (a segment streams eight more)
  p.split = work_split((int64_t)p.tiles_x * p.tiles_y, d.nz, (int64_t)di.sms * occ, d.nz == 1 ? 1 : 2, 4.0);
  weno7_fused_kernel<<<p.split.ctas, W7Tile::NT, W7Tile::SMEM, s>>>(p);
  ADV_CUDA_TRY(cudaGetLastError());
  if (count) count_launches(1);
  return ADV_OK;
}

// The face + residual launches of one FP64 stage (stage 0..4), the update fused into the last axis.
adv_status weno7_stage64(const adv_weno7_desc& d, double* u, const W7Work& w, int stage, const double* dt_dev,
                         void* maxkey, const int* active, bool count, cudaStream_t s) {
  using K = KeyOf<double>::type;
  const W7Geom g{d.nx, d.ny, d.nz, (int64_t)d.nx * d.ny * d.nz};
  const int grid = weno7_grid(d);
  const int nd = weno7_ndim(d);
  double* hp = reinterpret_cast<double*>(w.hp);
  double* hn = reinterpret_cast<double*>(w.hn);
  double* acc = reinterpret_cast<double*>(w.acc);
  double* r = reinterpret_cast<double*>(w.r);
  K* mk = static_cast<K*>(maxkey);
  weno7_face_launch<double, 0>(u, hp, hn, g, active, grid, s);
  weno7_residual_launch<double, 0, true, false>(hp, hn, acc, r, u, g, d.dx, stage, dt_dev, mk, active, grid, s);
  weno7_face_launch<double, 1>(u, hp, hn, g, active, grid, s);
  if (nd == 2) {
    weno7_residual_launch<double, 1, false, true>(hp, hn, acc, r, u, g, d.dy, stage, dt_dev, mk, active, grid, s);
  } else {
    weno7_residual_launch<double, 1, false, false>(hp, hn, acc, r, u, g, d.dy, stage, dt_dev, mk, active, grid, s);
    weno7_face_launch<double, 2>(u, hp, hn, g, active, grid, s);
    weno7_residual_launch<double, 2, false, true>(hp, hn, acc, r, u, g, d.dz, stage, dt_dev, mk, active, grid, s);
  }
  ADV_CUDA_TRY(cudaGetLastError());
  if (count) count_launches(2 * nd);
  return ADV_OK;
}

// One of a step's five stages. FP32 goes u -> a -> b -> a -> b -> u through the work arrays hp, hn.
adv_status weno7_stage(const adv_weno7_desc& d, void* u, const W7Work& w, int stage, const double* dt_dev,
                       void* maxkey, const int* active, bool count, cudaStream_t s) {
  if (d.dtype == ADV_F64) return weno7_stage64(d, static_cast<double*>(u), w, stage, dt_dev, maxkey, active, count, s);
  float* const a = reinterpret_cast<float*>(w.hp);
  float* const b = reinterpret_cast<float*>(w.hn);
  float* const v[6] = {static_cast<float*>(u), a, b, a, b, static_cast<float*>(u)};
  return weno7_fused(d, v[stage], v[stage + 1], reinterpret_cast<float*>(w.r), stage, dt_dev, maxkey, active, count, s);
}

int weno7_stage_launches(const adv_weno7_desc& d) { return d.dtype == ADV_F64 ? 2 * weno7_ndim(d) : 1; }

// The right-hand side alone (the summed residuals, no update), FP64.
adv_status weno7_rhs64(const adv_weno7_desc& d, const double* u, double* L, const W7Work& w, cudaStream_t s) {
  const W7Geom g{d.nx, d.ny, d.nz, (int64_t)d.nx * d.ny * d.nz};
  const int grid = weno7_grid(d);
  const int nd = weno7_ndim(d);
  double* hp = reinterpret_cast<double*>(w.hp);
  double* hn = reinterpret_cast<double*>(w.hn);
  weno7_face_launch<double, 0>(u, hp, hn, g, nullptr, grid, s);
  weno7_residual_launch<double, 0, true, false>(hp, hn, L, nullptr, nullptr, g, d.dx, 0, nullptr, nullptr, nullptr, grid, s);
  weno7_face_launch<double, 1>(u, hp, hn, g, nullptr, grid, s);
  weno7_residual_launch<double, 1, false, false>(hp, hn, L, nullptr, nullptr, g, d.dy, 0, nullptr, nullptr, nullptr, grid, s);
  if (nd == 3) {
    weno7_face_launch<double, 2>(u, hp, hn, g, nullptr, grid, s);
    weno7_residual_launch<double, 2, false, false>(hp, hn, L, nullptr, nullptr, g, d.dz, 0, nullptr, nullptr, nullptr, grid, s);
  }
  ADV_CUDA_TRY(cudaGetLastError());
  count_launches(2 * nd);
  return ADV_OK;
}

}  // namespace
}  // namespace adv

using namespace adv;

extern "C" {

adv_status adv_weno7_workspace_bytes(const adv_weno7_desc* d, size_t* bytes) {
  adv_status st = weno7_validate(d);
  if (st != ADV_OK) return st;
  if (!bytes) return set_error(ADV_ERR_INVALID_ARG, "weno7: null output");
  *bytes = 4 * weno7_array_bytes(*d) + (sizeof(BurgersLoopState) + 255) / 256 * 256;
  return ADV_OK;
}

adv_status adv_weno7_rhs(const adv_weno7_desc* d, const void* u, void* L, void* workspace, void* stream) {
  ADV_NVTX_RANGE("adv_weno7_rhs");
  adv_status st = weno7_validate(d);
  if (st != ADV_OK) return st;
  if (!u || !L || !workspace) return set_error(ADV_ERR_INVALID_ARG, "weno7: null buffer");
  if (u == L) return set_error(ADV_ERR_INVALID_ARG, "weno7: u and L must not alias");
  const W7Work w = weno7_work(*d, workspace);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (d->dtype == ADV_F32)
    return weno7_fused(*d, static_cast<const float*>(u), static_cast<float*>(L), nullptr, 0, nullptr, nullptr, nullptr, true, s);
  return weno7_rhs64(*d, static_cast<const double*>(u), static_cast<double*>(L), w, s);
}

adv_status adv_weno7_run(const adv_weno7_desc* d, void* u, void* workspace, double tEnd, double cfl,
                         int64_t max_steps, double* t_out, int64_t* steps_out, void* stream) {
  ADV_NVTX_RANGE("adv_weno7_run");
  adv_status st = weno7_validate(d);
  if (st != ADV_OK) return st;
  if (!u || !workspace) return set_error(ADV_ERR_INVALID_ARG, "weno7: null buffer");
  if (!(cfl > 0) || !std::isfinite(tEnd) || max_steps < 0) return set_error(ADV_ERR_INVALID_ARG, "weno7: bad cfl/tEnd/max_steps");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if ((st = reject_capture(s, "weno7 run")) != ADV_OK) return st;
  const W7Work w = weno7_work(*d, workspace);
  const size_t n = (size_t)d->nx * d->ny * d->nz;
  const size_t es = d->dtype == ADV_F32 ? 4 : 8;
  // loop state: the Burgers loop's dt rule MAXU (dt = CFL dx / max|u|, trimmed to tEnd)
  adv_burgers_desc bd{};
  bd.nx = d->nx; bd.ny = d->ny; bd.nz = d->nz;
  bd.dx = d->dx; bd.dy = d->dy; bd.dz = d->dz;
  BurgersLoopState h = burgers_loop_state(bd, tEnd, cfl, ADV_DT_MAXU, 0.0, max_steps);
  ADV_CUDA_TRY(cudaMemcpyAsync(w.st, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  ADV_CUDA_TRY(cudaMemsetAsync(w.r, 0, n * es, s));  // the 2N-storage register starts at zero
  void* key0 = d->dtype == ADV_F32 ? (void*)&w.st->maxbits[0] : (void*)&w.st->maxbits64[0];
  if ((st = max_abs_launch(d->dtype, u, (int64_t)n, key0, s)) != ADV_OK) return st;
  // one time step: the step-start kernel (dt, t, loop condition), then five stages; the last one
  // reduces max|u| for the next step into slot 0
  auto body = [&](cudaStream_t cs, unsigned long long cond, int use_cond) -> adv_status {
    adv_status r = burgers_loop_begin_step(w.st, d->dtype, cond, use_cond, cs);
    for (int stg = 0; stg < 5 && r == ADV_OK; ++stg)
      r = weno7_stage(*d, u, w, stg, &w.st->dt, stg == 4 ? key0 : nullptr, &w.st->active, !use_cond, cs);
    return r;
  };
  const int64_t launched_per_step = 1 + 5 * weno7_stage_launches(*d);
  bool graph_ran = false;
  // A run of a few launches at most: they cost less queued one by one, predicated on the loop state, than captured
  // and instantiated as a graph (about 0.1 ms; then 3 us less a step in FP32, 60 us in FP64 3D). us directly / as a
  // graph: FP32 24^3 (six launches a step) 1 step 138 / 229, 4 370 / 420, 8 676 / 679; FP64 (31) 1 step
  // 981 / 1081, 3 2812 / 2775.
  const bool direct = max_steps > 0 && max_steps <= 48 / launched_per_step;
  if (direct && tEnd > 0.0) {
    for (int64_t i = 0; i < max_steps; ++i)
      if ((st = body(s, 0, 0)) != ADV_OK) return st;
  } else if (max_steps > 0 && tEnd > 0.0) {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    cudaStream_t cs;
    ADV_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t e = cudaGraphCreate(&g, 0);
    cudaGraphConditionalHandle h_cond = 0;
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&h_cond, g, 1, cudaGraphCondAssignDefault);
    cudaGraphNode_t node;
    cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
    cp.conditional.handle = h_cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if (e == cudaSuccess) e = cudaGraphAddNode(&node, g, nullptr, nullptr, 0, &cp);
    adv_status bst = ADV_OK;
    if (e == cudaSuccess) {
      e = cudaStreamBeginCaptureToGraph(cs, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        bst = body(cs, (unsigned long long)h_cond, 1);
        cudaGraph_t outg = nullptr;
        e = cudaStreamEndCapture(cs, &outg);
      }
      if (e == cudaSuccess && bst == ADV_OK) e = cudaGraphInstantiate(&ge, g, 0);
    }
    if (g) cudaGraphDestroy(g);
    cudaStreamDestroy(cs);
    if (bst != ADV_OK) {
      if (ge) cudaGraphExecDestroy(ge);
      return bst;
    }
    if (e == cudaSuccess && ge) {
      graph_ran = true;
      e = cudaGraphLaunch(ge, s);
      cudaError_t e2 = cudaStreamSynchronize(s);
      cudaGraphExecDestroy(ge);
      if (e != cudaSuccess) return cuda_error(e, "weno7: graph launch");
      if (e2 != cudaSuccess) return cuda_error(e2, "weno7: run");
    } else {
      cudaGetLastError();  // conditional nodes unavailable: one step at a time from the host
      if (ge) cudaGraphExecDestroy(ge);
      for (int64_t i = 0; i < max_steps; ++i) {
        if ((st = body(s, 0, 0)) != ADV_OK) return st;
        int active = 0;
        ADV_CUDA_TRY(cudaMemcpyAsync(&active, &w.st->active, sizeof(int), cudaMemcpyDeviceToHost, s));
        ADV_CUDA_TRY(cudaStreamSynchronize(s));
        if (!active) break;
      }
    }
  }
  ADV_CUDA_TRY(cudaMemcpyAsync(&h, w.st, sizeof(h), cudaMemcpyDeviceToHost, s));
  ADV_CUDA_TRY(cudaStreamSynchronize(s));
  if (graph_ran) count_launches(launched_per_step * h.step);  // (the host loop counted its own)
  else if (direct && tEnd > 0.0) count_launches(launched_per_step * (h.step - max_steps));  // steps past the end: none
  if (t_out) *t_out = h.t;
  if (steps_out) *steps_out = h.step;
  return read_and_clear_device_status(s);
}

}  // extern "C"
