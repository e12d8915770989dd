// burgers_adjoint.cu -- discrete adjoint of the periodic, local Lax-Friedrichs WENO5 / WENO5-Z
// SSP-RK3 Burgers step, and the checkpointed forward / backward runs (adv_burgers_forward,
// adv_burgers_backward, adv_burgers_adjoint_step in advdiff.h). No reference counterpart.
//
// One adjoint stage computes, for the stage input v and the incoming adjoint lam,
//   t = lam + dt J(v)^T lam,   J = dL/dv,   L_i = -sum_a (F_{i+1/2} - F_{i-1/2}) / h_a
// and combines t into the stage outputs (see below). With psi_f = (lam_{i+1} - lam_i)/h_a the
// weight of face f = i+1/2, (J^T lam)_j = sum_f psi_f dF_f/dv_j. A face's flux is
// side(f+ at i-2..i+2) + side(f- at i+3..i-1); reverse-mode differentiation of each side gives
// five partials, which land on the ten cells of the face's stencil through f+-'(v) =
// v/2 +- |v| (local LF: f+- = v (v/4 +- |v|/2)). A cell therefore collects from the faces
// i-3..i+2 of each axis, which reach cells up to 5 away, so the adjoint needs a halo of 5 for v
// and 3 for lam.
//
// Work layout (one wave of CTAs, balanced (tile, z-plane) segments as in the forward stage): a
// CTA owns 32 x 16 columns, two adjacent in x per thread, and streams the planes z-5 .. z+4 of its
// segment through shared-memory rings (cp.async; v with a 5-cell periodic halo, lam with 3 cells, two
// planes behind). Per streamed plane p each thread advances its columns' f+- windows and differentiates
// the z-faces p-3+1/2, pushing the partials into per-column accumulators for cells p-5..p; cell p-5 is
// then complete in z. For that plane f+- go to shared memory in two layouts (pairs of rows for the
// x-faces, pairs of columns for the y-faces, as in the forward stage: an operand pair is one load), and the
// 37 x 16 x-faces and 32 x 21 y-faces of the tile are differentiated two at a time in one go: an x-face's
// partials go to its warp's cells by shuffles, a y-face's through shared memory (structure of arrays), and the
// 120 pairs past the tile to four warps, one per scheduler, others each plane. Then each cell gathers its ten
// partials per axis, and the stage output is written; three barriers per plane.
// Every face is differentiated once per pass. Bound by issue, as the forward stage: 128^3 FP32 WENO5-Z
// 146.6 -> 84.4 us per stage back to back, FP64 64^3 1326 -> 591, against one face per thread with its two
// sides packed into a pair, the weights' full form (about 125 paired instructions a side against 84) and
// an index division per staged element; with the x- and y-faces in turn, each with its own faces past the
// tile waited for, five barriers: 89.9 and 629.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "adv_device.cuh"
#include "adv_internal.h"
#include "adv_math.cuh"
#include "nvtx_range.h"
#include "weno.cuh"

namespace adv {

namespace {

struct AdjTile {
  static constexpr int BX = 32, BY = 16, NT = 256, PX = BX / 2;
  static constexpr int H = 5, HL = 3;                    // halos of v and lam
  static constexpr int PADX = 6, SW = BX + 2 * PADX;     // v: shared column 0 holds x0 - 6 (pairs aligned)
  static constexpr int SH = BY + 2 * H, PLANE = SW * SH;
  static constexpr int PADL = 4, SWL = BX + 2 * PADL;    // lam: column 0 holds x0 - 4
  static constexpr int SHL = BY + 2 * HL, PLANEL = SWL * SHL;
  static constexpr int NS = 8, NSL = 6;                  // ring slots: v p-5 .. p+2, lam p-5 .. p
  static constexpr int FY = BY + 5, NF = FY * PX;        // y-faces j+1/2, j = -3 .. 17, pairs of columns
  // x-faces i+1/2, i = -3 .. 33, per pair of rows: lane l's is i = l - 3, the last five go through shared
  // memory, each part behind five zeros
  static constexpr int EX = 10, NEX = 10 * EX;
  static constexpr int XS = BX + 2 * H;                  // x-face operands per pair of rows: cells x0-5 .. x0+36
};

template <class T>
struct AdjSmem {
  using TL = AdjTile;
  static constexpr int SLOT = ((TL::PLANE * (int)sizeof(T) + 127) / 128 * 128) / (int)sizeof(T);
  static constexpr int SLOTL = ((TL::PLANEL * (int)sizeof(T) + 127) / 128 * 128) / (int)sizeof(T);
  static constexpr size_t RING = (size_t)(TL::NS * SLOT + TL::NSL * SLOTL) * sizeof(T);
  static constexpr int PART = TL::BY / 2 * TL::XS + TL::SH * TL::PX;            // pairs of one split part
  static constexpr size_t FB = (size_t)(10 * TL::NF + TL::BY / 2 * TL::NEX) * 2 * sizeof(T);  // face partials (SoA)
  static constexpr size_t JX = (size_t)TL::BX * TL::BY * sizeof(T);             // x part of J^T lam per cell
  static constexpr size_t TOTAL = RING + (size_t)2 * PART * 2 * sizeof(T) + FB + JX + TL::PLANE * sizeof(uint32_t);
};

template <class T>
struct AdjArgs {
  const T* v;       // stage input (forward state)
  const T* lam;     // incoming adjoint of the stage output
  const T* acc_in;  // accumulated adjoint of u^n (stages 2, 1)
  T* out;           // outgoing adjoint (lam of the previous stage, or of u^n at stage 1)
  T* acc_out;       // accumulated adjoint of u^n (stages 3, 2); may equal acc_in
  int nx, ny, nz, stage;
  int tiles_x, tiles_y;
  WorkSplit split;  // of the (tile, plane) pairs over the CTAs
  int vec_ok;  // outputs and acc_in: pairs of nodes aligned for one access
  T dt, rdx, rdy, rdz;
  int* status;
};

// Periodic index. Inside the domain (every element of an interior tile) it is the index itself,
// without the integer division of the general case.
__device__ __forceinline__ int wrap(int i, int n) {
  if (i >= 0 && i < n) return i;
  i %= n;
  return i < 0 ? i + n : i;
}

__device__ __forceinline__ float2 vrcp(float2 x) {  // one Newton step on the approximation: 1 ulp
  const float2 r = make_float2(rcp_approx(-x.x), rcp_approx(-x.y));
  const float2 n = vfma(vfma(x, r, vc<float2>(1)), r, r);
  return make_float2(-n.x, -n.y);
}
__device__ __forceinline__ double2 vrcp(double2 x) { return make_double2(1.0 / x.x, 1.0 / x.y); }
// sign(d) t, 0 where d is 0
__device__ __forceinline__ float sgn_mul(float d, float t) { return d == 0.f ? 0.f : __uint_as_float(__float_as_uint(t) ^ (__float_as_uint(d) & 0x80000000u)); }
__device__ __forceinline__ double sgn_mul(double d, double t) { return d > 0.0 ? t : d < 0.0 ? -t : 0.0; }

// Reverse mode of one WENO side (weno_side2 in weno.cuh) for two faces at once: g[k] = psi d side / d f_k
// of f = a..e at i-2 .. i+2. The side is c + C/2 - t1/6 - q/2, q = num / den, num = 2/3 e0 (t1-t0) +
// e2 (t2-t1), den = e0 + 6 e1 + 3 e2; bars of e, b, s, t and of the first differences follow in turn (the
// bars of e and b carry a factor 2).
template <bool Z, class V>
__device__ __forceinline__ void side_rev(V a, V b, V c, V d, V e, V psi, V (&g)[5]) {
  V t[3], s[3], k[3], w[3];  // (the forward run's own indicators: see Candidates in weno.cuh)
  weno_indicators(a, b, c, d, e, t, s, k, w);
  const V t0 = t[0], t1 = t[1], t2 = t[2], s0 = s[0], s1 = s[1], s2 = s[2], k0 = k[0], k1 = k[1], k2 = k[2];
  const V b0 = w[0], b1 = w[1], b2 = w[2];
  const V p12 = vmul(b1, b2), p02 = vmul(b0, b2), p01 = vmul(b0, b1);
  const V da = vsub(t1, t0), db = vsub(t2, t1);
  V e0, e1, e2, d02, tau;
  if (Z) {
    d02 = vsub(b0, b2);
    tau = vabs(d02);
    const V P = vmul(b0, p12);
    e0 = vfma(tau, p12, P);
    e1 = vfma(tau, p02, P);
    e2 = vfma(tau, p01, P);
  } else {
    e0 = vmul(p12, p12);
    e1 = vmul(p02, p02);
    e2 = vmul(p01, p01);
  }
  const V r = vrcp(vfma(vc<V>(3), e2, vfma(vc<V>(6), e1, e0)));
  const V da3 = vmul(vc<V>(2.0 / 3.0), da);
  const V q = vmul(vfma(e2, db, vmul(e0, da3)), r);
  const V gr = vmul(vmul(vc<V>(-1), psi), r);  // 2 x the bar of num
  const V x0 = vmul(gr, vsub(da3, q)), x1 = vmul(vmul(vc<V>(-6), gr), q), x2 = vmul(gr, vfma(vc<V>(-3), q, db));
  V y0, y1, y2;  // 2 x the bars of b0, b1, b2
  if (Z) {
    const V X = vadd(vadd(x0, x1), x2);
    const V z0 = vmul(tau, x0), z1 = vmul(tau, x1), z2 = vmul(tau, x2);
    const V tb = vfma(x2, p01, vfma(x1, p02, vmul(x0, p12)));
    const V st = {sgn_mul(d02.x, tb.x), sgn_mul(d02.y, tb.y)};
    y0 = vadd(vfma(z1, b2, vfma(z2, b1, vmul(X, p12))), st);
    y1 = vfma(z0, b2, vfma(z2, b0, vmul(X, p02)));
    y2 = vsub(vfma(z0, b1, vfma(z1, b0, vmul(X, p01))), st);
  } else {
    const V two = vc<V>(2);
    const V z0 = vmul(vmul(two, p12), x0), z1 = vmul(vmul(two, p02), x1), z2 = vmul(vmul(two, p01), x2);
    y0 = vfma(z1, b2, vmul(z2, b1));
    y1 = vfma(z0, b2, vmul(z2, b0));
    y2 = vfma(z0, b1, vmul(z1, b0));
  }
  const V dab = vmul(vmul(vc<V>(1.0 / 3.0), e0), gr), dbb = vmul(vmul(vc<V>(0.5), e2), gr);  // bars of t1-t0, t2-t1
  const V u0 = vmul(s0, y0), u1 = vmul(s1, y1), u2 = vmul(s2, y2);                            // bars of s0, s1, s2
  const V T0 = vsub(vfma(k0, y0, u0), dab);
  const V T1 = vfma(vc<V>(-1.0 / 6.0), psi, vfma(k1, y1, vsub(dab, dbb)));
  const V T2 = vadd(vfma(k2, y2, u2), dbb);
  const V Bb = vadd(vfma(vc<V>(2), u0, u1), vsub(T0, T1));
  const V Cb = vadd(vfma(vc<V>(-2), u2, u1), vfma(vc<V>(0.5), psi, vsub(T1, T2)));
  g[0] = T0;
  g[1] = vsub(vmul(vc<V>(-1), T0), Bb);
  g[2] = vadd(vsub(Bb, Cb), psi);
  g[3] = vsub(Cb, T2);
  g[4] = T2;
}

template <class T, bool Z>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) burgers_adjoint_kernel(const __grid_constant__ AdjArgs<T> a) {
  using TL = AdjTile;
  using SM = AdjSmem<T>;
  using V = typename Vec2<T>::type;
  constexpr int H = TL::H, SW = TL::SW, SWL = TL::SWL, PX = TL::PX, XS = TL::XS, PART = SM::PART, NF = TL::NF;
  constexpr int YP = TL::BY / 2 * XS;  // y-face operands of a part, after its x-face operands
  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* const ring = reinterpret_cast<T*>(smem_raw);
  T* const ringl = ring + TL::NS * SM::SLOT;
  V* const part = reinterpret_cast<V*>(smem_raw + SM::RING);  // f+; f- follows PART pairs later
  V* const FB = part + 2 * PART;                              // y: [10][NF]: P0..P4, M0..M4
  V* const FE = FB + 10 * NF;                                 // x: [BY/2][10][EX], the last five faces
  T* const jx = reinterpret_cast<T*>(FE + TL::BY / 2 * TL::NEX);  // [BY][BX], a warp's rows its own
  uint32_t* const src = reinterpret_cast<uint32_t*>(jx + TL::BX * TL::BY);  // in-plane offsets of v's staged elements

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cp = tid & (PX - 1), row = tid / PX;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const size_t sxy = (size_t)nx * ny;
  const int own = (row + H) * SW + TL::PADX + 2 * cp;           // this thread's cells in a plane of v ..
  const int ownl = (row + TL::HL) * SWL + TL::PADL + 2 * cp;    // .. and of lam
  // halo splits, two values each: threads [0, 160) the ten halo rows, pairs of columns; [160, 240) the ten
  // halo columns, pairs of rows
  const bool halo = tid < 10 * PX + 10 * (TL::BY / 2);
  int h_src, h_step;
  V* h_dst;
  if (tid < 10 * PX) {
    const int h = tid / PX, r = h < H ? h : h + TL::BY;
    h_src = r * SW + TL::PADX + 2 * cp;
    h_step = 1;
    h_dst = part + YP + r * PX + cp;
  } else {
    const int i = tid - 10 * PX, rp = (i / 10) % (TL::BY / 2), h = i % 10, c = h < H ? h : h + TL::BX;
    h_src = (2 * rp + H) * SW + c + TL::PADX - H;
    h_step = SW;
    h_dst = part + rp * XS + c;
  }
  auto split = [](V u, V& fp, V& fm) { lf_split2(u, vabs(u), fp, fm); };
  for (int e = tid; e < TL::BY / 2 * TL::NEX; e += TL::NT)
    if (e % TL::EX < 5) FE[e] = vc<V>(0);
  int64_t seg_a, seg_b;
  split_range(a.split, blockIdx.x, nz, &seg_a, &seg_b);

  for (int64_t pos = seg_a; pos < seg_b;) {
    const int64_t tile = div_units(pos, nz);
    const int zs = (int)(pos - tile * nz);
    const int ze = (int)min((int64_t)nz, zs + (seg_b - pos));
    pos += ze - zs;
    const int64_t ty = div_units(tile, a.tiles_x);
    const int x0 = (int)(tile - ty * a.tiles_x) * TL::BX, y0 = (int)ty * TL::BY;
    const int Q = (ze - zs) + 10;  // planes zs-5 .. ze+4
    __syncthreads();  // the previous segment's copies have all been issued, its planes read
    for (int e = tid; e < TL::PLANE; e += TL::NT) {
      const int r = e / SW, c = e - r * SW;
      src[e] = (uint32_t)((int64_t)wrap(y0 - H + r, ny) * nx + wrap(x0 - TL::PADX + c, nx));
    }
    __syncthreads();
    // stream entry q: v of plane zs-5+q and lam of the plane two before it
    auto issue = [&](int q) {
      if (q < Q) {
        T* const dv = ring + (q % TL::NS) * SM::SLOT;
        const T* const pv = a.v + (size_t)wrap(zs - 5 + q, nz) * sxy;
#pragma unroll 2
        for (int e = tid; e < TL::PLANE; e += TL::NT)
          cp_async_zfill<sizeof(T)>(dv + e, pv + src[e], ADV_IN_RANGE(pv + src[e] - a.v, sxy * nz, a.status));
        if (q >= 2) {
          T* const dl = ringl + ((q - 2) % TL::NSL) * SM::SLOTL;
          const T* const pl = a.lam + (size_t)wrap(zs - 7 + q, nz) * sxy;
#pragma unroll 2
          for (int e = tid; e < TL::PLANEL; e += TL::NT) {
            const int r = e / SWL, c = e - r * SWL;
            const uint32_t o = src[(r + H - TL::HL) * SW + c + TL::PADX - TL::PADL];
            cp_async_zfill<sizeof(T)>(dl + e, pl + o, ADV_IN_RANGE(pl + o - a.lam, sxy * nz, a.status));
          }
        }
      }
      cp_async_commit();
    };
    issue(0);
    issue(1);

    V fpw[5], fmw[5], fp_new = vc<V>(0);  // f+ at p-5 .. p-1, f- at p-4 .. p, f+ at p
    V accP[6], accM[6];                   // partial sums for cells p-5 .. p
#pragma unroll
    for (int k = 0; k < 6; ++k) { accP[k] = vc<V>(0); accM[k] = vc<V>(0); }
#pragma unroll
    for (int k = 0; k < 5; ++k) { fpw[k] = vc<V>(0); fmw[k] = vc<V>(0); }

#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      cp_async_wait<1>();
      __syncthreads();  // entry q visible; entry q - 6's slots and the face buffers free
      issue(q + 2);
      const T* const vq = ring + (q % TL::NS) * SM::SLOT;
      const T* const vo = ring + ((q + 3) % TL::NS) * SM::SLOT;            // plane q - 5
      const T* const lo = ringl + ((q + 1) % TL::NSL) * SM::SLOTL;         // lam of plane q - 5
      const bool out = q >= 10;
      if (out) {
        V fp, fm;
        split(*reinterpret_cast<const V*>(vo + own), fp, fm);
        V* const yw = part + YP + H * PX + tid;
        yw[0] = fp;
        yw[PART] = fm;
        T* const xw = reinterpret_cast<T*>(part + warp * XS + 2 * cp + H) + (row & 1);
        xw[0] = fp.x; xw[2] = fp.y;
        xw[2 * PART] = fm.x; xw[2 * PART + 2] = fm.y;
        if (halo) {
          split(V{vo[h_src], vo[h_src + h_step]}, fp, fm);
          h_dst[0] = fp;
          h_dst[PART] = fm;
        }
      }
      // ---- z: windows and the face p-3+1/2 (p = plane q)
      {
        V fp, fm;
        split(*reinterpret_cast<const V*>(vq + own), fp, fm);
#pragma unroll
        for (int k = 0; k < 4; ++k) { fpw[k] = fpw[k + 1]; fmw[k] = fmw[k + 1]; }
        fpw[4] = fp_new;
        fp_new = fp;
        fmw[4] = fm;
      }
      if (q >= 5) {
        const V l3 = *reinterpret_cast<const V*>(ringl + ((q + 3) % TL::NSL) * SM::SLOTL + ownl);
        const V l2 = *reinterpret_cast<const V*>(ringl + ((q + 4) % TL::NSL) * SM::SLOTL + ownl);
        const V psi = vmul(V{a.rdz, a.rdz}, vsub(l2, l3));
        V g[5];
        side_rev<Z>(fpw[0], fpw[1], fpw[2], fpw[3], fpw[4], psi, g);
#pragma unroll
        for (int k = 0; k < 5; ++k) accP[k] = vadd(accP[k], g[k]);
        side_rev<Z>(fmw[4], fmw[3], fmw[2], fmw[1], fmw[0], psi, g);
#pragma unroll
        for (int k = 0; k < 5; ++k) accM[k + 1] = vadd(accM[k + 1], g[4 - k]);
      }
      if (out) {
        __syncthreads();  // f+- in place
        // one face pair: operands at p (f+; f- PART later) with stride st
        auto face = [&](const V* p, int st, V psi, V (&g)[5], V (&h)[5]) {
          side_rev<Z>(p[0], p[st], p[2 * st], p[3 * st], p[4 * st], psi, g);
          const V* const m = p + PART;
          side_rev<Z>(m[5 * st], m[4 * st], m[3 * st], m[2 * st], m[st], psi, h);
        };
        V sx, tx;  // x part of J^T lam from the f+ and f- partials: rows 2 warp, 2 warp + 1 of column `lane`
        {
          const T* const l = lo + (2 * warp + TL::HL) * SWL + TL::PADL + lane - 3;  // lam of cell lane - 3, both rows
          const V psi = vmul(V{a.rdx, a.rdx}, vsub(V{l[1], l[SWL + 1]}, V{l[0], l[SWL]}));
          V g[5], h[5];
          face(part + warp * XS + lane, 1, psi, g, h);
          auto from = [&](V w, int d) {  // lane + d's, where the warp has it
            const V v = {__shfl_down_sync(0xffffffffu, w.x, d), __shfl_down_sync(0xffffffffu, w.y, d)};
            return lane + d < 32 ? v : vc<V>(0);
          };
          sx = vadd(from(g[2], 3), vadd(vadd(from(g[4], 1), from(g[3], 2)), vadd(from(g[1], 4), from(g[0], 5))));
          tx = vadd(from(h[3], 3), vadd(vadd(h[0], from(h[1], 1)), vadd(from(h[2], 2), from(h[4], 4))));
        }
        {  // y-faces: f = 16 (j + 3) + column pair
          const T* const l = lo + (row - 3 + TL::HL) * SWL + TL::PADL + 2 * cp;  // lam of row j
          const V psi = vmul(V{a.rdy, a.rdy}, vsub(*reinterpret_cast<const V*>(l + SWL), *reinterpret_cast<const V*>(l)));
          V g[5], h[5];
          face(part + YP + tid, PX, psi, g, h);
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            FB[k * NF + tid] = g[k];
            FB[(5 + k) * NF + tid] = h[4 - k];
          }
        }
        // the faces left over, 5 x 8 in x and 5 x 16 in y: 30 for each of four warps in turn, one per scheduler
        const int e = ((warp - q) & 7) * 30 + lane;
        if (lane < 30 && e < 5 * (TL::BY / 2) + 5 * PX) {
          const bool ex = e < 5 * (TL::BY / 2);
          const int ey = e - 5 * (TL::BY / 2), r = ex ? e / 5 : TL::BY + ey / PX, c = ex ? 32 + e % 5 : ey % PX;
          const T* const l = lo + (ex ? (2 * r + TL::HL) * SWL + TL::PADL + c - 3 : (r - 3 + TL::HL) * SWL + TL::PADL + 2 * c);
          const V psi = vmul(ex ? V{a.rdx, a.rdx} : V{a.rdy, a.rdy},
                             vsub(V{ex ? l[1] : l[SWL], l[SWL + 1]}, V{l[0], ex ? l[SWL] : l[1]}));
          V g[5], h[5];
          face(part + (ex ? r * XS + c : YP + r * PX + c), ex ? 1 : PX, psi, g, h);
          V* const d = ex ? FE + r * TL::NEX + 5 + c - 32 : FB + r * PX + c;
          const int ds = ex ? TL::EX : NF;
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            d[k * ds] = g[k];
            d[(5 + k) * ds] = h[4 - k];
          }
        }
        __syncthreads();
        {
          if (lane >= 27) {
            const V* const P = FE + warp * TL::NEX + 5 + lane - 32;
            const V* const M = P + 5 * TL::EX;
            sx = vadd(sx, vadd(vadd(P[2 * TL::EX + 3], P[4 * TL::EX + 1]), vadd(vadd(P[3 * TL::EX + 2], P[TL::EX + 4]), P[5])));
            tx = vadd(tx, vadd(vadd(M[TL::EX + 3], M[3 * TL::EX + 1]), vadd(M[2 * TL::EX + 2], M[4])));
          }
          const T* const uu = vo + (2 * warp + H) * SW + TL::PADX + lane;
          const V u = {uu[0], uu[SW]};
          const V hu = vmul(vc<V>(0.5), u), au = vabs(u);
          const V j = vfma(vadd(hu, au), sx, vmul(vsub(hu, au), tx));
          jx[(2 * warp) * TL::BX + lane] = j.x;
          jx[(2 * warp + 1) * TL::BX + lane] = j.y;
        }
        __syncwarp();
        const int ko = wrap(zs - 10 + q, nz);
        const V* const P = FB + (row + 3) * PX + cp;
        const V sp = vadd(accP[0], vadd(P[2 * NF], vadd(vadd(P[4 * NF - 2 * PX], P[3 * NF - PX]), vadd(P[NF + PX], P[2 * PX]))));
        const V* const M = P + 5 * NF;
        const V sm = vadd(accM[0], vadd(M[NF], vadd(vadd(M[4 * NF - 3 * PX], M[3 * NF - 2 * PX]), vadd(M[2 * NF - PX], M[PX]))));
        const V u = *reinterpret_cast<const V*>(vo + own), lam = *reinterpret_cast<const V*>(lo + ownl);
        const V hu = vmul(vc<V>(0.5), u), au = vabs(u);
        const V jt = vadd(*reinterpret_cast<const V*>(jx + row * TL::BX + 2 * cp),
                          vfma(vadd(hu, au), sp, vmul(vsub(hu, au), sm)));
        const V t = vfma(V{a.dt, a.dt}, jt, lam);
        const int x = x0 + 2 * cp, y = y0 + row;
        const bool in0 = x < nx && y < ny, in1 = x + 1 < nx && y < ny;
        const size_t o = (size_t)ko * sxy + (size_t)y * nx + x;
        const bool vec = a.vec_ok && in1;
        V acc = vc<V>(0);
        if (a.stage != 3) {
          if (vec) {
            if (ADV_IN_RANGE(o + 1, sxy * nz, a.status)) acc = *reinterpret_cast<const V*>(a.acc_in + o);
          } else {
            if (in0 && ADV_IN_RANGE(o, sxy * nz, a.status)) acc.x = a.acc_in[o];
            if (in1 && ADV_IN_RANGE(o + 1, sxy * nz, a.status)) acc.y = a.acc_in[o + 1];
          }
        }
        auto put = [&](T* dst, V w) {
          if (vec) {
            if (ADV_IN_RANGE(o + 1, sxy * nz, a.status)) *reinterpret_cast<V*>(dst + o) = w;
          } else {
            if (in0 && ADV_IN_RANGE(o, sxy * nz, a.status)) dst[o] = w.x;
            if (in1 && ADV_IN_RANGE(o + 1, sxy * nz, a.status)) dst[o + 1] = w.y;
          }
        };
        if (a.stage == 3) {
          put(a.out, vmul(vc<V>(2.0 / 3.0), t));
          put(a.acc_out, vmul(vc<V>(1.0 / 3.0), lam));
        } else if (a.stage == 2) {
          put(a.out, vmul(vc<V>(0.25), t));
          put(a.acc_out, vfma(vc<V>(0.75), lam, acc));
        } else {
          put(a.out, vadd(acc, t));
        }
      }
      // shift the z accumulators: cell p-5 leaves, p+1 enters
      if (q >= 5) {
#pragma unroll
        for (int k = 0; k < 5; ++k) { accP[k] = accP[k + 1]; accM[k] = accM[k + 1]; }
        accP[5] = vc<V>(0);
        accM[5] = vc<V>(0);
      }
    }
  }
}

}  // namespace

// ------------------------------------------------------------------------------ host
namespace {

adv_status adjoint_validate(const adv_burgers_desc* d) {
  adv_status st = burgers_validate(d);
  if (st != ADV_OK) return st;
  if (d->bc != ADV_BC_PERIODIC || d->lf != ADV_LF_LOCAL || d->kx != 0.0 || d->ky != 0.0 || d->kz != 0.0)
    return set_error(ADV_ERR_UNSUPPORTED,
                     "burgers adjoint: periodic, local Lax-Friedrichs, inviscid schemes only");
  if (d->nz == 1) return set_error(ADV_ERR_UNSUPPORTED, "burgers adjoint: 3D grids only (nz >= 6)");
  return ADV_OK;
}

void* adjoint_kernel(const adv_burgers_desc& d) {
  const bool z = d.weno == ADV_WENO5_Z;
  if (d.dtype == ADV_F32)
    return z ? reinterpret_cast<void*>(&burgers_adjoint_kernel<float, true>)
             : reinterpret_cast<void*>(&burgers_adjoint_kernel<float, false>);
  return z ? reinterpret_cast<void*>(&burgers_adjoint_kernel<double, true>)
           : reinterpret_cast<void*>(&burgers_adjoint_kernel<double, false>);
}

template <class T>
adv_status adjoint_stage_t(const adv_burgers_desc& d, int stage, const void* v, const void* lam, const void* acc_in,
                           void* out, void* acc_out, double dt, cudaStream_t s) {
  DeviceInfo di;
  adv_status st = device_info(&di);
  if (st != ADV_OK) return st;
  AdjArgs<T> a;
  a.v = static_cast<const T*>(v);
  a.lam = static_cast<const T*>(lam);
  a.acc_in = static_cast<const T*>(acc_in);
  a.out = static_cast<T*>(out);
  a.acc_out = static_cast<T*>(acc_out);
  a.nx = d.nx; a.ny = d.ny; a.nz = d.nz;
  a.stage = stage;
  a.tiles_x = (d.nx + AdjTile::BX - 1) / AdjTile::BX;
  a.tiles_y = (d.ny + AdjTile::BY - 1) / AdjTile::BY;
  const uintptr_t pair = 2 * sizeof(T);
  a.vec_ok = d.nx % 2 == 0 && (uintptr_t)out % pair == 0 && (uintptr_t)acc_in % pair == 0 && (uintptr_t)acc_out % pair == 0;
  a.dt = (T)dt;
  a.status = device_status_ptr();
  a.rdx = (T)(1.0 / d.dx); a.rdy = (T)(1.0 / d.dy); a.rdz = (T)(1.0 / d.dz);
  void* k = adjoint_kernel(d);
  const size_t smem = AdjSmem<T>::TOTAL;
  int occ = 0;
  if ((st = kernel_setup(k, 256, smem, &occ)) != ADV_OK) return st;
  // one wave of equal shares (128^3: 92 us per stage, two waves 96, four 112: a segment streams ten extra
  // planes), at least two planes each (48^3: 16.8 us, four 23.1, eight 35.6)
  a.split = work_split((int64_t)a.tiles_x * a.tiles_y, d.nz, (int64_t)di.sms * occ, 2, 6.0);
  void* args[] = {&a};
  ADV_CUDA_TRY(cudaLaunchKernel(k, dim3(a.split.ctas), dim3(256), args, smem, s));
  count_launches(1);
  return ADV_OK;
}

adv_status adjoint_stage(const adv_burgers_desc& d, int stage, const void* v, const void* lam, const void* acc_in,
                         void* out, void* acc_out, double dt, cudaStream_t s) {
  return d.dtype == ADV_F32 ? adjoint_stage_t<float>(d, stage, v, lam, acc_in, out, acc_out, dt, s)
                            : adjoint_stage_t<double>(d, stage, v, lam, acc_in, out, acc_out, dt, s);
}

size_t one_array(const adv_burgers_desc& d) {
  return ((size_t)d.nx * d.ny * d.nz * (d.dtype == ADV_F32 ? 4 : 8) + 255) / 256 * 256;
}

// One adjoint step with scratch lamB, lamC, acc (3 arrays): lam (dJ/du^{n+1}) -> dJ/du^n.
adv_status adjoint_step(const adv_burgers_desc& d, const void* un, const void* u1, const void* u2, double dt, void* lam,
                        char* scratch, cudaStream_t s) {
  const size_t one = one_array(d);
  char* lamB = scratch;
  char* lamC = scratch + one;
  char* acc = scratch + 2 * one;
  adv_status st = adjoint_stage(d, 3, u2, lam, nullptr, lamB, acc, dt, s);
  if (st == ADV_OK) st = adjoint_stage(d, 2, u1, lamB, acc, lamC, acc, dt, s);
  if (st == ADV_OK) st = adjoint_stage(d, 1, un, lamC, acc, lam, nullptr, dt, s);
  return st;
}

// One forward step with a fixed dt from u_n into u1, u2 and u_next (u_next may be u_n).
adv_status forward_step(const adv_burgers_desc& d, const void* un, void* u1, void* u2, void* unext, double dt,
                        cudaStream_t s) {
  BurgersLaunch L;
  BurgersStageArgs a{};
  a.dt_host = dt;
  adv_status st = burgers_prepare(d, un, &L, true);
  a.stage = 1; a.u_in = un; a.u_n = un; a.u_out = u1;
  if (st == ADV_OK) st = burgers_launch(d, L, a, s);
  if (st == ADV_OK) st = burgers_prepare(d, u1, &L, true);
  a.stage = 2; a.u_in = u1; a.u_n = un; a.u_out = u2;
  if (st == ADV_OK) st = burgers_launch(d, L, a, s);
  if (st == ADV_OK) st = burgers_prepare(d, u2, &L, true);
  a.stage = 3; a.u_in = u2; a.u_n = un; a.u_out = unext;
  if (st == ADV_OK) st = burgers_launch(d, L, a, s);
  return st;
}

}  // namespace
}  // namespace adv

using namespace adv;

extern "C" {

adv_status adv_burgers_adjoint_step(const adv_burgers_desc* d, const void* u_n, const void* u1, const void* u2,
                                    double dt, void* lam, void* work, void* stream) {
  ADV_NVTX_RANGE("adv_burgers_adjoint_step");
  adv_status st = adjoint_validate(d);
  if (st != ADV_OK) return st;
  if (!u_n || !u1 || !u2 || !lam || !work) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: null buffer");
  return adjoint_step(*d, u_n, u1, u2, dt, lam, static_cast<char*>(work), static_cast<cudaStream_t>(stream));
}

adv_status adv_burgers_checkpoint_bytes(const adv_burgers_desc* d, int64_t nsteps, int64_t interval,
                                        size_t* ckpt_bytes, size_t* work_bytes) {
  adv_status st = adjoint_validate(d);
  if (st != ADV_OK) return st;
  if (nsteps < 0 || interval < 1) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: bad nsteps/interval");
  const size_t one = one_array(*d);
  const int64_t m = (nsteps + interval - 1) / interval;
  if (ckpt_bytes) *ckpt_bytes = (size_t)std::max<int64_t>(m, 1) * one;
  // backward: u1, u2 of the segment's first step, (u^n, u1, u2) of the others, 3 adjoint arrays;
  // forward: 2 stage arrays
  if (work_bytes) *work_bytes = (size_t)(3 * interval + 2) * one;
  return ADV_OK;
}

adv_status adv_burgers_forward(const adv_burgers_desc* d, void* u, double dt, int64_t nsteps, int64_t interval,
                               void* ckpt, void* work, void* stream) {
  ADV_NVTX_RANGE("adv_burgers_forward");
  adv_status st = adjoint_validate(d);
  if (st != ADV_OK) return st;
  if (!u || !work) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: null buffer");
  if (nsteps < 0 || interval < 1 || !(dt > 0)) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: bad nsteps/interval/dt");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t one = one_array(*d);
  const size_t nb = (size_t)d->nx * d->ny * d->nz * (d->dtype == ADV_F32 ? 4 : 8);
  char* const ub = static_cast<char*>(u);
  char* const states = static_cast<char*>(work);
  // Steps before the last checkpoint interval run in place on u through two stage arrays. The
  // last interval (with checkpoints) writes its stage inputs where adv_burgers_backward would
  // recompute them -- step r of the interval: u1 at 3r, u2 at 3r + 1, its result u^{n+1} at
  // 3r + 2 -- and its last step writes u; with interval >= nsteps the whole run is kept and the
  // backward run recomputes nothing.
  const int64_t m = (nsteps + interval - 1) / interval;
  const int64_t n_last = ckpt && nsteps > 0 ? (m - 1) * interval : nsteps;
  for (int64_t n = 0; n < nsteps; ++n) {
    if (ckpt && n % interval == 0)
      ADV_CUDA_TRY(cudaMemcpyAsync(static_cast<char*>(ckpt) + (n / interval) * one, u, nb, cudaMemcpyDeviceToDevice, s));
    if (n < n_last) {
      st = forward_step(*d, ub, states, states + one, ub, dt, s);
    } else {
      const int64_t r = n - n_last;
      const char* un = r == 0 ? ub : states + (3 * r - 1) * one;
      char* next = n + 1 < nsteps ? states + (3 * r + 2) * one : ub;
      st = forward_step(*d, un, states + 3 * r * one, states + (3 * r + 1) * one, next, dt, s);
    }
    if (st != ADV_OK) return st;
  }
  return ADV_OK;
}

adv_status adv_burgers_backward(const adv_burgers_desc* d, double dt, int64_t nsteps, int64_t interval,
                                const void* ckpt, void* lam, void* work, int flags, void* stream) {
  ADV_NVTX_RANGE("adv_burgers_backward");
  adv_status st = adjoint_validate(d);
  if (st != ADV_OK) return st;
  if (!ckpt || !lam || !work) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: null buffer");
  if (nsteps < 0 || interval < 1 || !(dt > 0)) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: bad nsteps/interval/dt");
  if (flags & ~ADV_BURGERS_LAST_INTERVAL_IN_WORK) return set_error(ADV_ERR_INVALID_ARG, "burgers adjoint: unknown flags");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t one = one_array(*d);
  char* states = static_cast<char*>(work);             // 3 interval - 1 arrays
  char* scratch = states + (size_t)(3 * interval - 1) * one;  // 3 arrays
  const int64_t m = (nsteps + interval - 1) / interval;
  for (int64_t seg = m - 1; seg >= 0; --seg) {
    const int64_t n0 = seg * interval, n1 = std::min(nsteps, n0 + interval);
    const char* base = static_cast<const char*>(ckpt) + seg * one;
    // step n (relative r = n - n0) keeps u^n at index 3r - 1 (the checkpoint for r = 0), u1 at
    // 3r, u2 at 3r + 1
    auto un = [&](int64_t r) -> const char* { return r == 0 ? base : states + (3 * r - 1) * one; };
    auto u1 = [&](int64_t r) { return states + (3 * r) * one; };
    auto u2 = [&](int64_t r) { return states + (3 * r + 1) * one; };
    const bool kept = seg == m - 1 && (flags & ADV_BURGERS_LAST_INTERVAL_IN_WORK);
    for (int64_t r = 0; !kept && r < n1 - n0; ++r) {
      char* next = r + 1 < n1 - n0 ? states + (3 * (r + 1) - 1) * one : nullptr;
      if (next) {
        if ((st = forward_step(*d, un(r), u1(r), u2(r), next, dt, s)) != ADV_OK) return st;
      } else {
        // the last step of the segment needs only its stage inputs: stages 1 and 2
        BurgersLaunch L;
        BurgersStageArgs a{};
        a.dt_host = dt;
        if ((st = burgers_prepare(*d, un(r), &L, true)) != ADV_OK) return st;
        a.stage = 1; a.u_in = un(r); a.u_n = un(r); a.u_out = u1(r);
        if ((st = burgers_launch(*d, L, a, s)) != ADV_OK) return st;
        if ((st = burgers_prepare(*d, u1(r), &L, true)) != ADV_OK) return st;
        a.stage = 2; a.u_in = u1(r); a.u_n = un(r); a.u_out = u2(r);
        if ((st = burgers_launch(*d, L, a, s)) != ADV_OK) return st;
      }
    }
    for (int64_t r = n1 - n0 - 1; r >= 0; --r)
      if ((st = adjoint_step(*d, un(r), u1(r), u2(r), dt, lam, scratch, s)) != ADV_OK) return st;
  }
  return ADV_OK;
}

}  // extern "C"
