// burgers_kernels.cuh -- fused WENO5 / WENO5-Z Burgers SSP-RK3 stage for sm_103a.
//
// One launch per stage replaces the reference's five (Compute_dF, Compute_dG, Compute_dH,
// Compute_Laplace_Async, Compute_RK: SingleGPU/Burgers3d_WENO5/kernels.cu:197-530, driven by
// main.cpp:143-149) and its per-step device copy.
//
// Work layout: a CTA owns a 32 x 16 tile of x-y columns (256 threads, two columns adjacent in x per
// thread) and marches through a chunk of z planes. Each plane of the tile plus a 3-cell halo is
// staged in an 8-slot shared-memory ring by TMA (x start rounded down to a 16-byte boundary; periodic
// tiles at a domain edge patch their wrapped halo after the copy lands). Per streamed plane q:
//   * f+- of the output plane (q - 3) go to shared memory once (Lax-Friedrichs split), in two
//     layouts: rows for the y-faces, pairs of rows interleaved for the x-faces, so that every
//     operand pair of the two-value arithmetic is one load and needs no packing;
//   * each thread's two z-faces come from its columns' line state (WenoLine: what neighbouring faces
//     share is computed once per cell), advanced by plane q;
//   * the 33x16 x-faces and 32x17 y-faces are reconstructed by all threads, two at a time;
//   * L = -(dF/dx + dG/dy + dH/dz) (+ viscous O4 term), the SSP-RK3 combine, the store and a
//     warp-shuffle max|u_out| reduction (one atomicMax per CTA) for the next stage's
//     Lax-Friedrichs constant and time step all happen in the same pass.
// Two barriers per plane: the one after the split also releases the ring slot of the output plane
// (nothing reads it later), the one after the faces hands them to their cells.
// Every node is read from HBM once per stage and written once. Bound by issue: at 256^3 FP32 WENO5-Z
// a plane takes 561 issue slots per pair of cells, half of them paired FP32 instructions (832 and 290
// before neighbouring faces shared their differences, pairs were loaded instead of packed, and the six
// quotients per cell went through the paired correction of vnquot): 334 -> 215 us per stage back to
// back, 50.3 -> 78.0 Gcell-stage/s; the FMA pipe is 57% busy, 58% of the issue slots are used. A 2D problem (nz == 1) streams its one
// plane alone: no z faces, no z halo (1000 x 900 FP32: 61 -> 14.5 us per stage against streaming the
// plane seven times). FP64 is bound by its pipe (78% busy at 128 x 112 x 101): warps whose faces no updated
// node reads reconstruct none, and the faces left over are one value per lane of two warps
// (121 x 101 x 97: 2378 -> 2086 us per stage, 64 x 53 x 60: 519 -> 409; 1714 and 386 with weno_ref_quot).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "adv_device.cuh"
#include "adv_math.cuh"
#include "weno.cuh"

namespace adv {

template <class T>
struct BurgersParams {
  const T* uin;
  const T* un;
  T* out;
  int nx, ny, nz;
  int stage;
  int periodic;  // 1: periodic wrap; 0: the reference's frozen outer 3 layers
  int bug_b2;
  int tiles_x, tiles_y;
  WorkSplit split;  // of the (tile, plane) pairs over the CTAs of a single-grid launch
  int tma;
  int un_is_uin;
  int vec_ok;  // u_n and u_out: pairs of nodes aligned for one access
  int lf_global;
  T dx, dy, dz;
  T rdx, rdy, rdz;  // 1/h, divided in FP64
  T kx, ky, kz;
  double dt_host, alpha_host;
  const double* dt_dev;
  const double* alpha_dev;
  const void* alpha_key;
  void* maxabs_key;
  const int* active;
  int* status;
};

struct BurgersTile {
  static constexpr int BX = 32, BY = 16, NT = 256;
  static constexpr int R = 3;
  static constexpr int PADX = 4;  // shared column 0 holds x0 - 4 (16-byte aligned for FP32 and FP64)
  static constexpr int SW = BX + 2 * PADX;  // 40
  static constexpr int SH = BY + 2 * R;     // 22
  static constexpr int PLANE = SW * SH;     // 880
  // ring: 8 slots (a power of two: slot and phase parity of a stream entry are bits of its number);
  // once plane q-3 (the output plane) has been split, plane q+4 is requested, so three planes stay in
  // flight ahead of the one awaited
  static constexpr int NS = 8;
  static constexpr int P = 3;
  static constexpr int PX = BX / 2;      // column pairs per row
  static constexpr int XS = BX + 8;      // x-face operands: cells x0-3 .. x0+34 of a row pair (38 used)
  static constexpr int XF = BX + 2;      // x-faces per row (33 used)
};

template <class T>
struct BurgersSmem {
  static constexpr int SLOT_ELEMS = ((BurgersTile::PLANE * (int)sizeof(T) + 127) / 128 * 128) / (int)sizeof(T);
  static constexpr size_t RING = (size_t)BurgersTile::NS * SLOT_ELEMS * sizeof(T);
  // one split part, in pairs: by row pairs for the x-faces [BY/2][XS], by rows for the y-faces [SH][PX]
  static constexpr int PART = (BurgersTile::BY / 2) * BurgersTile::XS + BurgersTile::SH * BurgersTile::PX;
  static constexpr int NFY = (BurgersTile::BY + 1) * BurgersTile::PX;  // pairs of y-faces
  static constexpr size_t TOTAL = RING + (2 * PART + NFY) * 2 * sizeof(T) + (size_t)BurgersTile::BY * BurgersTile::XF * sizeof(T);
};

__device__ __forceinline__ int wrapi(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// Face reconstruction and Lax-Friedrichs split of two values at once (V = float2 or double2): FP32,
// and FP64 with ADV_DIV_FAST, take the common-denominator form (one division per side, of kind D);
// FP64 otherwise the reference's literal operand order. Line: the z-face of a column pair, advanced
// one plane at a time; u_a, u_b: the states on both sides of the face (planes q-3 and q-2).
template <class T, bool Z, class D>
struct Face {
  using V = typename Vec2<T>::type;
  __device__ __forceinline__ static V f(V p0, V p1, V p2, V p3, V p4, V m0, V m1, V m2, V m3, V m4) {
    return weno_face2<Z, D>(p0, p1, p2, p3, p4, m0, m1, m2, m3, m4);
  }
  __device__ __forceinline__ static void split(V u, V a, V& fp, V& fm) { lf_split2(u, a, fp, fm); }
  struct Line {
    WenoLine<V> p, m;
    V fp_new;  // f+ of the newest plane, one plane behind f- (its stencil ends one cell lower)
    __device__ __forceinline__ void clear() { p.clear(); m.clear(); fp_new = vc<V>(0); }
    __device__ __forceinline__ V push(V fp, V fm, V u_a, V u_b, bool want) {
      V tp, tm;
      const V qp = p.template push<Z, D, true>(fp_new, want, tp);
      const V qm = m.template push<Z, D, false>(fm, want, tm);
      fp_new = fp;
      // both sides' linear parts: (f_i + f_{i+1})/2 with f+ + f- = u^2/2
      const V lin = vmul(vc<V>(0.25), vfma(u_a, u_a, vmul(u_b, u_b)));
      return vfma(vc<V>(0.5), vsub(qp, qm), vfma(vc<V>(-1.0 / 6.0), vadd(tp, tm), lin));
    }
  };
};
template <bool Z>
struct Face<double, Z, double> {
  using V = double2;
  __device__ __forceinline__ static V f(V p0, V p1, V p2, V p3, V p4, V m0, V m1, V m2, V m3, V m4) {
    return make_double2(weno_face_ref<Z, double>(p0.x, p1.x, p2.x, p3.x, p4.x, m0.x, m1.x, m2.x, m3.x, m4.x),
                        weno_face_ref<Z, double>(p0.y, p1.y, p2.y, p3.y, p4.y, m0.y, m1.y, m2.y, m3.y, m4.y));
  }
  __device__ __forceinline__ static void split(V u, V a, V& fp, V& fm) {
    lf_split<double>(u.x, a.x, fp.x, fm.x);
    lf_split<double>(u.y, a.y, fp.y, fm.y);
  }
  struct Line {
    WenoRefLine<Z, true> p;
    WenoRefLine<Z, false> m;
    V fp_new;  // f+ of the newest plane, one plane behind f-
    __device__ __forceinline__ void clear() { p.clear(); m.clear(); fp_new = vc<V>(0); }
    __device__ __forceinline__ V push(V fp, V fm, V, V, bool want) {
      const V qp = p.push(fp_new, want), qm = m.push(fm, want);
      fp_new = fp;
      return vadd(qp, qm);
    }
  };
};

// The candidates' weighted mean (weno.cuh): a z-face from the last four cells of each part and the newest.
template <class D>
struct Face<float, true, Candidates<D>> {
  using V = float2;
  __device__ __forceinline__ static V f(V p0, V p1, V p2, V p3, V p4, V m0, V m1, V m2, V m3, V m4) {
    return weno_face_mean<D>(p0, p1, p2, p3, p4, m0, m1, m2, m3, m4);
  }
  __device__ __forceinline__ static void split(V u, V a, V& fp, V& fm) { lf_split2(u, a, fp, fm); }
  struct Line {
    V p[5], m[4];  // f+ one plane behind f-
    __device__ __forceinline__ void clear() {
#pragma unroll
      for (int i = 0; i < 5; ++i) p[i] = vc<V>(0);
#pragma unroll
      for (int i = 0; i < 4; ++i) m[i] = vc<V>(0);
    }
    __device__ __forceinline__ V push(V fp, V fm, V, V, bool want) {
      V r = vc<V>(0);
      if (want) r = f(p[0], p[1], p[2], p[3], p[4], m[0], m[1], m[2], m[3], fm);
      p[0] = p[1]; p[1] = p[2]; p[2] = p[3]; p[3] = p[4]; p[4] = fp;
      m[0] = m[1]; m[1] = m[2]; m[2] = m[3]; m[3] = fm;
      return r;
    }
  };
};

// Stream entries a CTA has waited for so far (entry n lives in slot n % NS and is that slot's phase
// n / NS); kPipeAborted after a wait that timed out.
constexpr unsigned kPipeAborted = 0xffffffffu;

// Shared-memory objects of the Burgers pipeline (one set per CTA, whichever kernel runs it).
__device__ __forceinline__ uint64_t* burgers_bars() {
  __shared__ uint64_t bars[BurgersTile::NS];
  return bars;
}
__device__ __forceinline__ int* burgers_abort_flag() {
  __shared__ int flag;
  return &flag;
}
// TMA: a periodic edge tile's patch list, the staged plane's elements that lie outside the domain
// (slot index) and the in-plane offset of the wrapped node each takes. cp.async loads: the in-plane
// offset of every element of the staged plane (wrapped when periodic), -1 outside the domain.
struct BurgersPatch {
  int n;
  uint16_t slot[BurgersTile::PLANE];
  int64_t src[BurgersTile::PLANE];
};
static_assert(BurgersTile::PLANE <= 65535, "patch slots are 16-bit");
__device__ __forceinline__ BurgersPatch* burgers_patch() {
  __shared__ BurgersPatch patch;
  return &patch;
}

// The stage's Lax-Friedrichs constant and dt, rounded to the state's type by one thread per CTA: in every
// thread and segment the conversions queued for the FP64 pipe, two lanes per SM and cycle
// (us per stage, before -> after: FP32 2D 1000 x 900 14.17 -> 13.79, 64^3 12.13 -> 11.80, 96^3 21.2 -> 20.7, 256^3
// 215.2 -> 213.9).
template <class T>
struct BurgersScalars {
  T alpha, dt;
};
template <class T>
__device__ __forceinline__ BurgersScalars<T>* burgers_scalars() {
  __shared__ BurgersScalars<T> s;
  return &s;
}
// (visible to the CTA after its next barrier)
template <class T>
__device__ __forceinline__ void burgers_load_scalars(const BurgersParams<T>& p) {
  using K = typename KeyOf<T>::type;
  if (threadIdx.x != 0) return;
  T alpha;
  if (p.alpha_dev) alpha = (T)*p.alpha_dev;
  else if (p.alpha_key) alpha = (T)key_to_value(*static_cast<const K*>(p.alpha_key));
  else alpha = (T)p.alpha_host;
  *burgers_scalars<T>() = BurgersScalars<T>{alpha, (T)(p.dt_dev ? *p.dt_dev : p.dt_host)};
}

// The CTA's running max|u_out| key (8 bytes hold either state type's).
__device__ __forceinline__ unsigned long long* burgers_block_max() {
  __shared__ unsigned long long m;
  return &m;
}
// Merges every thread's key into *key (nullable) with one global atomic per CTA: one per warp and segment
// to the same address took longer than a small grid's stage (2D 1000 x 900: 13,000 of them per launch).
template <class K>
__device__ __forceinline__ void burgers_flush_max(K kmax, void* key) {
  if (!key) return;
  K* const m = reinterpret_cast<K*>(burgers_block_max());
  __syncthreads();
  if (threadIdx.x == 0) *m = 0;
  __syncthreads();
  kmax = warp_max(kmax);
  if ((threadIdx.x & 31) == 0 && kmax) atomicMax(m, kmax);
  __syncthreads();
  if (threadIdx.x == 0 && *m) atomicMax(static_cast<K*>(key), *m);
}

template <class T>
__device__ __forceinline__ void burgers_cta_init(const CUtensorMap* tmap, bool tma) {
  if (threadIdx.x == 0) {
    if (tma) {
      uint64_t* bars = burgers_bars();
      for (int s = 0; s < BurgersTile::NS; ++s) mbar_init(&bars[s], 1);
      mbar_fence_init();
      if (tmap) tma_prefetch_desc(tmap);
    }
    *burgers_abort_flag() = 0;
  }
  __syncthreads();
}

// How a kernel loads its planes and which problems it takes: 3D with TMA loads, 3D with element copies
// (cp.async: rows or bases TMA cannot describe), or any (2D problems, nz == 1, with either load).
// The common modes carry none of the others' tests in their plane loop.
enum BurgersMode { BURGERS_3D_TMA = 0, BURGERS_3D_COPY = 1, BURGERS_ANY = 2 };

// |u| or the global constant as one bit operation: (u & m) | o.
__device__ __forceinline__ float bits_and_or(float u, unsigned m, float o) {
  return __uint_as_float((__float_as_uint(u) & m) | __float_as_uint(o));
}
__device__ __forceinline__ double bits_and_or(double u, unsigned m, double o) {
  return __hiloint2double((__double2hiint(u) & (int)m) | __double2hiint(o),
                          (__double2loint(u) & ((int)m >> 30 & 1 ? -1 : 0)) | __double2loint(o));
}

// Stage combination of a pair, the operations of stage_combine in its order (FP32: paired).
__device__ __forceinline__ double2 combine2(int stage, double2 un, double2 u, double dt, double2 L) {
  return make_double2(stage_combine<double>(stage, un.x, u.x, dt, L.x), stage_combine<double>(stage, un.y, u.y, dt, L.y));
}
__device__ __forceinline__ float2 combine2(int stage, float2 un, float2 u, float dt, float2 L) {
  const float2 dL = vmul_alone(make_float2(dt, dt), L);
  if (stage == 2) return vadd(vmul_alone(vc<float2>(0.75), un), vmul(vc<float2>(0.25), vadd(u, dL)));  // (u/4 is exact)
  if (stage == 3) return div3(vfma(vc<float2>(2), vadd(u, dL), un));
  return vadd(un, dL);
}

// One segment: output planes [zs, ze) of the column tile at (x0, y0), streamed through the
// ring, whose first entry is number n0. Raises kmax to this thread's max|u_out| key. Returns the next
// segment's first entry number, kPipeAborted if a wait timed out (the CTA must then return).
template <class T, bool Z, class D, bool VISC, int MODE>
__device__ __forceinline__ unsigned burgers_segment(const CUtensorMap* tmap, const BurgersParams<T>& p, int x0, int y0,
                                                    int zs, int ze, unsigned n0, typename KeyOf<T>::type& kmax) {
  using TL = BurgersTile;
  using SM = BurgersSmem<T>;
  using K = typename KeyOf<T>::type;
  using V = typename Vec2<T>::type;
  using F = Face<T, Z, D>;
  // FP64 (unless ADV_DIV_FAST): reference operand order, correctly rounded
  constexpr bool EXACT = sizeof(T) == 8 && !std::is_same<D, FastDiv>::value;
  constexpr int PX = TL::PX, R = TL::R, SW = TL::SW, XS = TL::XS, PART = SM::PART;
  constexpr int YP = (TL::BY / 2) * XS;  // the y-face operands of a part, after its x-face operands

  extern __shared__ __align__(128) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  V* const part = reinterpret_cast<V*>(smem_raw + SM::RING);  // f+; f- follows PART pairs later
  V* const fyS = part + 2 * PART;                             // y-faces [BY+1][PX]
  T* const fxS = reinterpret_cast<T*>(fyS + SM::NFY);         // x-faces [BY][XF]
  uint64_t* bars = burgers_bars();
  int* abort_flag = burgers_abort_flag();

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nx = p.nx, ny = p.ny, nz = p.nz;
  const size_t sxy = (size_t)nx * ny;
  const bool per = p.periodic != 0;
  const bool tma = MODE == BURGERS_3D_TMA || (MODE == BURGERS_ANY && p.tma);
  // 2D (nz == 1): the one plane is streamed alone; its z faces would be equal and their difference
  // exactly zero, and no z layer is frozen. 3D: the output plane runs `lag` planes behind.
  const bool twod = MODE == BURGERS_ANY && nz == 1;
  const int lag = twod ? 0 : R;

  // Lax-Friedrichs constant and dt for this stage.
  const T alpha = burgers_scalars<T>()->alpha, dt = burgers_scalars<T>()->dt;
  const unsigned speed_m = p.lf_global ? 0u : 0x7fffffffu;
  const T speed_o = p.lf_global ? alpha : T(0);
  auto split = [&](V u, V& fp, V& fm) {
    F::split(u, V{bits_and_or(u.x, speed_m, speed_o), bits_and_or(u.y, speed_m, speed_o)}, fp, fm);
  };

  // This thread's columns: 2 cp, 2 cp + 1 of row `row` (a warp holds two rows, one row pair).
  const int cp = tid & (PX - 1), row = tid / PX;
  const int own = (row + R) * SW + TL::PADX + 2 * cp;  // its place in a staged plane
  const int x = x0 + 2 * cp, y = y0 + row;
  const bool in0 = x < nx && y < ny, in1 = x + 1 < nx && y < ny;  // partial tiles extend past the domain
  const int FR = per ? 0 : 3;
  const bool yok = per || (y >= FR && y < ny - FR);
  const bool upd0 = in0 && yok && (per || (x >= FR && x < nx - FR));
  const bool upd1 = in1 && yok && (per || (x + 1 >= FR && x + 1 < nx - FR));
  const bool vec = p.vec_ok && in1;
  // FP64: what this warp reconstructs. Faces no updated node reads (frozen rows, rows and tiles past the
  // domain) are left out; a warp's x- and z-faces serve its own two rows, its y-faces the row below them as
  // well. (FP32, bound by issue and latency, lost 2-4% to the extra predicates.)
  const bool all = sizeof(T) == 4;
  const int yw0 = y0 + 2 * warp;
  const bool cols = all || per || (x0 + TL::BX > FR && x0 < nx - FR);
  const bool need = all || (cols && yw0 + 1 >= FR && yw0 < ny - FR);
  const bool need_y = all || (cols && yw0 + 1 >= FR && yw0 - 1 < ny - FR);
  // Operand places of this thread's share of the splits and faces.
  T* const xw = reinterpret_cast<T*>(part + warp * XS + 2 * cp + R) + (row & 1);  // its cells, x layout
  V* const yw = part + YP + R * PX + tid;                                        // its cells, y layout
  const V* const xr = part + warp * XS + lane;  // x-face `lane` (between cells lane-1 and lane) of its row pair
  const V* const yr = part + YP + tid;          // the y-faces below its cells
  // halo splits, two values each: threads [0, 96) the six halo rows, pairs of columns; [96, 144) the
  // six halo columns, pairs of rows
  const bool halo = tid < 6 * PX + 6 * (TL::BY / 2);
  int h_src, h_step;
  V* h_dst;
  if (tid < 6 * PX) {
    const int h = tid / PX, r = h < R ? h : h + TL::BY;
    h_src = r * SW + TL::PADX + 2 * cp;
    h_step = 1;
    h_dst = part + YP + r * PX + cp;
  } else {
    const int i = tid - 6 * PX, rp = (i / 6) % (TL::BY / 2), h = i % 6, c = h < R ? h : h + TL::BX;
    h_src = (2 * rp + R) * SW + c + TL::PADX - R;
    h_step = SW;
    h_dst = part + rp * XS + c;
  }
  // the last x-face of each row pair (lanes [0, 8)) and the top row of y-faces (lanes [8, 24)): one
  // warp, another each plane
  const bool l_x = lane < TL::BY / 2;
  const int l_st = l_x ? 1 : PX;
  const int l_src = l_x ? lane * XS + TL::BX : YP + TL::BY * PX + (lane - TL::BY / 2);

  const int Q = (ze - zs) + 2 * lag;
  const int p0 = zs - lag;
  const bool edge = per && (x0 - TL::PADX < 0 || x0 + TL::BX + TL::PADX > nx || y0 - R < 0 || y0 + TL::BY + R > ny);
  // Periodic plane index: within one period of the domain (the usual case) a conditional add or
  // subtract, not the integer division of wrapi (5% of the stage at 256^3).
  auto plane_z = [&](int q) {
    int z = p0 + q;
    if (per) {
      if (z < 0) z += nz;
      else if (z >= nz) z -= nz;
      if ((unsigned)z >= (unsigned)nz) z = wrapi(z, nz);
    }
    return z;
  };
  // Periodic edge tile: the TMA box zero-fills what lies outside the domain. The three layers there that
  // a face of the domain's cells reads are listed once per segment (CTA-uniform branch), and each plane
  // copies their wrapped neighbours over the zeros, asynchronously: nothing reads them before the barrier
  // one plane later. Element copies (cp.async) take every element's place in its plane from the same
  // list, so a plane's staging has no index arithmetic.
  BurgersPatch* patch = burgers_patch();
  if (!tma) {
    for (int e = tid; e < TL::PLANE; e += TL::NT) {
      const int r = e / SW, c = e - r * SW;
      int gx = x0 - TL::PADX + c, gy = y0 - R + r;
      if (per) { gx = wrapi(gx, nx); gy = wrapi(gy, ny); }
      const bool ok = gx >= 0 && gx < nx && gy >= 0 && gy < ny;
      patch->src[e] = ok ? (int64_t)gy * nx + gx : -1;
    }
    // each thread reads back only what it wrote: no barrier
  } else if (edge) {
    if (tid == 0) patch->n = 0;  // (the previous segment's list was last read before its last barrier)
    __syncthreads();
    for (int e = tid; e < TL::PLANE; e += TL::NT) {
      const int r = e / SW, c = e - r * SW;
      const int gx = x0 - TL::PADX + c, gy = y0 - R + r;
      if ((gx < 0 || gx >= nx || gy < 0 || gy >= ny) && gx >= -R && gx < nx + R && gy >= -R && gy < ny + R) {
        const int k = atomicAdd(&patch->n, 1);
        patch->slot[k] = (uint16_t)e;
        patch->src[k] = (int64_t)wrapi(gy, ny) * nx + wrapi(gx, nx);
      }
    }
    __syncthreads();
  }
  auto slot = [&](int q) { return ring + ((n0 + (unsigned)q) % TL::NS) * SM::SLOT_ELEMS; };  // of stream entry q
  auto issue = [&](int q) {
    if (tma) {
      if (tid == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        uint64_t* bar = &bars[(n0 + (unsigned)q) % TL::NS];
        mbar_arrive_expect_tx(bar, TL::PLANE * (unsigned)sizeof(T));
        tma_load_3d(slot(q), tmap, x0 - TL::PADX, y0 - R, plane_z(q), bar);
      }
    } else {
      T* dst = slot(q);
      const int z = plane_z(q);
      const bool zok = z >= 0 && z < nz;
      const T* plane = p.uin + (zok ? (size_t)z * sxy : 0);
      for (int e = tid; e < TL::PLANE; e += TL::NT) {
        const int64_t o = patch->src[e];
        const bool ok = zok && o >= 0;
        const T* src = ok ? plane + o : p.uin;
        cp_async_zfill<sizeof(T)>(dst + e, src, ok && ADV_IN_RANGE(src - p.uin, sxy * nz, p.status));
      }
      cp_async_commit();
    }
  };
  auto wait = [&](int q) {
    const unsigned n = n0 + (unsigned)q;
    return mbar_wait_bounded(&bars[n % TL::NS], (n / TL::NS) & 1u, p.status);
  };

  for (int q = 0; q <= TL::P && q < Q; ++q) issue(q);
  if (!tma)
    for (int q = Q; q <= TL::P; ++q) cp_async_commit();  // one group per plane index

  typename F::Line line;
  line.clear();
  V fz_prev = vc<V>(0), uc = vc<V>(0);  // z-face below the output plane; u of plane q-3
  V ub = vc<V>(0), ua = vc<V>(0);       // viscous variant: u of planes q-4, q-5
  size_t gi = (size_t)zs * sxy + (size_t)y * nx + x;  // this thread's nodes of the output plane
#pragma unroll 1
  for (int q = 0; q < Q; ++q) {
    T* plq = slot(q);
    const T* plc = slot(q - lag);  // the output plane
    if (tma) {
      if (!wait(q)) *abort_flag = 1;  // every lane waits (converged)
      if (edge) {
        // the listed elements of plane q take their wrapped neighbours; they are read only from the
        // second plane after this one on (2D: after this barrier)
        const size_t zo = (size_t)plane_z(q) * sxy;
        for (int k = tid; k < patch->n; k += TL::NT) {
          const size_t gs = zo + (size_t)patch->src[k];
          const int e = patch->slot[k];
          if (ADV_IN_RANGE(gs, sxy * nz, p.status) && ADV_IN_RANGE(e, TL::PLANE, p.status))
            cp_async_zfill<sizeof(T)>(plq + e, p.uin + gs, true);
        }
        cp_async_commit();
        if (twod) {
          cp_async_wait<0>();
          __syncthreads();
        }
      }
    } else {
      cp_async_wait<TL::P>();
      __syncthreads();  // the other threads' copies of plane q
    }
    const int k = zs + q - 2 * lag;  // output plane (q >= 2 lag)
    const bool out = q >= 2 * lag;
    const bool any_upd = out && (per || twod || (k >= FR && k < nz - FR));  // CTA-uniform
    V visc = vc<V>(0);
    if (twod) uc = *reinterpret_cast<const V*>(plc + own);
    if (any_upd) {
      // f+- of the output plane into shared memory: this thread's cells in both layouts, and the halos
      V fp, fm;
      split(uc, fp, fm);
      yw[0] = fp;
      yw[PART] = fm;
      xw[0] = fp.x; xw[2] = fp.y;
      xw[2 * PART] = fm.x; xw[2 * PART + 2] = fm.y;
      if (halo) {
        split(V{plc[h_src], plc[h_src + h_step]}, fp, fm);
        h_dst[0] = fp;
        h_dst[PART] = fm;
      }
      if (VISC) {
        const T* const r0 = plc + own;
        const V xl = *reinterpret_cast<const V*>(r0 - 2), xh = *reinterpret_cast<const V*>(r0 + 2);
        const V ym2 = *reinterpret_cast<const V*>(r0 - 2 * SW), ym1 = *reinterpret_cast<const V*>(r0 - SW);
        const V yp1 = *reinterpret_cast<const V*>(r0 + SW), yp2 = *reinterpret_cast<const V*>(r0 + 2 * SW);
        auto o4 = [](T m2, T m1, T c, T p1, T p2) {
          // (products by 16 are exact)
          return sub_rn(fma_rn_(T(16), p1, sub_rn(fma_rn_(T(16), m1, -m2), mul_rn(T(30), c))), p2);
        };
        V vz = vc<V>(0);
        if (!twod) {
          const V up1 = *reinterpret_cast<const V*>(slot(q - 2) + own), up2 = *reinterpret_cast<const V*>(slot(q - 1) + own);
          vz.x = o4(ua.x, ub.x, uc.x, up1.x, up2.x);
          vz.y = o4(ua.y, ub.y, uc.y, up1.y, up2.y);
        }
        visc.x = add_rn(add_rn(mul_rn(p.kx, o4(xl.x, xl.y, uc.x, uc.y, xh.x)),
                               mul_rn(p.ky, o4(ym2.x, ym1.x, uc.x, yp1.x, yp2.x))), mul_rn(p.kz, vz.x));
        visc.y = add_rn(add_rn(mul_rn(p.kx, o4(xl.y, uc.x, uc.y, xh.x, xh.y)),
                               mul_rn(p.ky, o4(ym2.y, ym1.y, uc.y, yp1.y, yp2.y))), mul_rn(p.kz, vz.y));
      }
    }
    // ---- the z-face between planes q-3 and q-2, once the line holds planes q-5 .. q
    V fz = vc<V>(0), u2 = uc;
    if (!twod) {
      const V uq = *reinterpret_cast<const V*>(plq + own);
      u2 = *reinterpret_cast<const V*>(slot(q - 2) + own);  // (before plane 2: a stale slot, not used)
      V fp, fm;
      split(uq, fp, fm);
      fz = line.push(fp, fm, uc, u2, need && q >= 2 * R - 1);
    }
    if (tma && edge) cp_async_wait<1>();  // this thread's patch of plane q - 1
    __syncthreads();  // f+- in place; every read of the output plane's slot is done
    if (tma && *abort_flag != 0) {
      // A wait expired: let the copies already issued (planes q+1 .. q+P) land before returning.
      if (tid == 0)
        for (int m = q + 1; m < Q && m <= q + TL::P; ++m) wait(m);
      return kPipeAborted;
    }
    if (q + TL::P + 1 < Q) issue(q + TL::P + 1);
    else if (!tma) cp_async_commit();
    if (out) {
      V un = uc, res = uc;
      if (any_upd) {
        if (!p.un_is_uin) {  // requested before the faces, used after them
          if (vec) {
            if (ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) un = *reinterpret_cast<const V*>(p.un + gi);
          } else {
            if (in0 && ADV_IN_RANGE(gi, sxy * nz, p.status)) un.x = p.un[gi];
            if (in1 && ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) un.y = p.un[gi + 1];
          }
        }
        auto face = [](const V* a, int st) {
          const V* const m = a + PART;
          return F::f(a[0], a[st], a[2 * st], a[3 * st], a[4 * st], m[st], m[2 * st], m[3 * st], m[4 * st], m[5 * st]);
        };
        if (need) {
          const V fx = face(xr, 1);
          fxS[(2 * warp) * TL::XF + lane] = fx.x;
          fxS[(2 * warp + 1) * TL::XF + lane] = fx.y;
        }
        V fym;
        if (need_y) {
          fym = face(yr, PX);
          fyS[tid] = fym;
        } else {
          fym = vc<V>(0);
        }
        if constexpr (EXACT) {
          // one value per lane of two warps: the FP64 pipe is each scheduler's own, and a warp's extra
          // work is waited for by all
          const int e = ((q & 7) == warp) ? lane : ((q + 1) & 7) == warp ? 32 + lane : TL::BY + TL::BX;
          if (cols && e < TL::BY + TL::BX) {
            const bool ex = e < TL::BY;
            const int i = ex ? e : e - TL::BY, st = ex ? 2 : 2 * PX;
            const T* const a = reinterpret_cast<const T*>(part + (ex ? (i / 2) * XS + TL::BX : YP + TL::BY * PX + i / 2)) + (i & 1);
            const T* const m = a + 2 * PART;
            const T f = weno_face_ref<Z, T>(a[0], a[st], a[2 * st], a[3 * st], a[4 * st], m[st], m[2 * st], m[3 * st],
                                            m[4 * st], m[5 * st]);
            if (ex) fxS[i * TL::XF + TL::BX] = f;
            else reinterpret_cast<T*>(fyS + TL::BY * PX)[i] = f;
          }
        } else if (warp == (q & 7) && cols && lane < TL::BY / 2 + PX) {
          const V f = face(part + l_src, l_st);
          if (l_x) {
            fxS[(2 * lane) * TL::XF + TL::BX] = f.x;
            fxS[(2 * lane + 1) * TL::XF + TL::BX] = f.y;
          } else {
            fyS[TL::BY * PX + lane - TL::BY / 2] = f;
          }
        }
        __syncthreads();
        // ---- RHS, stage combine
        const V fx0 = *reinterpret_cast<const V*>(fxS + row * TL::XF + 2 * cp);  // faces 2 cp, 2 cp + 1
        const V fx1 = {fx0.y, fxS[row * TL::XF + 2 * cp + 2]};
        const V fyp = fyS[tid + PX];
        V L;
        if constexpr (EXACT) {
          auto rhs = [&](T fxm, T fxp, T fym1, T fyp1, T fzm, T fzp) {
            return sub_rn(sub_rn(div_by(-sub_rn(fxp, fxm), p.dx, p.rdx), div_by(sub_rn(fyp1, fym1), p.dy, p.rdy)),
                          div_by(sub_rn(fzp, fzm), p.dz, p.rdz));
          };
          L = {rhs(fx0.x, fx1.x, fym.x, fyp.x, fz_prev.x, fz.x), rhs(fx0.y, fx1.y, fym.y, fyp.y, fz_prev.y, fz.y)};
        } else if constexpr (IsCandidates<D>::value) {
          L = vfma(vsub(fz_prev, fz), V{p.rdz, p.rdz},
                   vfma(vsub(fx0, fx1), V{p.rdx, p.rdx}, vmul(vsub(fym, fyp), V{p.rdy, p.rdy})));
        } else {
          L = vfma(vsub(fz_prev, fz), V{p.rdz, p.rdz},
                   vfma(vsub(fym, fyp), V{p.rdy, p.rdy}, vmul(vsub(fx0, fx1), V{p.rdx, p.rdx})));
        }
        if (VISC) {
          L = vadd(L, visc);
          // The reference's first viscous z-block starts at slab 3 yet runs 16 slabs, adding
          // slabs 16..18 twice (kernels.cu:464-491); reproduced only on request.
          if (p.bug_b2 && !per && k >= 16 && k <= 18 && k <= nz - 3) L = vadd(L, visc);
        }
        const V c = combine2(p.stage, un, uc, dt, L);
        if (upd0) res.x = c.x;
        if (upd1) res.y = c.y;
      }
      if (vec) {
        if (ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) *reinterpret_cast<V*>(p.out + gi) = res;
      } else {
        if (in0 && ADV_IN_RANGE(gi, sxy * nz, p.status)) p.out[gi] = res.x;
        if (in1 && ADV_IN_RANGE(gi + 1, sxy * nz, p.status)) p.out[gi + 1] = res.y;
      }
      const K k0 = in0 ? abs_key(res.x) : K(0), k1 = in1 ? abs_key(res.y) : K(0);
      kmax = k0 > kmax ? k0 : kmax;
      kmax = k1 > kmax ? k1 : kmax;
      gi += sxy;
    }
    fz_prev = fz;
    if (VISC) { ua = ub; ub = uc; }
    uc = u2;
  }
  if (tma && edge) cp_async_wait<0>();
  return n0 + (unsigned)Q;
}

// Minimum resident CTAs per SM the compiler must allow for (it caps registers accordingly): three for
// FP32 (80 registers; without the bound it takes 108 and two CTAs fit), two for FP64.
template <class T>
constexpr int burgers_min_ctas() {
  return sizeof(T) == 4 ? 3 : 2;
}

// CTA b's share of one grid's stage (work_split.h); a share crossing a tile boundary becomes segments.
template <class T, bool Z, class D, bool VISC, int MODE>
__device__ __forceinline__ void burgers_share(const CUtensorMap* tmap, const BurgersParams<T>& p, unsigned b) {
  using TL = BurgersTile;
  if (p.active && *p.active == 0) return;
  const int nz = p.nz;
  int64_t seg_a, seg_b;
  split_range(p.split, b, nz, &seg_a, &seg_b);
  burgers_load_scalars<T>(p);
  burgers_cta_init<T>(tmap, p.tma != 0);
  unsigned entries = 0;
  typename KeyOf<T>::type kmax = 0;
  for (int64_t pos = seg_a; pos < seg_b;) {
    const int64_t tile = div_units(pos, nz);
    const int zs = (int)(pos - tile * nz);
    const int ze = (int)min((int64_t)nz, zs + (seg_b - pos));
    pos += ze - zs;
    const int64_t ty = div_units(tile, p.tiles_x);
    const int x0 = (int)(tile - ty * p.tiles_x) * TL::BX, y0 = (int)ty * TL::BY;
    entries = burgers_segment<T, Z, D, VISC, MODE>(tmap, p, x0, y0, zs, ze, entries, kmax);
    if (entries == kPipeAborted) return;
  }
  burgers_flush_max(kmax, p.maxabs_key);
}

template <class T, bool Z, class D, bool VISC, int MODE>
__global__ void __launch_bounds__(256, burgers_min_ctas<T>())
burgers_stage_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ BurgersParams<T> p) {
  burgers_share<T, Z, D, VISC, MODE>(&tmap, p, blockIdx.x);
}

// One instance of a batched Burgers stage: the tensor map of its stage input and the stage's
// parameters (per-instance buffers, dt / Lax-Friedrichs sources, max|u| key, active flag).
template <class T>
struct alignas(64) BurgersBatchInst {
  CUtensorMap tmap;
  BurgersParams<T> p;
  int64_t unit_begin;  // first unit of this instance
  int64_t pad[7];
};

// Batched stage over more instances than a BurgersGroup holds: the units (instance, tile, z-plane) of all instances,
// instance-major then tile-major, are cut into gridDim.x equal contiguous ranges. Instances
// whose active flag is 0 are skipped (the choice is per segment, so uniform over the CTA).
template <class T, bool Z, class D, bool VISC, int MODE>
__global__ void __launch_bounds__(256, burgers_min_ctas<T>())
burgers_batch_kernel(const BurgersBatchInst<T>* __restrict__ inst, int n_inst, int64_t total_units, int tma) {
  using TL = BurgersTile;
  const int64_t seg_a = total_units * blockIdx.x / gridDim.x, seg_b = total_units * (blockIdx.x + 1) / gridDim.x;
  burgers_cta_init<T>(nullptr, tma != 0);
  unsigned entries = 0;
  int i = 0;
  {
    int lo = 0, hi = n_inst - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (inst[mid].unit_begin <= seg_a) lo = mid; else hi = mid - 1;
    }
    i = lo;
  }
  for (int64_t pos = seg_a; pos < seg_b;) {
    while (i + 1 < n_inst && inst[i + 1].unit_begin <= pos) ++i;
    // This segment's parameters, staged in shared memory and read from there on use (as the
    // single-problem kernel reads its constant-bank parameters). A register copy spilled 168
    // bytes per thread; with this staging the ensemble ran 2.4% faster.
    __shared__ BurgersParams<T> ps;
    __syncthreads();  // every thread is done with the previous segment's parameters
    if (threadIdx.x == 0) {
      ps = inst[i].p;
      burgers_load_scalars<T>(ps);
    }
    __syncthreads();
    const BurgersParams<T>& p = ps;
    const int64_t local = pos - inst[i].unit_begin;
    const int64_t inst_end = i + 1 < n_inst ? inst[i + 1].unit_begin : total_units;
    const int64_t tile = div_units(local, p.nz);
    const int zs = (int)(local - tile * p.nz);
    const int64_t stop = min(seg_b, inst_end);
    const int ze = (int)min((int64_t)p.nz, zs + (stop - pos));
    pos += ze - zs;
    if (p.active && *p.active == 0) continue;
    const int64_t ty = div_units(tile, p.tiles_x);
    const int x0 = (int)(tile - ty * p.tiles_x) * TL::BX, y0 = (int)ty * TL::BY;
    const CUtensorMap* tm = &inst[i].tmap;
    if (tma && threadIdx.x == 0) tma_prefetch_desc(tm);
    typename KeyOf<T>::type kmax = 0;
    entries = burgers_segment<T, Z, D, VISC, MODE>(tm, p, x0, y0, zs, ze, entries, kmax);
    if (entries == kPipeAborted) return;
    burgers_flush_max(kmax, p.maxabs_key);
  }
}

// A stage of up to MAX instances, each with CTAs [cta_begin[i], cta_begin[i + 1]) of its own (the host shares
// them out so that no instance's longest share stands out). The instances' parameters are the kernel's own:
// read from the constant bank like a single grid's, they cost no registers, where the table of
// burgers_batch_kernel, staged in shared memory and read again after every barrier, spilled 120-180 bytes per
// thread (us per stage of one 160^3 member: 83 in a batch, 68 in a group, 68 alone).
template <class T>
struct BurgersGroup {
  static constexpr int MAX = 64;
  const CUtensorMap* tmap;  // instance i's, i * stride bytes on
  size_t stride;
  int n;
  unsigned cta_begin[MAX];
  BurgersParams<T> p[MAX];
};

template <class T, bool Z, class D, bool VISC, int MODE>
__global__ void __launch_bounds__(256, burgers_min_ctas<T>())
burgers_group_kernel(const __grid_constant__ BurgersGroup<T> g) {
  int i = 0, hi = g.n - 1;
  while (i < hi) {
    const int mid = (i + hi + 1) / 2;
    if (g.cta_begin[mid] <= blockIdx.x) i = mid; else hi = mid - 1;
  }
  const CUtensorMap* tm = reinterpret_cast<const CUtensorMap*>(reinterpret_cast<const char*>(g.tmap) + i * g.stride);
  burgers_share<T, Z, D, VISC, MODE>(tm, g.p[i], blockIdx.x - g.cta_begin[i]);
}

}  // namespace adv
