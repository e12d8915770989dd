// heat2d_multi.cu -- 2D FP32 heat, several time steps per launch (overlapped temporal tiling) for
// adv_heat_run.
//
// A 2D grid of the reference's sizes (SingleGPU/Diffusion2d: 512^2 .. 1001^2 nodes, 1-4 MB per
// array) is too small to hide a launch per stage: a single-stage launch spends most of its time
// in launch gaps and in the load -> compute -> store latency of one plane. Here a CTA loads a
// 64 x 64 block of nodes into registers once, advances it K steps in place -- after each stage the
// values are valid on a block smaller by the stencil radius R on every side, so the tile it writes
// is what is left after the last one -- and writes that tile once: one launch and one pass over
// memory per K steps (FP32; in FP64 the recomputed halo costs more on the FP64 pipe than the
// launches it saves, so FP64 keeps one stage per launch).
//
// Layout: a warp owns 8 whole rows, a lane two adjacent nodes of each, so y neighbours are the
// thread's own registers, x neighbours one shuffle per side, the arithmetic runs two nodes at a time
// in paired FP32 instructions, and only a warp's outermost R rows go through shared memory (double
// buffered: one barrier per stage). The form before this kept the block in shared memory (six
// accesses per node and step, scalar arithmetic) at 14.5 us per 8 steps of a 512^2 grid.
// Each node's update is the fused single-stage kernel's expression (lap / combine of
// heat_stage.cuh, the fused multiply-add form), applied to the same neighbour values, so the result
// equals the single-stage launches bit for bit.
#include <algorithm>

#include "adv_device.cuh"
#include "adv_internal.h"
#include "heat_stage.cuh"

namespace adv {

template <int ORDER, bool RK3, int STEPS>
struct Heat2Multi {
  static constexpr int WARPS = 8, RY = 8;          // warps per CTA, rows per warp
  static constexpr int EX = 64, EY = WARPS * RY;   // block held in registers
  static constexpr int R = ORDER / 2;
  static constexpr int K = STEPS;                  // steps per launch at most
  static constexpr int H = K * (RK3 ? 3 : 1) * R;  // halo: one radius per stage
  static constexpr int BX = EX - 2 * H, BY = EY - 2 * H;  // nodes written
  static_assert(BX >= 32 && BY >= 32 && H % 2 == 0, "tile");
};

struct Heat2MultiParams {
  const float* in;
  float* out;
  int nx, ny, frozen, zero_boundary, steps;
  int vec_ok;  // pairs of nodes aligned for one access
  float kx, ky, dt;
  int* status;  // device status word (bounds-checked build)
};

template <int ORDER, bool RK3, int STEPS>
__global__ void __launch_bounds__(256) heat2d_multi_kernel(const __grid_constant__ Heat2MultiParams p) {
  using M = Heat2Multi<ORDER, RK3, STEPS>;
  constexpr int R = M::R, RY = M::RY, WARPS = M::WARPS;
  // [parity][warp][its first R rows, its last R rows]
  __shared__ float2 rows[2][WARPS][2 * R][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nx = p.nx, ny = p.ny, F = p.frozen;
  const int x = (int)blockIdx.x * M::BX - M::H + 2 * lane;          // grid coordinates of this thread's
  const int y = (int)blockIdx.y * M::BY - M::H + RY * warp;          // first node
  const size_t total = (size_t)nx * ny;
  // nodes off the grid read as 0; no update of a node that is written ever reads them
  float2 u[RY];
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    const size_t o = (size_t)(y + r) * nx + x;
    const bool row = y + r >= 0 && y + r < ny;
    if (p.vec_ok) {  // x is even, and so is nx: both nodes on the grid or neither
      u[r] = row && x >= 0 && x < nx && ADV_IN_RANGE(o + 1, total, p.status)
                 ? *reinterpret_cast<const float2*>(p.in + o) : make_float2(0.f, 0.f);
    } else {
      u[r].x = row && x >= 0 && x < nx && ADV_IN_RANGE(o, total, p.status) ? p.in[o] : 0.f;
      u[r].y = row && x + 1 >= 0 && x + 1 < nx && ADV_IN_RANGE(o + 1, total, p.status) ? p.in[o + 1] : 0.f;
    }
  }
  // Every stage updates the whole block with the interior formula, without per-node domain tests:
  // values that are no longer valid (a ring that grows by R per stage, fed at the block's edges by
  // whatever the shuffle or the clamped row gives), and values of nodes off the grid, are never read
  // by a valid interior node (those are at least F >= R nodes inside the grid). Frozen nodes of the
  // grid then take their own rule (kept, or 0 on the outermost layer with zero_boundary); only CTAs
  // whose block reaches into the frozen layers test for them.
  const int bx0 = (int)blockIdx.x * M::BX - M::H, by0 = (int)blockIdx.y * M::BY - M::H;
  const bool inner = bx0 >= F && bx0 + M::EX <= nx - F && by0 >= F && by0 + M::EY <= ny - F;
  // frozen columns of this thread (the same in every row) and rows of this warp (bit r)
  const bool fx0 = x < F || x >= nx - F, fx1 = x + 1 < F || x + 1 >= nx - F;
  const bool zx0 = p.zero_boundary && (x == 0 || x == nx - 1), zx1 = p.zero_boundary && (x + 1 == 0 || x + 1 == nx - 1);
  unsigned frow = 0, zrow = 0;
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    if (y + r < F || y + r >= ny - F) frow |= 1u << r;
    if (p.zero_boundary && (y + r == 0 || y + r == ny - 1)) zrow |= 1u << r;
  }
  const float2 kx = make_float2(p.kx, p.kx), ky = make_float2(p.ky, p.ky), dt = make_float2(p.dt, p.dt);
  float2 un[RK3 ? RY : 1];
  int par = 0;
  auto stage = [&](auto stage_c) {
    constexpr int STAGE = decltype(stage_c)::value;
#pragma unroll
    for (int d = 0; d < R; ++d) {
      rows[par][warp][d][lane] = u[d];
      rows[par][warp][R + d][lane] = u[RY - R + d];
    }
    __syncthreads();
    float2 up[R], dn[R];  // the R rows above (nearest last) and below (nearest first)
    const int wu = warp > 0 ? warp - 1 : 0, wd = warp < WARPS - 1 ? warp + 1 : warp;
#pragma unroll
    for (int d = 0; d < R; ++d) {
      up[d] = rows[par][wu][R + d][lane];
      dn[d] = rows[par][wd][d][lane];
    }
    par ^= 1;
    // FROZEN: 0 no frozen node in the block, 1 frozen columns only in this warp's rows, 2 any
    auto update = [&](auto frozen_c) {
      constexpr int FROZEN = decltype(frozen_c)::value;
      float2 m1 = up[R - 1], m2 = up[0];  // old rows r-1 and r-2
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        const float2 c = u[r];
        auto below = [&](int d) {  // old row r + d
          const int j = r + d;
          return j < RY ? u[j < RY ? j : 0] : dn[j < RY ? 0 : j - RY < R ? j - RY : 0];
        };
        const float2 p1 = below(1);
        const float ly = __shfl_up_sync(0xffffffffu, c.y, 1), rx = __shfl_down_sync(0xffffffffu, c.x, 1);
        float2 L;
        if constexpr (ORDER == 2) {
          // lap's operations; the x part node by node (as pairs its neighbours would straddle the
          // register pairs: packing them cost 13% at 2048^2)
          const float2 Sx = make_float2(add_rn(fma_rn(-2.f, c.x, c.y), ly), add_rn(fma_rn(-2.f, c.y, rx), c.x));
          const float2 Sy = add_rn(fma_rn(make_float2(-2.f, -2.f), c, p1), m1);
          L = fma_rn(ky, Sy, mul_rn(kx, Sx));
        } else {
          const float lx = __shfl_up_sync(0xffffffffu, c.x, 1), ry = __shfl_down_sync(0xffffffffu, c.y, 1);
          L = lap<float2, ORDER, 2, true>(make_float2(lx, ly), make_float2(ly, c.x), c, make_float2(c.y, rx),
                                          make_float2(rx, ry), m2, m1, p1, below(2), c, c, c, c, kx, ky, kx);
        }
        float2 v = combine<float2, true>(STAGE, STAGE == 1 ? c : un[RK3 ? r : 0], c, dt, L);
        if (FROZEN) {
          const bool fr = FROZEN == 2 && (frow >> r & 1u), zr = FROZEN == 2 && (zrow >> r & 1u);
          if (fx0 || fr) v.x = zx0 || zr ? 0.f : c.x;
          if (fx1 || fr) v.y = zx1 || zr ? 0.f : c.y;
        }
        u[r] = v;
        m2 = m1;
        m1 = c;
      }
    };
    if (inner) update(std::integral_constant<int, 0>{});
    else if (frow == 0) update(std::integral_constant<int, 1>{});  // (the same choice in all lanes of a warp)
    else update(std::integral_constant<int, 2>{});
  };
#pragma unroll 1
  for (int s = 0; s < p.steps; ++s) {
    if constexpr (RK3) {
#pragma unroll
      for (int r = 0; r < RY; ++r) un[r] = u[r];
      stage(std::integral_constant<int, 1>{});
      stage(std::integral_constant<int, 2>{});
      stage(std::integral_constant<int, 3>{});
    } else {
      stage(std::integral_constant<int, 1>{});
    }
  }
  // the tile itself: lanes and rows H nodes inside the block
  if (2 * lane < M::H || 2 * lane >= M::H + M::BX) return;
#pragma unroll
  for (int r = 0; r < RY; ++r) {
    const int j = RY * warp + r;
    if (j < M::H || j >= M::H + M::BY || y + r >= ny) continue;
    const size_t o = (size_t)(y + r) * nx + x;
    if (p.vec_ok) {
      if (x < nx && ADV_IN_RANGE(o + 1, total, p.status)) *reinterpret_cast<float2*>(p.out + o) = u[r];
    } else {
      if (x < nx && ADV_IN_RANGE(o, total, p.status)) p.out[o] = u[r].x;
      if (x + 1 < nx && ADV_IN_RANGE(o + 1, total, p.status)) p.out[o + 1] = u[r].y;
    }
  }
}

namespace {
template <int ORDER, bool RK3, int STEPS>
adv_status launch_t(const adv_heat_desc& d, const void* in, void* out, int steps, cudaStream_t s) {
  using M = Heat2Multi<ORDER, RK3, STEPS>;
  Heat2MultiParams p;
  p.in = static_cast<const float*>(in);
  p.out = static_cast<float*>(out);
  p.nx = d.nx;
  p.ny = d.ny;
  p.frozen = d.frozen;
  p.zero_boundary = d.zero_boundary;
  p.steps = steps;
  p.vec_ok = d.nx % 2 == 0 && (uintptr_t)in % 8 == 0 && (uintptr_t)out % 8 == 0 ? 1 : 0;
  p.kx = (float)d.kx;
  p.ky = (float)d.ky;
  p.dt = (float)d.dt;
  p.status = device_status_ptr();
  const dim3 grid((unsigned)((d.nx + M::BX - 1) / M::BX), (unsigned)((d.ny + M::BY - 1) / M::BY));
  heat2d_multi_kernel<ORDER, RK3, STEPS><<<grid, 32 * M::WARPS, 0, s>>>(p);
  ADV_CUDA_TRY(cudaGetLastError());
  count_launches(1);
  return ADV_OK;
}
}  // namespace

bool heat2d_multi_eligible(const adv_heat_desc& d) {
  // grid.y of the launch (at least 32 rows per CTA)
  return d.ndim == 2 && d.dtype == ADV_F32 && (d.ny + 31) / 32 <= 65535;
}

// Steps per launch: SSP-RK3 2 (six stages); O4 forward Euler 8; O2 16 where the 32-node tiles it leaves
// still give every CTA an SM of its own, else 8 (48-node tiles: fewer nodes computed twice).
int heat2d_multi_steps(const adv_heat_desc& d, int time_scheme) {
  if (time_scheme == ADV_SSPRK3) return 2;
  if (d.order != 2) return 8;
  DeviceInfo di;
  const int sms = device_info(&di) == ADV_OK ? di.sms : 152;
  return (int64_t)((d.nx + 31) / 32) * ((d.ny + 31) / 32) <= sms ? 16 : 8;
}

adv_status heat2d_multi_launch(const adv_heat_desc& d, int time_scheme, const void* in, void* out, int steps,
                               cudaStream_t s) {
  const int most = heat2d_multi_steps(d, time_scheme);
  if (!heat2d_multi_eligible(d) || steps < 1 || steps > most || in == out)
    return set_error(ADV_ERR_INVALID_ARG, "heat2d multi-step: bad arguments");
  if (time_scheme == ADV_SSPRK3)
    return d.order == 2 ? launch_t<2, true, 2>(d, in, out, steps, s) : launch_t<4, true, 2>(d, in, out, steps, s);
  if (d.order == 4) return launch_t<4, false, 8>(d, in, out, steps, s);
  return most == 16 ? launch_t<2, false, 16>(d, in, out, steps, s) : launch_t<2, false, 8>(d, in, out, steps, s);
}

}  // namespace adv
