// burgers_launch.cuh -- host-side launch of the fused Burgers stage for one state type.
// Included by burgers_f32.cu and burgers_f64.cu so the two precisions compile in parallel.
#pragma once
#include "adv_internal.h"
#include "burgers_kernels.cuh"

namespace adv {

template <class T>
void* burgers_kernel_for(const adv_burgers_desc& d, int mode, bool differentiated);

// The kernel of a scheme and mode among all instantiations of K<Z, D, VISC, MODE>. FP32 divides alike
// for ADV_DIV_F32 and ADV_DIV_F64 (an FP64 quotient rounded to FP32 is the correctly rounded one).
#define ADV_BURGERS_PICK(d, mode, D, K)                                                                        \
  do {                                                                                                         \
    const bool z_ = (d).weno == ADV_WENO5_Z, fast_ = (d).div == ADV_DIV_FAST;                                  \
    const bool visc_ = (d).kx != 0.0 || (d).ky != 0.0 || (d).kz != 0.0;                                        \
    ADV_BURGERS_PICK_MODE(BURGERS_3D_TMA, mode, D, K)                                                          \
    ADV_BURGERS_PICK_MODE(BURGERS_3D_COPY, mode, D, K)                                                         \
    ADV_BURGERS_PICK_MODE(BURGERS_ANY, mode, D, K)                                                             \
  } while (0)
#define ADV_BURGERS_PICK_MODE(M, mode, D, K)                                                                   \
  if ((mode) == M) {                                                                                           \
    if (z_) return fast_ ? (visc_ ? K(true, FastDiv, true, M) : K(true, FastDiv, false, M))                    \
                         : (visc_ ? K(true, D, true, M) : K(true, D, false, M));                               \
    return fast_ ? (visc_ ? K(false, FastDiv, true, M) : K(false, FastDiv, false, M))                          \
                 : (visc_ ? K(false, D, true, M) : K(false, D, false, M));                                     \
  }

// Stage parameters of one launch (or of one instance of a batched launch).
template <class T>
BurgersParams<T> burgers_params(const adv_burgers_desc& d, const BurgersLaunch& L, const BurgersStageArgs& a) {
  BurgersParams<T> p;
  p.uin = static_cast<const T*>(a.u_in);
  p.un = static_cast<const T*>(a.u_n);
  p.out = static_cast<T*>(a.u_out);
  p.nx = d.nx; p.ny = d.ny; p.nz = d.nz;
  p.stage = a.stage;
  p.periodic = d.bc == ADV_BC_PERIODIC ? 1 : 0;
  p.bug_b2 = d.bug_b2;
  p.tiles_x = L.tiles_x;
  p.tiles_y = L.tiles_y;
  p.split = L.split;
  p.tma = L.tma ? 1 : 0;
  p.un_is_uin = a.u_n == a.u_in ? 1 : 0;
  const uintptr_t pair = 2 * sizeof(T);
  p.vec_ok = d.nx % 2 == 0 && (uintptr_t)a.u_n % pair == 0 && (uintptr_t)a.u_out % pair == 0 ? 1 : 0;
  p.lf_global = d.lf == ADV_LF_GLOBAL ? 1 : 0;
  p.dx = (T)d.dx; p.dy = (T)d.dy; p.dz = (T)d.dz;
  p.rdx = (T)(1.0 / d.dx); p.rdy = (T)(1.0 / d.dy); p.rdz = (T)(1.0 / d.dz);
  p.kx = (T)d.kx; p.ky = (T)d.ky; p.kz = (T)d.kz;
  p.dt_host = a.dt_host;
  p.alpha_host = a.alpha_host;
  p.dt_dev = a.dt_dev;
  p.alpha_dev = a.alpha_dev;
  p.alpha_key = a.alpha_key;
  p.maxabs_key = a.maxabs_key;
  p.active = a.active;
  p.status = device_status_ptr();
  return p;
}

template <class T>
adv_status burgers_launch_t(const adv_burgers_desc& d, const BurgersLaunch& L, const BurgersStageArgs& a,
                            cudaStream_t s) {
  BurgersParams<T> p = burgers_params<T>(d, L, a);
  void* k = burgers_kernel_for<T>(d, L.mode, L.differentiated);
  if (!k) return set_error(ADV_ERR_UNSUPPORTED, "burgers: no kernel for this configuration");
  void* args[] = {const_cast<CUtensorMap*>(&L.tmap_in), &p};
  ADV_CUDA_TRY(cudaLaunchKernel(k, L.grid, L.block, args, L.smem, s));
  count_launches(1);
  return ADV_OK;
}

}  // namespace adv
