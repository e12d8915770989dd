// burgers_f32.cu -- FP32-state instantiations of the fused Burgers stage.
#include "burgers_launch.cuh"

namespace adv {

template <>
void* burgers_kernel_for<float>(const adv_burgers_desc& d, int mode, bool differentiated) {
  // (3D inviscid grids only have gradients; a FastDiv quotient and WENO5-JS keep the one form)
  if (differentiated && d.weno == ADV_WENO5_Z && d.div != ADV_DIV_FAST) {
    using C = Candidates<float>;
    return mode == BURGERS_3D_TMA ? reinterpret_cast<void*>(&burgers_stage_kernel<float, true, C, false, BURGERS_3D_TMA>)
                                  : reinterpret_cast<void*>(&burgers_stage_kernel<float, true, C, false, BURGERS_3D_COPY>);
  }
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_stage_kernel<float, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, float, K);
#undef K
  return nullptr;
}

adv_status burgers_launch_f32(const adv_burgers_desc& d, const BurgersLaunch& L, const BurgersStageArgs& a,
                              cudaStream_t s) {
  return burgers_launch_t<float>(d, L, a, s);
}

size_t burgers_smem_f32() { return BurgersSmem<float>::TOTAL; }

}  // namespace adv
