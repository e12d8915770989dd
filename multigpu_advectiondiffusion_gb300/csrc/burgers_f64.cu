// burgers_f64.cu -- FP64-state instantiations of the fused Burgers stage (the reference's own
// precision): reconstruction in the reference's operand order, bit-exact against the oracle,
// or, with ADV_DIV_FAST, the common-denominator form (one division per WENO side).
#include "burgers_launch.cuh"

namespace adv {

template <>
void* burgers_kernel_for<double>(const adv_burgers_desc& d, int mode, bool) {
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_stage_kernel<double, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, double, K);
#undef K
  return nullptr;
}

adv_status burgers_launch_f64(const adv_burgers_desc& d, const BurgersLaunch& L, const BurgersStageArgs& a,
                              cudaStream_t s) {
  return burgers_launch_t<double>(d, L, a, s);
}

size_t burgers_smem_f64() { return BurgersSmem<double>::TOTAL; }

}  // namespace adv
