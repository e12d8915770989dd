// burgers_batch_f32.cu -- FP32-state instantiations of the batched Burgers stage
// (burgers_batch_kernel in burgers_kernels.cuh) used by the ensembles.
#include "burgers_launch.cuh"

namespace adv {

template <class T>
void* burgers_batch_kernel_for(const adv_burgers_desc& d, int mode);
template <class T>
void* burgers_group_kernel_for(const adv_burgers_desc& d, int mode);

template <>
void* burgers_batch_kernel_for<float>(const adv_burgers_desc& d, int mode) {
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_batch_kernel<float, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, float, K);
#undef K
  return nullptr;
}

template <>
void* burgers_group_kernel_for<float>(const adv_burgers_desc& d, int mode) {
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_group_kernel<float, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, float, K);
#undef K
  return nullptr;
}

}  // namespace adv
