// burgers_batch_f64.cu -- FP64-state instantiations of the batched Burgers stage
// (burgers_batch_kernel in burgers_kernels.cuh) used by the ensembles.
#include "burgers_launch.cuh"

namespace adv {

template <class T>
void* burgers_batch_kernel_for(const adv_burgers_desc& d, int mode);
template <class T>
void* burgers_group_kernel_for(const adv_burgers_desc& d, int mode);

template <>
void* burgers_batch_kernel_for<double>(const adv_burgers_desc& d, int mode) {
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_batch_kernel<double, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, double, K);
#undef K
  return nullptr;
}

template <>
void* burgers_group_kernel_for<double>(const adv_burgers_desc& d, int mode) {
#define K(Z, D, V, M) reinterpret_cast<void*>(&burgers_group_kernel<double, Z, D, V, M>)
  ADV_BURGERS_PICK(d, mode, double, K);
#undef K
  return nullptr;
}

}  // namespace adv
