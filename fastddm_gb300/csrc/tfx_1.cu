// Fixed-point temporal kernels of the float-float tier (tfx.cuh): any plan, none, and 2 x 2^6 points.
// tfx_1.cu .. tfx_4.cu hold the variants so that they compile in parallel.
#include "tfx.cuh"

namespace fddm {
TfxKernels tfx_kernels_1(int variant) {
  switch (variant) {
    case 0: return {&k_tfx<0>, &k_tfx_list<0>};
    case 1: return {&k_tfx<1>, &k_tfx_list<1>};
    case 6: return {&k_tfx<6>, &k_tfx_list<6>};
    default: return {nullptr, nullptr};
  }
}
}  // namespace fddm
