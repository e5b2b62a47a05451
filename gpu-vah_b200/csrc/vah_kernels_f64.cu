// vah_kernels_f64.cu -- the step and set-up kernels with FP64 state storage.
#include "vah_kernels_impl.cuh"

namespace vah {
VAH_INSTANTIATE_SETUP(double)
VAH_INSTANTIATE_STAGE(double)
}  // namespace vah
