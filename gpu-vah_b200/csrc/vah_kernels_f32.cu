// vah_kernels_f32.cu -- the step and set-up kernels with FP32 state storage (the FP32 form).
#include "vah_kernels_impl.cuh"

namespace vah {
VAH_INSTANTIATE_SETUP(float)
VAH_INSTANTIATE_SPLIT(float)
}  // namespace vah
