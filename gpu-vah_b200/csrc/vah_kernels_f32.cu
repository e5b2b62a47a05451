// vah_kernels_f32.cu -- the set-up and validity kernels with FP32 state storage.
#include "vah_kernels_impl.cuh"

namespace vah {
VAH_INSTANTIATE_SETUP(float)
}  // namespace vah
