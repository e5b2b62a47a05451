// vah_kernels_f64.cu -- the step and set-up kernels with FP64 state storage.
#include "vah_kernels_impl.cuh"

namespace vah {
VAH_INSTANTIATE_SETUP(double)
VAH_INSTANTIATE_SPLIT(double)
template cudaError_t launch_stage<double>(const StageArgs<double> &, int, cudaStream_t);
}  // namespace vah
