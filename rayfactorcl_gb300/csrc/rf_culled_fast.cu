// rf_culled_fast.cu -- the culled and narrow kernels with the FP32 hardware
// approximations; default contraction like rf_kern_fast.cu.
#include "rf_culled.cuh"
#include "rf_narrow.cuh"

namespace rf {
template cudaError_t launch_culled<MFast>(const TraceParams &, bool, bool, int, cudaStream_t);
template cudaError_t launch_narrow<MFast>(const TraceParams &, int, bool, int, cudaStream_t);
}  // namespace rf
