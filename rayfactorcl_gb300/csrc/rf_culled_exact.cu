// rf_culled_exact.cu -- the culled and narrow kernels with the IEEE FP32 op mapping;
// compiled with -fmad=false like rf_kern_exact.cu.
#include "rf_culled.cuh"
#include "rf_narrow.cuh"

namespace rf {
template cudaError_t launch_culled<MExact>(const TraceParams &, bool, bool, int, cudaStream_t);
template cudaError_t launch_narrow<MExact>(const TraceParams &, int, bool, int, cudaStream_t);
}  // namespace rf
