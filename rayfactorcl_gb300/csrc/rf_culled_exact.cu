// rf_culled_exact.cu -- the culled kernel with the IEEE FP32 op mapping; compiled with
// -fmad=false like rf_kern_exact.cu.
#include "rf_culled.cuh"

namespace rf {
template cudaError_t launch_culled<MExact>(const TraceParams &, bool, bool, int, cudaStream_t);
}  // namespace rf
