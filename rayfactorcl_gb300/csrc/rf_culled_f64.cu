// rf_culled_f64.cu -- the culled kernel in FP64; compiled with -fmad=false like
// rf_kern_exact.cu.
#include "rf_culled.cuh"

namespace rf {
template cudaError_t launch_culled<MF64>(const TraceParams &, bool, bool, int, cudaStream_t);
}  // namespace rf
