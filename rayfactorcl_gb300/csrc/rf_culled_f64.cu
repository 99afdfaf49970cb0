// rf_culled_f64.cu -- the culled and narrow kernels in FP64; compiled with -fmad=false
// like rf_kern_exact.cu.
#include "rf_culled.cuh"
#include "rf_narrow.cuh"

namespace rf {
template cudaError_t launch_culled<MF64>(const TraceParams &, bool, bool, int, cudaStream_t);
template cudaError_t launch_narrow<MF64>(const TraceParams &, int, bool, int, cudaStream_t);
}  // namespace rf
