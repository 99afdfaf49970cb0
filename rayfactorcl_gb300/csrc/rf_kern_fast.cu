// rf_kern_fast.cu -- single-scene kernels with the FP32 hardware
// approximations (the counterparts of OpenCL native_*), compiled with the
// default contraction of products and sums into FMA: the plain kernel and the
// small-scene mixed-precision kernel.
#include "rf_trace_kernels.cuh"
#include "rf_batched.cuh"
#include "rf_mixed_small.cuh"

namespace rf {
template cudaError_t launch_trace<MFast>(const LaunchCfg &, const TraceParams &, cudaStream_t);
template int trace_blocks_per_sm<MFast>(const LaunchCfg &);

template <int GPT, bool REC, bool PAIR>
static cudaError_t launch_s(const TraceParams &p, int grid, cudaStream_t st)
{
    mixed_small_kernel<GPT, REC, PAIR><<<grid, kSmallThreads, 0, st>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_mixed_small(const TraceParams &p, int gpt, bool rec, int grid, cudaStream_t st)
{
    if (p.n <= 0 || p.n > kSmallMax) return cudaErrorInvalidValue;
    if (rec) return launch_s<1, true, false>(p, grid, st);
    if (gpt == 2) return launch_s<2, false, false>(p, grid, st);
    return p.n < kPairMin ? launch_s<1, false, false>(p, grid, st) : launch_s<1, false, true>(p, grid, st);
}

cudaError_t launch_mixed_small_bv(const TraceParams &p, bool rec, int grid, cudaStream_t st)
{
    if (p.n <= 0 || p.n > kSmallMax || p.nbv <= 0 || p.nbv > kBatchMaxBV) return cudaErrorInvalidValue;
    if (rec)
        mixed_small_bv_kernel<true><<<grid, kSmallThreads, 0, st>>>(p);
    else
        mixed_small_bv_kernel<false><<<grid, kSmallThreads, 0, st>>>(p);
    return cudaGetLastError();
}

// Resident blocks per SM, queried once per process (every GPU of a run is the same part).
template <int GPT, bool REC, bool PAIR>
static int occ_s()
{
    static const int nb = [] {
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, mixed_small_kernel<GPT, REC, PAIR>, kSmallThreads, 0) !=
            cudaSuccess)
            r = 0;
        return r;
    }();
    return nb;
}

int mixed_small_blocks_per_sm(int n, int gpt, bool rec)
{
    if (rec) return occ_s<1, true, false>();
    if (gpt == 2) return occ_s<2, false, false>();
    return n < kPairMin ? occ_s<1, false, false>() : occ_s<1, false, true>();
}

}  // namespace rf
