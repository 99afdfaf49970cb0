// rf_kern_batched.cu -- launchers of the batched mixed-precision persistent
// kernel (every instantiation: record / resident / counting / segment-stack variants).
#include "rf_trace_kernels.cuh"
#include "rf_batched.cuh"

namespace rf {

static_assert(kBatchThreads * kBatchDraws == kBatchChunkDraws, "chunk size");
static_assert(kBatchThreads == kBatchBlock, "block size");

size_t batched_smem_bytes() { return sizeof(BatchSmem); }

static_assert(sizeof(BatchSmem) <= 227 * 1024, "the batched kernel's shared memory exceeds a block's 227 KB");

template <bool REC, bool RES, bool CNT, bool STK>
static cudaError_t launch_k(const TraceParams &p, int grid, cudaStream_t st)
{
    const size_t smem = sizeof(BatchSmem);
    auto k = batched_kernel<REC, RES, CNT, STK>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k<<<grid, kBatchThreads, smem, st>>>(p);
    return cudaGetLastError();
}

template <bool STK>
static cudaError_t launch_b(const TraceParams &p, bool rec, bool resident, bool count, int grid, cudaStream_t st)
{
    if (rec) return resident ? launch_k<true, true, false, STK>(p, grid, st) : launch_k<true, false, false, STK>(p, grid, st);
    if (count) return resident ? launch_k<false, true, true, STK>(p, grid, st) : launch_k<false, false, true, STK>(p, grid, st);
    return resident ? launch_k<false, true, false, STK>(p, grid, st) : launch_k<false, false, false, STK>(p, grid, st);
}

cudaError_t launch_batched(const TraceParams &p, bool rec, bool resident, bool count, bool stacks, int grid,
                           cudaStream_t st)
{
    return stacks ? launch_b<true>(p, rec, resident, count, grid, st) : launch_b<false>(p, rec, resident, count, grid, st);
}

// Resident blocks per SM, queried once per process (every GPU of a run is the same
// part): the query costs microseconds on each launch otherwise.
template <bool REC, bool RES>
static int occ_b()
{
    static const int nb = [] {
        const size_t smem = sizeof(BatchSmem);
        int r = 0;
        auto k = batched_kernel<REC, RES, false, false>;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k, kBatchThreads, smem) != cudaSuccess) r = 0;
        return r;
    }();
    return nb;
}

int batched_blocks_per_sm(bool rec, bool resident)
{
    if (rec) return resident ? occ_b<true, true>() : occ_b<true, false>();
    return resident ? occ_b<false, true>() : occ_b<false, false>();
}

int batched_tile() { return kBatchTile; }

}  // namespace rf
