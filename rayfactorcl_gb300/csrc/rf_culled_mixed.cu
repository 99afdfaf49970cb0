// rf_culled_mixed.cu -- the culled kernel in mixed precision, for scenes with
// bounding surfaces or segment stacks, and the narrow kernel; default contraction
// like rf_kern_batched.cu, so that their tests are the batched kernel's.
#include "rf_culled.cuh"
#include "rf_narrow.cuh"

namespace rf {

cudaError_t launch_mixed_culled(const TraceParams &p, bool bv, bool rec, bool count, int blocks, cudaStream_t st)
{
    if (!culled_fits(p, bv) || p.n > kBatchTile) return cudaErrorInvalidValue;
    if (bv) {
        if (rec) return launch_culled_k<MMixed, true, true, true>(p, blocks, st);
        return count ? launch_culled_k<MMixed, true, false, true, true>(p, blocks, st)
                     : launch_culled_k<MMixed, true, false, true>(p, blocks, st);
    }
    if (rec) return launch_culled_k<MMixed, false, true, true>(p, blocks, st);
    return count ? launch_culled_k<MMixed, false, false, true, true>(p, blocks, st)
                 : launch_culled_k<MMixed, false, false, true>(p, blocks, st);
}

cudaError_t launch_mixed_narrow(const TraceParams &p, int split, bool rec, int sms, cudaStream_t st)
{
    return launch_narrow<MMixed>(p, split, rec, sms, st);
}

}  // namespace rf
