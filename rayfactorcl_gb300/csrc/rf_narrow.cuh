// rf_narrow.cuh -- traces of few rays: one ray a thread, its surfaces split over
// the warps of a block.
//
// The other kernels leave a GPU mostly idle below a few hundred thousand rays: the
// plain one gives a thread four or eight rays, the culled and batched ones sort at
// least 4096 into packets, and 1e4 rays are then a few warps with a long serial chain
// of tests each (400 surfaces, 1e4 rays: 230 us of which 200 are one warp's latency).
// Here a block of eight warps takes 256 / SPLIT rays: warp w holds the rays of slot
// w / SPLIT and tests part w % SPLIT of the surfaces in index order, every ray against
// every surface (RayFactorGPU.cl:445-472), so that the surface is the same in all its
// lanes; the parts' nearest hits meet in shared memory, the earlier part winning a tie
// as in the single loop.  A part repeats the emission, about 16 tests' time.  What
// bounds it is a warp's latency (n / SPLIT tests one after the other) until the GPU is
// full, then issue: past 1e5 to 3e5 rays the kernels that sort do less work.
// The arithmetic is the other kernels' own, so the results are theirs ray for ray; in
// mixed arithmetic, where those of larger traces count a hit only when the ray's own gate
// admits its surface (p.gate), the winner is held against that gate, and a ray whose
// winner fails it is traced again over the surfaces it admits.
// Measured, us, the kernel used before / this one: 20 surfaces 1e4 rays EXACT 24 / 9.6,
// FAST 14.5 / 7.7, MIXED 23 / 10; 48 surfaces FP64 183 / 105; 400 surfaces 1e4 rays
// EXACT 230 / 34, MIXED 135 / 36, 1e5 rays EXACT 304 / 165.  (The rule: rf_capi.cu,
// narrow_split.)
#pragma once

#include "rf_culled.cuh"

namespace rf {

template <class M, int SPLIT, bool REC>
__global__ void __launch_bounds__(kNarrowThreads, M::kF64 ? 2 : kNarrowBlocks) narrow_kernel(const TraceParams p)
{
    using T = typename M::T;
    constexpr bool kMixed = kIsMixed<M>;
    constexpr int kRays = kNarrowThreads / SPLIT;  // rays of a chunk
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HitRec *s_tab = reinterpret_cast<HitRec *>(smem_raw);
    double *s_tab64 = reinterpret_cast<double *>(s_tab + p.n);  // FP64: invm, 12 doubles a surface
    __shared__ rf_primitive s_emit;
    __shared__ Emit64 s_emit64;  // FP64
    __shared__ float4 s_frame[kMixed ? kFrameWords : 1];
    __shared__ T s_t[SPLIT > 1 ? kNarrowThreads : 1];
    __shared__ int s_i[SPLIT > 1 ? kNarrowThreads : 1];
    __shared__ int s_lo[SPLIT + 1];  // first surface of each part

    const int n = p.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = warp % SPLIT, slot = (warp / SPLIT) * 32 + lane;  // the ray's place in the chunk
    const bool sc = (p.compat & RF_COMPAT_SPHERE) != 0;
    const T eps = T(p.eps);
    for (int i = tid; i < 4 * n; i += kNarrowThreads)
        reinterpret_cast<float4 *>(s_tab)[i] = __ldg(reinterpret_cast<const float4 *>(p.tab) + i);
    if (M::kF64)
        for (int i = tid; i < 12 * n; i += kNarrowThreads)
            s_tab64[i] = __ldg(reinterpret_cast<const float *>(p.tab + i / 12) + i % 12);
    if (tid <= SPLIT) s_lo[tid] = n * tid / SPLIT;
    __syncthreads();
    if (kMixed && SPLIT > 1)  // no part begins inside a segment stack, which is one test
        for (int i = tid; i < n; i += kNarrowThreads) {
            const HitRec &h = s_tab[i];
            if (!is_stack(__float_as_int(h.aux.x))) continue;
            const int end = stack_end(h, i);
            for (int q = 1; q < SPLIT; ++q)
                if (i < n * q / SPLIT && n * q / SPLIT < end) s_lo[q] = end;
        }
    __syncthreads();
    const int lo = s_lo[part], hi = s_lo[part + 1];

    const int64_t c0 = p.total_chunks * (int64_t)blockIdx.x / gridDim.x;
    const int64_t c1 = p.total_chunks * (int64_t)(blockIdx.x + 1) / gridDim.x;
    int64_t seg_next = -1;
    Segment sg;
    sg.emitter = -1;
    int nref = 0;
    for (int64_t c = c0; c < c1; ++c) {
        if (c >= seg_next) {  // block-uniform
            const int s = find_segment(p.seg, p.nseg, c);
            sg = p.seg[s];
            seg_next = s + 1 < p.nseg ? p.seg[s + 1].chunk_begin : INT64_MAX;
            __syncthreads();
            if (tid < (int)(sizeof(rf_primitive) / 4))
                reinterpret_cast<float *>(&s_emit)[tid] = reinterpret_cast<const float *>(p.emit + sg.emitter)[tid];
            if (M::kF64) fill_emit64(s_emit64, p.emit[sg.emitter], tid);
            if (kMixed && tid < kFrameWords) s_frame[tid] = p.frame[(int64_t)sg.emitter * kFrameWords + tid];
            __syncthreads();
        }
        const int64_t rid = (sg.ray_begin & ~(int64_t)3) + (c - sg.chunk_begin) * kRays + slot;
        const bool valid = rid >= sg.ray_begin && rid < sg.ray_end;
        const uint4 u = stream_bits(p.compat, p.key1, (p.compat & RF_COMPAT_STREAMS) ? 0u : p.scene_id, sg.emitter, rid >> 2);
        const float uf[4] = {u01(u.x), u01(u.y), u01(u.z), u01(u.w)};
        float r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = (i + (int)(rid & 3) + 1) & 3;
            r[i] = q == 0 ? uf[0] : (q == 1 ? uf[1] : (q == 2 ? uf[2] : uf[3]));
        }
        Ray<T> ray;
        if constexpr (kMixed)
            ray = emit_mixed(s_emit, s_frame, r);
        else if constexpr (M::kF64)
            ray = emit_ray<M>(s_emit64, r);
        else
            ray = emit_ray<M>(s_emit, r);
        const int skip = kMixed && planar(s_emit.type) ? sg.emitter : -1;
        int cell = 0;  // the batched kernel's sort key of the ray
        if constexpr (kMixed)
            if (p.gate == 2) cell = ray_key(ray, r);
        T tb = M::inf();
        int bi = -1;
#pragma unroll 1
        for (int j = lo; j < hi; ++j) {  // the same in every lane
            const HitRec h = s_tab[j];
            const int type = __float_as_int(h.aux.x);
            if constexpr (kMixed) {
                if (j == skip) continue;
                bool defer = false;
                int idx;
                float t = test_mixed<true>(type, h, j, s_tab, true, ray, eps, sc, defer, idx);
                if (__any_sync(0xffffffffu, defer) && defer) {
                    const float2 f = deferred_f64(s_tab + j, j, ray, eps, sc);
                    t = f.x;
                    idx = __float_as_int(f.y);
                    nref += valid;
                }
                if (t < tb) {
                    tb = t;
                    bi = idx;
                }
                if (is_stack(type)) j = stack_end(h, j) - 1;
            } else {
                T t;
                if constexpr (M::kF64) {
                    const HitRec64::Row *q = reinterpret_cast<const HitRec64::Row *>(s_tab64 + 12 * j);
                    t = hit_any<M>(type, HitRec64{q[0], q[1], q[2], h.aux}, ray, eps, sc, M::inf());
                } else {
                    t = hit_any<M>(type, h, ray, eps, sc, M::inf());
                }
                if (t < tb) {
                    tb = t;
                    bi = j;
                }
            }
        }
        if (SPLIT > 1) {
            s_t[tid] = tb;
            s_i[tid] = bi;
            __syncthreads();
            if (part == 0) {
#pragma unroll
                for (int q = 1; q < SPLIT; ++q) {
                    if (s_t[tid + 32 * q] < tb) {  // (a tie: the earlier part's, the lower index)
                        tb = s_t[tid + 32 * q];
                        bi = s_i[tid + 32 * q];
                    }
                }
            }
        }
        if constexpr (kMixed) {
            if (p.gate && part == 0 && valid && bi >= 0) {
                const float4 b = __ldg(p.bsph + bi);
                if (p.gate == 1) {  // the culled kernel's
                    const float idd = MFast::rcp(dot3(ray.cx, ray.cy, ray.cz, ray.cx, ray.cy, ray.cz));
                    if (!reaches(ray, idd, b)) {
                        const int2 q = retrace_f64<true, true>(n, s_tab, p.bsph, nullptr, ray, idd, eps, sc, skip);
                        bi = q.x;
                        nref += q.y;
                    }
                } else {  // the batched kernel's
                    const float idd = MFast::rcp(ray.cx * ray.cx + ray.cy * ray.cy + ray.cz * ray.cz);
                    const int64_t mo = p.mask_off ? p.mask_off[sg.emitter] : -1;
                    const uint32_t *mcell = mo < 0 ? nullptr : p.cmask + mo + cell * ((n + 31) >> 5);
                    if (!own_gate(mcell, bi, ray, idd, b)) {
                        const int2 q = retrace_f64<true>(n, s_tab, p.bsph, mcell, ray, idd, eps, sc, skip);
                        bi = q.x;
                        nref += q.y;
                    }
                }
            }
        }
        if (part == 0) {  // warp-uniform
            if (REC) {
                if (valid) p.rec[rid - p.rec_base] = bi;
            } else {
                warp_tally_global(p.hits + (int64_t)sg.emitter * n, valid ? bi : -1);
            }
        }
        if (SPLIT > 1) __syncthreads();  // before the next chunk's parts
    }
    if (kMixed) {
#pragma unroll
        for (int o = 16; o; o >>= 1) nref += __shfl_xor_sync(0xffffffffu, nref, o);
        if (lane == 0 && nref) atomicAdd(p.refined, (unsigned long long)nref);
    }
}

template <class M, int SPLIT>
static cudaError_t launch_narrow_s(const TraceParams &p, bool rec, int sms, cudaStream_t st)
{
    constexpr size_t kRec = sizeof(HitRec) + (M::kF64 ? 12 * sizeof(double) : 0);
    const size_t smem = p.n * kRec;
    const void *k = rec ? (const void *)narrow_kernel<M, SPLIT, true> : (const void *)narrow_kernel<M, SPLIT, false>;
    if (smem > 40 * 1024) {  // (the largest launch's size: see launch_culled_k)
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kNarrowMax * kRec));
        if (e != cudaSuccess) return e;
    }
    const int per_sm = M::kF64 ? 2 : kNarrowBlocks;
    const int grid = (int)max((int64_t)1, min((int64_t)sms * per_sm, p.total_chunks));
    if (rec)
        narrow_kernel<M, SPLIT, true><<<grid, kNarrowThreads, smem, st>>>(p);
    else
        narrow_kernel<M, SPLIT, false><<<grid, kNarrowThreads, smem, st>>>(p);
    return cudaGetLastError();
}

template <class M>
cudaError_t launch_narrow(const TraceParams &p, int split, bool rec, int sms, cudaStream_t st)
{
    if (p.n <= 0 || p.n > kNarrowMax) return cudaErrorInvalidValue;
    switch (split) {
    case 1: return launch_narrow_s<M, 1>(p, rec, sms, st);
    case 2: return launch_narrow_s<M, 2>(p, rec, sms, st);
    case 4: return launch_narrow_s<M, 4>(p, rec, sms, st);
    case 8: return launch_narrow_s<M, 8>(p, rec, sms, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace rf
