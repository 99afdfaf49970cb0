// rf_mixed_small.cuh -- mixed-precision tracing of one small scene with the
// plain kernel's launch shape (RayFactorGPU.cl:481-527's method: every ray
// against every surface).
//
// Below a few tens of surfaces the batched kernel's sorting and culling cost
// more than the tests they save.  This kernel keeps the scene's tables in shared
// memory, gives each thread 4 or 8 rays (one or two Philox draws) and tests them
// together against each surface in index order, like the plain kernel, with the
// batched kernel's arithmetic: the same emission (emit_mixed), the same mixed
// tests with FP64 re-evaluation of ill-conditioned quadrics, the same skipped
// self-test of a planar emitter (self_skip) and the same per-ray resolution
// (resolve_brute) as its small-scene path.  A scene traced here therefore gets,
// ray for ray, the batched kernel's results for it.
#pragma once

#include "rf_batched.cuh"

namespace rf {

static_assert(kSmallThreads % 32 == 0, "whole warps");

// Two rays a lane in packed FP32 (fma.rn.f32x2 and its like round each half as the
// scalar instruction does): one issue slot for two operations.  The kernel is bound
// by issue (75% of the slots, half of them FP32 multiplies and adds), so the rays of
// a thread are tested in pairs; comparisons, |x| and the function units' work stay
// scalar on the halves.  Each pair test gives t (anything when a quadric is
// ill-conditioned: that ray is traced again) as the scalar test of the same name
// does, operation by operation; a sign is moved into a negated factor where the packed
// forms have none.  16 surfaces, 2e7 rays: 0.87 -> 0.80 ms (about 15 to 22 issue slots
// saved of a quadric test's 57 to 85 instructions, less a block an SM for
// the registers).
struct Pair {
    float2 sx, sy, sz, cx, cy, cz;
};

// A surface for the pair tests: invm with each element twice, f = util1 - 1 and -f
// twice, and the record's aux.
struct PairRec {
    float4 m[6];  // rows r0..r2 as (x x y y), (z z w w)
    float4 f;     // f f -f -f
    float4 aux;
};

__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

__device__ __forceinline__ Pair xfrm_pair(const PairRec &h, const Pair &w)
{
    Pair o;
    const float4 a = h.m[0], b = h.m[1], c = h.m[2], d = h.m[3], e = h.m[4], f = h.m[5];
    o.sx = __ffma2_rn(lo2(a), w.sx, __ffma2_rn(hi2(a), w.sy, __ffma2_rn(lo2(b), w.sz, hi2(b))));
    o.cx = __ffma2_rn(lo2(a), w.cx, __ffma2_rn(hi2(a), w.cy, __fmul2_rn(lo2(b), w.cz)));
    o.sy = __ffma2_rn(lo2(c), w.sx, __ffma2_rn(hi2(c), w.sy, __ffma2_rn(lo2(d), w.sz, hi2(d))));
    o.cy = __ffma2_rn(lo2(c), w.cx, __ffma2_rn(hi2(c), w.cy, __fmul2_rn(lo2(d), w.cz)));
    o.sz = __ffma2_rn(lo2(e), w.sx, __ffma2_rn(hi2(e), w.sy, __ffma2_rn(lo2(f), w.sz, hi2(f))));
    o.cz = __ffma2_rn(lo2(e), w.cx, __ffma2_rn(hi2(e), w.cy, __fmul2_rn(lo2(f), w.cz)));
    return o;
}

__device__ __forceinline__ void plane_pair(const Pair &o, float2 &th, float2 &hx, float2 &hy)
{
    th = __fmul2_rn(o.sz, make_float2(MFast::rcp(-o.cz.x), MFast::rcp(-o.cz.y)));
    hx = __ffma2_rn(o.cx, th, o.sx);
    hy = __ffma2_rn(o.cy, th, o.sy);
}

__device__ __forceinline__ float pick_one(float t1, float t2, float z1, float z2, float eps)  // quadric_pick
{
    if (t1 < eps || z1 < 0.0f || z1 > 1.0f) t1 = MFast::inf();
    if (t2 < t1 && z2 > 0.0f && z2 < 1.0f && t2 > eps) return t2;
    return t1;
}

// Roots (B -+ disc) / A, nB = -B.
__device__ __forceinline__ float2 roots_pair(const Pair &o, float2 A, float2 nB, float2 d, float eps)
{
    const float2 disc = make_float2(MFast::sqrt(d.x), MFast::sqrt(d.y));  // NaN for a miss
    const float2 nra = make_float2(MFast::rcp(-A.x), MFast::rcp(-A.y));
    const float2 t1 = __fmul2_rn(nra, __fadd2_rn(nB, disc));
    const float2 t2 = __fmul2_rn(nra, make_float2(nB.x - disc.x, nB.y - disc.y));
    const float2 z1 = __ffma2_rn(o.cz, t1, o.sz), z2 = __ffma2_rn(o.cz, t2, o.sz);
    return make_float2(pick_one(t1.x, t2.x, z1.x, z2.x, eps), pick_one(t1.y, t2.y, z1.y, z2.y, eps));
}

template <int TYPE>
__device__ __forceinline__ float2 hit_pair(const PairRec &h, const Pair &w, float eps, bool &ill0, bool &ill1)
{
    const Pair o = xfrm_pair(h, w);
    const float inf = MFast::inf();
    if (TYPE == RF_RECTANGLE) {
        float2 th, hx, hy;
        plane_pair(o, th, hx, hy);
        return make_float2(fabsf(hx.x) > 1.0f || fabsf(hy.x) > 1.0f || th.x < eps ? inf : th.x,
                           fabsf(hx.y) > 1.0f || fabsf(hy.y) > 1.0f || th.y < eps ? inf : th.y);
    }
    if (TYPE == RF_DISC || TYPE == RF_ANNULUS) {
        float2 th, hx, hy;
        plane_pair(o, th, hx, hy);
        const float2 e = __ffma2_rn(hx, hx, __fmul2_rn(hy, hy));
        if (TYPE == RF_DISC)
            return make_float2(e.x <= 1.0f && th.x > eps ? th.x : inf, e.y <= 1.0f && th.y > eps ? th.y : inf);
        const float u1 = h.aux.y, u2 = h.aux.z;
        return make_float2(e.x >= u1 && e.x <= u2 && th.x > eps ? th.x : inf,
                           e.y >= u1 && e.y <= u2 && th.y > eps ? th.y : inf);
    }
    const float2 pw = __fmul2_rn(o.sy, o.cx);
    const float2 wz = make_float2(fmaf(o.sx.x, o.cy.x, -pw.x), fmaf(o.sx.y, o.cy.y, -pw.y));
    if (TYPE == RF_CYLINDER) {
        const float2 A = __ffma2_rn(o.cx, o.cx, __fmul2_rn(o.cy, o.cy));
        const float2 nB = __ffma2_rn(o.sx, o.cx, __fmul2_rn(o.sy, o.cy));
        const float2 d = make_float2(fmaf(-wz.x, wz.x, A.x), fmaf(-wz.y, wz.y, A.y));
        ill0 = ill_conditioned(d.x, fmaf(2.0f * fabsf(wz.x), fabsf(wz.x) + fabsf(pw.x), A.x));
        ill1 = ill_conditioned(d.y, fmaf(2.0f * fabsf(wz.y), fabsf(wz.y) + fabsf(pw.y), A.y));
        return roots_pair(o, A, nB, d, eps);
    }
    if (TYPE == RF_FRUSTUM) {
        const float2 f = lo2(h.f), nf = hi2(h.f);
        const float2 fdir = __fmul2_rn(f, o.cz), nfdir = __fmul2_rn(nf, o.cz);
        const float2 fstart = __ffma2_rn(f, o.sz, dup2(1.0f));
        const float2 A = __ffma2_rn(o.cx, o.cx, __ffma2_rn(o.cy, o.cy, __fmul2_rn(nfdir, fdir)));
        const float2 nB = __ffma2_rn(o.sx, o.cx, __ffma2_rn(o.sy, o.cy, __fmul2_rn(fstart, nfdir)));
        const float2 pu = __fmul2_rn(o.sx, nfdir), pv = __fmul2_rn(o.sy, nfdir);  // (negated)
        const float2 u = __ffma2_rn(o.cx, fstart, pu), v = __ffma2_rn(o.cy, fstart, pv);
        const float2 nw2 = make_float2(-wz.x * wz.x, -wz.y * wz.y);
        const float2 d = __ffma2_rn(u, u, __ffma2_rn(v, v, nw2));
        const float2 sq = __ffma2_rn(__fadd2_rn(wz, wz), wz, d);
        const float2 At = __ffma2_rn(fdir, fdir, __ffma2_rn(o.cx, o.cx, __fmul2_rn(o.cy, o.cy)));
        const float m0 = fmaf(3.0f, sq.x, 2.0f * fmaf(fabsf(u.x), fabsf(pu.x),
                                                      fmaf(fabsf(v.x), fabsf(pv.x), fabsf(wz.x) * fabsf(pw.x))));
        const float m1 = fmaf(3.0f, sq.y, 2.0f * fmaf(fabsf(u.y), fabsf(pu.y),
                                                      fmaf(fabsf(v.y), fabsf(pv.y), fabsf(wz.y) * fabsf(pw.y))));
        ill0 = ill_conditioned(d.x, m0) || fabsf(A.x) < kCondA * At.x;
        ill1 = ill_conditioned(d.y, m1) || fabsf(A.y) < kCondA * At.y;
        return roots_pair(o, A, nB, d, eps);
    }
    // RF_SPHERE (without RF_COMPAT_SPHERE)
    const float2 A = __ffma2_rn(o.cz, o.cz, __ffma2_rn(o.cx, o.cx, __fmul2_rn(o.cy, o.cy)));
    const float2 B = __ffma2_rn(o.cz, o.sz, __ffma2_rn(o.cx, o.sx, __fmul2_rn(o.cy, o.sy)));
    const float2 kx = make_float2(fmaf(o.cy.x, o.sz.x, -o.cz.x * o.sy.x), fmaf(o.cy.y, o.sz.y, -o.cz.y * o.sy.y));
    const float2 ky = make_float2(fmaf(o.cz.x, o.sx.x, -o.cx.x * o.sz.x), fmaf(o.cz.y, o.sx.y, -o.cx.y * o.sz.y));
    const float2 kz = make_float2(fmaf(o.cx.x, o.sy.x, -o.cy.x * o.sx.x), fmaf(o.cx.y, o.sy.y, -o.cy.y * o.sx.y));
    const float2 kk = __ffma2_rn(kx, kx, __ffma2_rn(ky, ky, __fmul2_rn(kz, kz)));
    const float2 d2 = make_float2(A.x - kk.x, A.y - kk.y);
    ill0 = ill_conditioned(d2.x, A.x * fmaf(4.0f, fabsf(o.sx.x) + fabsf(o.sy.x) + fabsf(o.sz.x), 1.0f));
    ill1 = ill_conditioned(d2.y, A.y * fmaf(4.0f, fabsf(o.sx.y) + fabsf(o.sy.y) + fabsf(o.sz.y), 1.0f));
    const float2 dd = make_float2(MFast::sqrt(d2.x), MFast::sqrt(d2.y));
    const float2 nra = make_float2(MFast::rcp(-A.x), MFast::rcp(-A.y));
    const float2 t1 = __fmul2_rn(__fadd2_rn(B, dd), nra);
    const float2 t2 = __fmul2_rn(make_float2(B.x - dd.x, B.y - dd.y), nra);
    return make_float2(t1.x > eps ? t1.x : (t2.x > eps ? t2.x : inf), t1.y > eps ? t1.y : (t2.y > eps ? t2.y : inf));
}

// PAIR: the pair tests, in 80 registers and three blocks an SM (four spill: 0.80 against
// 0.75 ms for the 16 surfaces of the stress scene, 2e7 rays); otherwise the scalar ones, in 64 and four, which
// is better while emission is most of the work.  Scalar / pairs, ms: 3 surfaces 3e7 rays
// 0.286 / 0.295, 6 surfaces 1e7 0.190 / 0.186, 12 surfaces 2e7 0.656 / 0.613, 16
// surfaces 2e7 0.874 / 0.799 -> pairs from kPairMin on; eight rays a thread (GPT 2, one
// block of 256 threads an SM) 16 surfaces 1.105 / 1.111, never pairs.
constexpr int kPairMin = 6;

template <int GPT, bool REC, bool PAIR>
__global__ void __launch_bounds__(kSmallThreads, GPT == 1 ? (PAIR ? 3 : 4) : 1) mixed_small_kernel(const TraceParams p)
{
    constexpr int R = 4 * GPT;
    static_assert(!PAIR || (GPT == 1 && !REC), "pairs: see kPairMin");
    __shared__ HitRec s_tab[kSmallMax];
    __shared__ PairRec s_pair[PAIR ? kSmallMax : 1];
    __shared__ int s_hist[kSmallMax];
    __shared__ rf_primitive s_emit;
    __shared__ float4 s_frame[kEmitFrameWords];

    const int n = p.n;
    const int tid = threadIdx.x, lane = tid & 31;
    const bool sc = (p.compat & RF_COMPAT_SPHERE) != 0;
    const float eps = p.eps;
    {
        const float4 *src = reinterpret_cast<const float4 *>(p.tab);
        float4 *dst = reinterpret_cast<float4 *>(s_tab);
        for (int i = tid; i < 4 * n; i += blockDim.x) dst[i] = __ldg(src + i);
        for (int i = tid; i < n; i += blockDim.x) s_hist[i] = 0;
        for (int i = tid; PAIR && i < 3 * n; i += blockDim.x) {
            const float4 r = __ldg(src + i / 3 * 4 + i % 3);
            PairRec &q = s_pair[i / 3];
            q.m[2 * (i % 3)] = make_float4(r.x, r.x, r.y, r.y);
            q.m[2 * (i % 3) + 1] = make_float4(r.z, r.z, r.w, r.w);
            if (i % 3 == 0) {
                const float4 aux = __ldg(src + i / 3 * 4 + 3);
                const float f = aux.y - 1.f;
                q.f = make_float4(f, f, -f, -f);
                q.aux = aux;
            }
        }
    }
    const int64_t c0 = (p.total_chunks * (int64_t)blockIdx.x) / gridDim.x;
    const int64_t c1 = (p.total_chunks * (int64_t)(blockIdx.x + 1)) / gridDim.x;
    int64_t seg_next = -1;
    Segment sg;
    sg.emitter = -1;
    int pending = 0, nref = 0;

    auto flush = [&](int emitter) {
        __syncthreads();
        unsigned long long *row = p.hits + (int64_t)emitter * n;
        for (int i = tid; i < n; i += blockDim.x) {
            const int v = s_hist[i];
            if (v) {
                atomicAdd(row + i, (unsigned long long)v);
                s_hist[i] = 0;
            }
        }
        __syncthreads();
    };

    for (int64_t c = c0; c < c1; ++c) {
        if (c >= seg_next) {  // block-uniform
            const int s = find_segment(p.seg, p.nseg, c);
            const Segment ns = p.seg[s];
            if (!REC && sg.emitter >= 0 && ns.emitter != sg.emitter) {
                flush(sg.emitter);
                pending = 0;
            }
            sg = ns;
            seg_next = (s + 1 < p.nseg) ? p.seg[s + 1].chunk_begin : INT64_MAX;
            __syncthreads();
            if (tid < (int)(sizeof(rf_primitive) / 4))
                reinterpret_cast<float *>(&s_emit)[tid] = reinterpret_cast<const float *>(p.emit + sg.emitter)[tid];
            if (tid < kEmitFrameWords) s_frame[tid] = p.frame[(int64_t)sg.emitter * kEmitFrameWords + tid];
            __syncthreads();
        }
        if (!REC && pending >= 4096) {  // keep the 32-bit bins far from overflow
            flush(sg.emitter);
            pending = 0;
        }
        ++pending;

        const int64_t gid0 = (sg.ray_begin >> 2) + (c - sg.chunk_begin) * (int64_t)(blockDim.x * GPT);
        Ray<float> ray[PAIR ? 1 : R];
        Pair w[PAIR ? R / 2 : 1];
        auto ray_of = [&](int k) -> decltype(auto) {
            if constexpr (PAIR) {
                const Pair &q = w[k >> 1];
                return k & 1 ? Ray<float>{q.sx.y, q.sy.y, q.sz.y, q.cx.y, q.cy.y, q.cz.y}
                             : Ray<float>{q.sx.x, q.sy.x, q.sz.x, q.cx.x, q.cy.x, q.cz.x};
            } else {
                return (ray[k]);
            }
        };
#pragma unroll
        for (int g = 0; g < GPT; ++g) {
            const int64_t gid = gid0 + (int64_t)g * blockDim.x + tid;
            const uint4 u = stream_bits(p.compat, p.key1, p.scene_id, sg.emitter, gid);
            const float uf[4] = {u01(u.x), u01(u.y), u01(u.z), u01(u.w)};
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                float r[4];
                rotate_uniforms(uf, v, r);
                const Ray<float> a = emit_mixed(s_emit, s_frame, r);
                if constexpr (PAIR) {
                    Pair &q = w[g * 2 + (v >> 1)];
                    (v & 1 ? q.sx.y : q.sx.x) = a.sx;
                    (v & 1 ? q.sy.y : q.sy.x) = a.sy;
                    (v & 1 ? q.sz.y : q.sz.x) = a.sz;
                    (v & 1 ? q.cx.y : q.cx.x) = a.cx;
                    (v & 1 ? q.cy.y : q.cy.x) = a.cy;
                    (v & 1 ? q.cz.y : q.cz.x) = a.cz;
                } else {
                    ray[g * 4 + v] = a;
                }
            }
        }
        float tb[R];
        int bi[R];
        uint32_t dmask = 0u;  // bit k: ray k deferred a test
#pragma unroll
        for (int k = 0; k < R; ++k) { tb[k] = MFast::inf(); bi[k] = -1; }
        const int skip = self_skip(s_emit, sg.emitter);  // block-uniform
        for (int j = 0; j < n; ++j) {
            if (j == skip) continue;
            const HitRec hr = s_tab[j];
            const int type = __float_as_int(hr.aux.x);
            auto pairs = [&](auto test) {
#pragma unroll
                for (int q = 0; q < R / 2; ++q) {
                    bool i0 = false, i1 = false;
                    const float2 t = test(w[q], i0, i1);
                    if (t.x < tb[2 * q]) { tb[2 * q] = t.x; bi[2 * q] = j; }
                    if (t.y < tb[2 * q + 1]) { tb[2 * q + 1] = t.y; bi[2 * q + 1] = j; }
                    if (i0) dmask |= 1u << (2 * q);
                    if (i1) dmask |= 2u << (2 * q);
                }
            };
            // the same per-type tests as hit_mixed, each case expanded for the thread's rays
            auto singles = [&](auto test) {
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    bool defer = false;
                    const float t = test(ray_of(k), defer);
                    if (t < tb[k]) { tb[k] = t; bi[k] = j; }
                    dmask |= defer ? (1u << k) : 0u;
                }
            };
#define RF_MIXED_ALL(T)                                                                                         \
    if constexpr (PAIR)                                                                                         \
        pairs([&](const Pair &q, bool &i0, bool &i1) { return hit_pair<T>(s_pair[j], q, eps, i0, i1); });       \
    else                                                                                                        \
        singles([&](const Ray<float> &q, bool &defer) { return hit_mixed(T, hr, q, eps, sc, defer); });
            switch (type) {  // warp-uniform
            case RF_DISC: RF_MIXED_ALL(RF_DISC) break;
            case RF_ANNULUS: RF_MIXED_ALL(RF_ANNULUS) break;
            case RF_RECTANGLE: RF_MIXED_ALL(RF_RECTANGLE) break;
            case RF_CYLINDER: RF_MIXED_ALL(RF_CYLINDER) break;
            case RF_FRUSTUM: RF_MIXED_ALL(RF_FRUSTUM) break;
            case RF_SPHERE:
                if (PAIR && sc)
                    singles([&](const Ray<float> &q, bool &) { return sphere_hit<MFast>(hr, q, eps, true); });
                else
                    RF_MIXED_ALL(RF_SPHERE)
                break;
            case kStackType: {  // one test for the segment stack j belongs to
                const int first = stack_first(hr, j);
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    bool defer = false;
                    int ring;
                    const float t = stack_mixed(hr, ray_of(k), eps, defer, ring);
                    if (t < tb[k]) { tb[k] = t; bi[k] = first + ring; }
                    dmask |= defer ? (1u << k) : 0u;
                }
                j = stack_end(hr, j) - 1;
                break;
            }
            case kPlateType: {  // one test for the plate j belongs to
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    int idx;
                    const float t = plate_mixed(hr, j, s_tab, true, ray_of(k), eps, idx);
                    if (t < tb[k]) { tb[k] = t; bi[k] = idx; }
                }
                j = stack_end(hr, j) - 1;
                break;
            }
            default: break;  // validated away on the host
            }
#undef RF_MIXED_ALL
        }
        unsigned long long *grow = p.hits + (int64_t)sg.emitter * n;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int64_t rid = (gid0 + (int64_t)(k >> 2) * blockDim.x + tid) * 4 + (k & 3);
            const bool valid = rid >= sg.ray_begin && rid < sg.ray_end;
            const int h = valid ? resolve_brute<true>(bi[k], (dmask >> k) & 1u, 0, n, s_tab, ray_of(k), eps, sc, skip, nref)
                                : -1;
            if (REC) {
                if (valid) p.rec[rid - p.rec_base] = h;
            } else {
                warp_tally(s_hist, h);  // every lane
            }
        }
    }
    if (!REC && sg.emitter >= 0) flush(sg.emitter);
    int tot = nref;
#pragma unroll
    for (int o = 16; o; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0 && tot && p.refined) atomicAdd(p.refined, (unsigned long long)tot);
}

// The bounding-surface walk (bv_select) of a scene of a few surfaces, one ray at a
// time: nothing to sort or cull for, and a walk's rays leave one another early.
// 2 surfaces under 2 bounding surfaces, 2e7 rays: 0.46 ms, 0.59 as a case of the
// batched kernel, 0.64 through the culled kernel's packets.
template <bool REC>
__global__ void __launch_bounds__(kSmallThreads, 4) mixed_small_bv_kernel(const TraceParams p)
{
    __shared__ HitRec s_tab[kSmallMax];
    __shared__ HitRec s_bvtab[kBatchMaxBV];
    __shared__ int4 s_bvinfo[kBatchMaxBV];
    __shared__ float4 s_bvbs[kBatchMaxBV];
    __shared__ int s_hist[kSmallMax];
    __shared__ rf_primitive s_emit;
    __shared__ float4 s_frame[kEmitFrameWords];

    const int n = p.n, tid = threadIdx.x, lane = tid & 31;
    const bool sc = (p.compat & RF_COMPAT_SPHERE) != 0, stale = (p.compat & RF_COMPAT_BV_STALE) != 0;
    const float eps = p.eps;
    for (int i = tid; i < 4 * n; i += blockDim.x)
        reinterpret_cast<float4 *>(s_tab)[i] = __ldg(reinterpret_cast<const float4 *>(p.tab) + i);
    for (int i = tid; i < 4 * p.nbv; i += blockDim.x)
        reinterpret_cast<float4 *>(s_bvtab)[i] = __ldg(reinterpret_cast<const float4 *>(p.bvtab) + i);
    for (int i = tid; i < p.nbv; i += blockDim.x) {
        s_bvinfo[i] = __ldg(p.bvinfo + i);
        s_bvbs[i] = __ldg(p.bvsph + i);
    }
    for (int i = tid; i < n; i += blockDim.x) s_hist[i] = 0;
    const int64_t c0 = (p.total_chunks * (int64_t)blockIdx.x) / gridDim.x;
    const int64_t c1 = (p.total_chunks * (int64_t)(blockIdx.x + 1)) / gridDim.x;
    int64_t seg_next = -1;
    Segment sg;
    sg.emitter = -1;
    int pending = 0, nref = 0;
    auto flush = [&](int emitter) {
        __syncthreads();
        unsigned long long *row = p.hits + (int64_t)emitter * n;
        for (int i = tid; i < n; i += blockDim.x) {
            const int v = s_hist[i];
            if (v) {
                atomicAdd(row + i, (unsigned long long)v);
                s_hist[i] = 0;
            }
        }
        __syncthreads();
    };
    for (int64_t c = c0; c < c1; ++c) {
        if (c >= seg_next) {  // block-uniform
            const int s = find_segment(p.seg, p.nseg, c);
            const Segment ns = p.seg[s];
            if (!REC && sg.emitter >= 0 && ns.emitter != sg.emitter) {
                flush(sg.emitter);
                pending = 0;
            }
            sg = ns;
            seg_next = (s + 1 < p.nseg) ? p.seg[s + 1].chunk_begin : INT64_MAX;
            __syncthreads();
            if (tid < (int)(sizeof(rf_primitive) / 4))
                reinterpret_cast<float *>(&s_emit)[tid] = reinterpret_cast<const float *>(p.emit + sg.emitter)[tid];
            if (tid < kEmitFrameWords) s_frame[tid] = p.frame[(int64_t)sg.emitter * kEmitFrameWords + tid];
            __syncthreads();
        }
        if (!REC && ++pending > 4096) {  // keep the 32-bit bins far from overflow
            flush(sg.emitter);
            pending = 1;
        }
        const int64_t gid = (sg.ray_begin >> 2) + (c - sg.chunk_begin) * (int64_t)blockDim.x + tid;
        const uint4 u = stream_bits(p.compat, p.key1, p.scene_id, sg.emitter, gid);
        const float uf[4] = {u01(u.x), u01(u.y), u01(u.z), u01(u.w)};
        const int skip = self_skip(s_emit, sg.emitter);  // block-uniform
#pragma unroll 1
        for (int v = 0; v < 4; ++v) {
            float r[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = (i + v + 1) & 3;
                r[i] = q == 0 ? uf[0] : (q == 1 ? uf[1] : (q == 2 ? uf[2] : uf[3]));
            }
            const Ray<float> ray = emit_mixed(s_emit, s_frame, r);
            const int64_t rid = gid * 4 + v;
            const bool valid = rid >= sg.ray_begin && rid < sg.ray_end;
            auto find = [&](int lo, int hi) {  // every child of [lo, hi), index order
                float tr = MFast::inf();
                int br = -1;
                bool dr = false;
#pragma unroll 1
                for (int j = lo; j < hi; ++j) {
                    if (j == skip) continue;
                    const HitRec h = s_tab[j];
                    const int type = __float_as_int(h.aux.x);
                    bool defer = false;
                    int idx;
                    const float t = test_mixed<true>(type, h, j, s_tab, true, ray, eps, sc, defer, idx);
                    if (t < tr) {
                        tr = t;
                        br = idx;
                    }
                    dr |= defer;
                    if (is_stack(type)) j = stack_end(h, j) - 1;
                }
                return resolve_brute<true>(br, dr, lo, hi, s_tab, ray, eps, sc, skip, nref);
            };
            const int h = valid ? bv_select(s_bvtab, s_bvinfo, s_bvbs, p.nbv, ray, eps, sc, stale, find) : -1;
            if (REC) {
                if (valid) p.rec[rid - p.rec_base] = h;
            } else {
                warp_tally(s_hist, h);  // every lane
            }
        }
    }
    if (!REC && sg.emitter >= 0) flush(sg.emitter);
#pragma unroll
    for (int o = 16; o; o >>= 1) nref += __shfl_xor_sync(0xffffffffu, nref, o);
    if (lane == 0 && nref && p.refined) atomicAdd(p.refined, (unsigned long long)nref);
}

}  // namespace rf
