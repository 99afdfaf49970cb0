// rf_masks.cu -- the batched kernel's cell masks (rf_batched.cuh), built on the
// device at each scene upload.
//
// For a row (scene, emitter) and each of the kMaskCells sort keys, bit j of the
// key's mask says whether any ray of that emitter whose key it is can reach
// surface j: origins in the ball of the key's parameter patch (16 per emitter),
// directions in the cone of its direction cell (cone[2*cell], axis and cos in
// xyzw, sin in the next entry's x), surfaces covered by up to kChainMax spheres
// (chain; radius < 0 ends the list) and, for planar surfaces, the plane (plane.xyz
// unit normal, w = normal . point; w NaN: not planar), which no ray crosses when
// the whole ball lies on one side and every direction of the cone points away from
// it.  A ray from a ball B(c, rho) with a direction within theta of axis a comes
// within R of a point C only if angle(C - c, a) <= theta + asin((R + rho) / |C - c|).
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "rf_internal.h"

namespace rf {
namespace {

__device__ void xf(const rf_primitive &e, double x, double y, double z, double w[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float *r = e.m + 4 * k;
        w[k] = (double)r[0] * x + (double)r[1] * y + (double)r[2] * z + (double)r[3];
    }
}

// Object-space box of parameter patch (pi, pj) of an emitter -- the points its
// rays start from when r[0] in [pi/4, (pi+1)/4) and r[1] in [pj/4, (pj+1)/4)
// (emission formulas RayFactorGPU.cl:298-443).  A patch's angles are a quarter
// turn, so sin and cos have their extremes at its ends, where they are 0 or +-1,
// and every coordinate is monotonic in the other parameter.  False when the
// formulas give no finite point (a frustum whose top radius is 1).
__device__ bool patch_box(const rf_primitive &e, int pi, int pj, double lo[3], double hi[3])
{
    const double a0 = pi / 4.0, a1 = (pi + 1) / 4.0, b0 = pj / 4.0, b1 = (pj + 1) / 4.0;
    const double u1 = e.util1, u2 = e.util2;
    if (e.type == RF_RECTANGLE) {
        lo[0] = 2 * a0 - 1;
        hi[0] = 2 * a1 - 1;
        lo[1] = 2 * b0 - 1;
        hi[1] = 2 * b1 - 1;
        lo[2] = hi[2] = 0.0;
        return true;
    }
    const bool flat = e.type == RF_DISC || e.type == RF_ANNULUS;
    const int quarter = (flat || e.type == RF_CYLINDER) ? pi : pj;  // which parameter is the angle
    double r0 = 1.0, r1 = 1.0, z0 = 0.0, z1 = 0.0;
    switch (e.type) {
    case RF_DISC: r0 = sqrt(b0); r1 = sqrt(b1); break;
    case RF_ANNULUS:
        r0 = sqrt(fmax(0.0, u1 + (u2 - u1) * b0));
        r1 = sqrt(fmax(0.0, u1 + (u2 - u1) * b1));
        break;
    case RF_CYLINDER: z0 = b0; z1 = b1; break;
    case RF_FRUSTUM:
        z0 = (sqrt(1.0 - a0 + a0 * u1 * u1) - 1.0) / (u1 - 1.0);
        z1 = (sqrt(1.0 - a1 + a1 * u1 * u1) - 1.0) / (u1 - 1.0);
        if (!isfinite(z0) || !isfinite(z1)) return false;
        r0 = 1.0 + z0 * (u1 - 1.0);
        r1 = 1.0 + z1 * (u1 - 1.0);
        break;
    case RF_SPHERE:
        z0 = 2 * a0 - 1;
        z1 = 2 * a1 - 1;
        r0 = sqrt(fmax(0.0, 1.0 - z0 * z0));
        r1 = sqrt(fmax(0.0, 1.0 - z1 * z1));
        break;
    default: return false;
    }
    // ends of the quarter turn: (cos, sin) = (1,0), (0,1), (-1,0), (0,-1); a disc's x
    // is the sine
    const double c0 = (quarter == 0) - (quarter == 2), s0 = (quarter == 1) - (quarter == 3);
    const double c1 = -s0, s1 = c0;
    const double xa = flat ? s0 : c0, xb = flat ? s1 : c1, ya = flat ? c0 : s0, yb = flat ? c1 : s1;
    lo[0] = fmin(fmin(r0 * xa, r0 * xb), fmin(r1 * xa, r1 * xb));
    hi[0] = fmax(fmax(r0 * xa, r0 * xb), fmax(r1 * xa, r1 * xb));
    lo[1] = fmin(fmin(r0 * ya, r0 * yb), fmin(r1 * ya, r1 * yb));
    hi[1] = fmax(fmax(r0 * ya, r0 * yb), fmax(r1 * ya, r1 * yb));
    lo[2] = fmin(z0, z1);
    hi[2] = fmax(z0, z1);
    return true;
}

// Ball around the image of an object-space box: the image of the box centre and
// the farthest image of a corner (the image is a parallelepiped: opposite corners
// are equally far), widened for the FP32 emission's rounding and approximations.
__device__ float4 box_ball(const rf_primitive &e, const double lo[3], const double hi[3])
{
    double c[3], rad2 = 0.0;
    xf(e, 0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2]), c);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        double w[3];
        xf(e, (q & 1) ? hi[0] : lo[0], (q & 2) ? hi[1] : lo[1], hi[2], w);
        rad2 = fmax(rad2, (w[0] - c[0]) * (w[0] - c[0]) + (w[1] - c[1]) * (w[1] - c[1]) + (w[2] - c[2]) * (w[2] - c[2]));
    }
    const double rad = sqrt(rad2), cn = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    return make_float4((float)c[0], (float)c[1], (float)c[2], (float)(rad * (1 + 1e-4) + 1e-5 * (cn + rad) + 1e-7));
}

// Spheres covering a surface: for a cylinder or frustum longer than it is wide,
// a chain of up to kChainMax spheres along its axis (points A + rho(z) (c0 cos +
// c1 sin) + Z z of slab [z0, z1] lie within rmax * max rho + |Z| (z1 - z0) / 2 of
// the slab's axis midpoint, rmax the largest radius of the ellipse spanned by the
// first two columns); otherwise the bounding sphere bs (radius in w).
__device__ void surface_chain(const rf_primitive &e, float4 bs, float4 *out)
{
    for (int k = 1; k < kChainMax; ++k) out[k] = make_float4(0.f, 0.f, 0.f, -1.f);
    out[0] = bs;
    if (e.type != RF_CYLINDER && e.type != RF_FRUSTUM) return;
    double A[3], Z[3], c0[3], c1[3];
    for (int k = 0; k < 3; ++k) {
        A[k] = e.m[4 * k + 3];
        c0[k] = e.m[4 * k + 0];
        c1[k] = e.m[4 * k + 1];
        Z[k] = e.m[4 * k + 2];
    }
    const double L = sqrt(Z[0] * Z[0] + Z[1] * Z[1] + Z[2] * Z[2]);
    const double g00 = c0[0] * c0[0] + c0[1] * c0[1] + c0[2] * c0[2];
    const double g11 = c1[0] * c1[0] + c1[1] * c1[1] + c1[2] * c1[2];
    const double g01 = c0[0] * c1[0] + c0[1] * c1[1] + c0[2] * c1[2];
    const double rmax = sqrt(0.5 * (g00 + g11 + sqrt((g00 - g11) * (g00 - g11) + 4 * g01 * g01)));
    const double top = e.type == RF_FRUSTUM ? (double)e.util1 : 1.0;
    const double wide = rmax * fmax(1.0, fabs(top));
    if (!(L > 0.0) || !(wide > 0.0) || !isfinite(L + wide)) return;
    const int K = (int)fmin((double)kChainMax, ceil(L / wide));
    if (K < 2) return;
    for (int k = 0; k < K; ++k) {
        const double z0 = (double)k / K, z1 = (double)(k + 1) / K, zm = 0.5 * (z0 + z1);
        const double rho = fmax(fabs(1.0 + z0 * (top - 1.0)), fabs(1.0 + z1 * (top - 1.0)));
        const double c[3] = {A[0] + Z[0] * zm, A[1] + Z[1] * zm, A[2] + Z[2] * zm};
        const double r = rmax * rho + 0.5 * L * (z1 - z0);
        const double cn = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
        out[k] = make_float4((float)c[0], (float)c[1], (float)c[2], (float)(r * (1 + 1e-4) + 1e-5 * (cn + r) + 1e-7));
    }
}

// Plane of a disc, annulus or rectangle: object z = 0 is row 2 of invm.
__device__ float4 surface_plane(const rf_primitive &e)
{
    const float4 none = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fc00000));
    if (e.type != RF_DISC && e.type != RF_ANNULUS && e.type != RF_RECTANGLE) return none;
    const double n[3] = {e.invm[8], e.invm[9], e.invm[10]};
    const double nn = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (!(nn > 0.0)) return none;
    return make_float4((float)(n[0] / nn), (float)(n[1] / nn), (float)(n[2] / nn), (float)(-(double)e.invm[11] / nn));
}

// The builder's inputs from the emission records, 16 threads per surface: one
// parameter patch each, the first also the sphere chain and the plane.  (On the
// host this took 4 us per surface, 10 ms for the 2535 surfaces of 24 scenes.)
__global__ void __launch_bounds__(128) mask_inputs_kernel(const rf_primitive *emit, const float4 *sph, int n,
                                                         float4 *patch, float4 *chain, float4 *plane)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, g = t >> 4, q = t & 15;
    if (g >= n) return;
    const rf_primitive e = emit[g];
    double lo[3], hi[3];
    // infinite radius when a patch has no finite bound: every surface is then a candidate
    patch[t] = patch_box(e, q >> 2, q & 3, lo, hi) ? box_ball(e, lo, hi)
                                                   : make_float4(0.f, 0.f, 0.f, __int_as_float(0x7f800000));
    if (q == 0) {
        surface_chain(e, sph[g], chain + (int64_t)g * kChainMax);
        plane[g] = surface_plane(e);
    }
}

// One block per (row, word of 32 surfaces, group of PP patches), one thread per
// direction cell.  What the cell test needs of a sphere depends on the patch
// alone, so a block works it out once per (sphere, patch) into shared memory and a
// thread is left with two broadcast loads, four FMA and a compare per sphere; the
// plane's normal against the direction is shared by the patches.  Bound by FP32 and
// shared-memory issue.  The earlier kernel gave each thread one mask word and read
// the spheres of 32 surfaces per lane from global memory: 25.3 ms for the 24 scenes
// (8.1e7 words) of a sweep of 10 to 400 surfaces, now 2.1 ms;
// 0.51 to 0.10 ms for 8 scenes of 10 to 100, 2.96 to 0.27 for the 252-surface furnace.
template <int PP>
__global__ void __launch_bounds__(256) build_masks_kernel(MaskInputs in, uint32_t *out)
{
    __shared__ float4 s_v[32][PP];  // sphere centre less ball centre, sqrt(L^2 - R^2) (-inf: the ball touches it)
    __shared__ float s_R[32][PP];   // radii plus margin
    __shared__ float4 s_plane[32];
    __shared__ int s_side[32][PP];  // the ball lies wholly on the + or - side of the plane, or 0
    __shared__ unsigned s_has;      // surfaces with a k-th sphere
    const int64_t first = (int64_t)blockIdx.x * kMaskCells;
    int lo = 0, hi = in.nrows - 1;  // the row holding this block's words (rows sorted by off)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (in.rows[mid].off <= first) lo = mid;
        else hi = mid - 1;
    }
    const MaskRow row = in.rows[lo];
    const SceneInfo si = in.scenes[row.scene];
    const int nwords = (si.n + 31) >> 5, w = (int)((first - row.off) / kMaskCells);
    const int tid = threadIdx.x, j0 = 32 * w, cnt = min(32, si.n - j0), p0 = blockIdx.y * PP;
    const float4 *ball = in.patch + (int64_t)(si.prim_off + row.emitter) * 16 + p0;
    const float4 ac = in.cone[2 * tid];
    const float sin_t = in.cone[2 * tid + 1].x;
    uint32_t bits[PP];
#pragma unroll
    for (int q = 0; q < PP; ++q) bits[q] = 0u;

    for (int k = 0; k < kChainMax; ++k) {
        __syncthreads();
        if (tid == 0) s_has = 0u;
        __syncthreads();
        for (int i = tid; i < cnt * PP; i += 256) {
            const int j = i / PP, q = i % PP, gj = si.prim_off + j0 + j;
            const float4 b = ball[q], sph = in.chain[(int64_t)gj * kChainMax + k];
            if (sph.w >= 0.0f) {
                const float vx = sph.x - b.x, vy = sph.y - b.y, vz = sph.z - b.z;
                const float L2 = vx * vx + vy * vy + vz * vz;
                const float R = (sph.w + b.w) * 1.0001f + 1e-5f * sqrtf(L2) + 1e-7f;
                const bool in_reach = !(L2 > R * R);
                s_v[j][q] = make_float4(vx, vy, vz, in_reach ? -__int_as_float(0x7f800000) : sqrtf(L2 - R * R));
                s_R[j][q] = in_reach ? 0.0f : R;
                if (q == 0) atomicOr(&s_has, 1u << j);
            }
            if (k == 0) {
                const float4 pl = in.plane[gj];
                int side = 0;
                if (pl.w == pl.w) {
                    const float h = pl.x * b.x + pl.y * b.y + pl.z * b.z - pl.w;
                    const float margin = b.w * 1e-4f + 1e-6f * (fabsf(pl.w) + b.w) + 1e-7f;
                    side = h > b.w + margin ? 1 : (h < -(b.w + margin) ? -1 : 0);
                }
                s_side[j][q] = side;
                if (q == 0) s_plane[j] = pl;
            }
        }
        __syncthreads();
        unsigned has = s_has;
        if (!has) break;  // (lists are contiguous: no later spheres either)
        for (; has; has &= has - 1) {
            const int j = __ffs(has) - 1;
#pragma unroll
            for (int q = 0; q < PP; ++q) {
                const float4 v = s_v[j][q];
                const float va = v.x * ac.x + v.y * ac.y + v.z * ac.z;
                if (va >= ac.w * v.w - sin_t * s_R[j][q]) bits[q] |= 1u << j;
            }
        }
    }
    for (int j = 0; j < cnt; ++j) {
        const float4 pl = s_plane[j];
        if (!(pl.w == pl.w)) continue;
        if (j0 + j == row.emitter) {  // a planar emitter cannot hit itself (self_skip)
#pragma unroll
            for (int q = 0; q < PP; ++q) bits[q] &= ~(1u << j);
            continue;
        }
        const float na = pl.x * ac.x + pl.y * ac.y + pl.z * ac.z;
#pragma unroll
        for (int q = 0; q < PP; ++q) {
            const int side = s_side[j][q];
            if ((side > 0 && na >= sin_t + 1e-4f) || (side < 0 && -na >= sin_t + 1e-4f)) bits[q] &= ~(1u << j);
        }
    }
    uint32_t *dst = out + row.off + (int64_t)(16 * tid + p0) * nwords + w;
#pragma unroll
    for (int q = 0; q < PP; ++q) dst[q * nwords] = bits[q];
}

}  // namespace

cudaError_t launch_mask_inputs(const rf_primitive *emit, const float4 *sph, int n, float4 *patch, float4 *chain,
                               float4 *plane, cudaStream_t st)
{
    mask_inputs_kernel<<<(n * 16 + 127) / 128, 128, 0, st>>>(emit, sph, n, patch, chain, plane);
    return cudaGetLastError();
}

cudaError_t launch_build_masks(const MaskInputs &in, uint32_t *out, cudaStream_t st)
{
    if (in.total_words <= 0) return cudaSuccess;
    const int64_t words32 = in.total_words / kMaskCells;  // (row, word) pairs
    if (words32 > 0x7fffffff) return cudaErrorInvalidValue;
    // a few small scenes have fewer pairs than the GPU's SMs take blocks: split the patches
    if (words32 < 1024)
        build_masks_kernel<4><<<dim3((unsigned)words32, 4), 256, 0, st>>>(in, out);
    else
        build_masks_kernel<16><<<dim3((unsigned)words32, 1), 256, 0, st>>>(in, out);
    return cudaGetLastError();
}

}  // namespace rf
