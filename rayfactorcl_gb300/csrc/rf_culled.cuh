// rf_culled.cuh -- nearest hits of one scene in the plain kernels' arithmetic
// (MExact, MFast, MF64), with the surfaces a ray cannot hit left out.
//
// The plain kernel (rf_trace_kernels.cuh) tests every ray against every surface,
// RayFactorGPU.cl:445-472.  Here a block sorts a chunk of one emitter's rays by
// direction and emission patch, its warps take packets of 32 similar rays, and a
// packet tests, in index order, the surfaces whose bounding sphere one of its
// rays reaches, each with the plain kernel's own arithmetic.  A surface is left
// out only when its test, rounding included, could not return a hit, so every
// ray gets the plain kernel's nearest hit bit for bit, whatever packet it is in:
//
// * rf_bounds.cu (cull_tables) bounds the points where a test can place a hit: the
//   object-space shape grown by the test's rounding (for quadrics |Q| <= 128 u S^2 at
//   the hit, from the cancellation in B^2 - AC, S the longest object-space
//   coordinate of a ray up to it), as a world sphere grown again by this file's own
//   FP32 rounding.  The bound of a cone fails for rays whose direction makes its
//   A = c^T N c vanish; `band` lets those through (a frustum's sphere carries the
//   sign bit in its radius as the mark).
// * A ray with a non-finite or vanishing component is tested against everything,
//   with the rest of its packet.
// * Consecutive cylinders with nearly the same linear part (to 1e-5) that tile a
//   longer cylinder (a furnace wall of rings) are first intersected as one, in FP32: the roots, with
//   error bounds, name the one or two rings that a ring's own test could accept,
//   and only those are tested, each lane its own.  Concentric annuli in one plane
//   whose radii meet share one plane hit, exactly: the same operations give the
//   same radius, and a binary search finds the member.
//
// What bounds it: FP32 issue, like the batched mixed-precision kernel whose
// structure it shares; in MF64 the FP64 pipe.  64 surfaces, EXACT, 1e8 rays: 5.7 ms
// (plain 18.2), of which draws, keys and sort 0.6, emission and packet bounds 1.3,
// the spheres 2.2 (9 candidates per packet) and the tests 1.7 (5.3 per packet, of
// which 2.4 find a hit for some ray; the plain kernel makes 64 per ray).  The
// furnace (180-ring wall, two plates, bounding surfaces), 1e7 rays: 1.04 ms EXACT
// (plain 7.9), 0.85 FAST (5.7); 1e6 rays in FP64 2.0 (35.4).  In mixed precision, 5e7
// rays: 2.48 ms with bounding surfaces (3.36 as a variant of the batched kernel, which
// spilled 600 bytes a thread), 1.99 without (2.30); the reference's furnace model,
// 2e7 rays, 0.96 (1.65).
#pragma once

#include "rf_trace_kernels.cuh"
#include "rf_batched.cuh"

namespace rf {

// Shared memory of a block: arrays sized by the launch's chunk (cd draws), the
// surfaces kept resident (nres, 0: read through L1), the histogram row (nhist,
// 0: global tallies) and the bounding surfaces (nbv).  live: the surfaces that can be
// candidates, in index order (a stack's first member stands for all), with bs in the
// same order: a furnace's 252 surfaces are 35.
struct CulledLayout {
    int cnt = 0, perm = 0, unif = 0, tab = 0, bs = 0, bvtab = 0, bvinfo = 0, bvbs = 0, hist = 0, live = 0, bytes = 0;
    __host__ __device__ constexpr CulledLayout(int cd, int nres, int nhist, int nbv)
    {
        cnt = 0;
        perm = cnt + kCells * 4;
        unif = perm + cd * 8;
        tab = unif + cd * 12;
        bs = tab + nres * (int)sizeof(HitRec);
        bvtab = bs + nres * 16;
        bvinfo = bvtab + nbv * (int)sizeof(HitRec);
        bvbs = bvinfo + nbv * 16;
        hist = bvbs + nbv * 16;
        live = hist + nhist * 4;
        bytes = live + (nres * 2 + 15) / 16 * 16;
    }
};

__device__ __forceinline__ Ray<float> to_f32(const Ray<float> &r) { return r; }
__device__ __forceinline__ Ray<float> to_f32(const Ray<double> &r)
{
    return Ray<float>{(float)r.sx, (float)r.sy, (float)r.sz, (float)r.cx, (float)r.cy, (float)r.cz};
}

__device__ __forceinline__ bool planar(int type) { return type == RF_DISC || type == RF_ANNULUS || type == RF_RECTANGLE; }

// Sort key of a ray from its uniforms alone: an approximate direction (hardware
// sin/cos, reciprocals) in the 256 octahedral cells above the 4 x 4 cell of the
// two surface parameters.  Any key is correct; similar rays should share one.
// f: a planar emitter's rotation (rows), set up once per emitter.
__device__ __forceinline__ int quick_key(const rf_primitive &e, const float4 *f, const float r[4])
{
    float so, co;
    MFast::sincos(r[2] * k2PiF, so, co);
    const float st = MFast::sqrt(r[3]);
    const float ox = st * co, oy = st * so, oz = MFast::sqrt(1.0f - r[3]);
    float cx, cy, cz;
    if (planar(e.type)) {
        cx = dot3(f[0].x, f[0].y, f[0].z, ox, oy, oz);
        cy = dot3(f[1].x, f[1].y, f[1].z, ox, oy, oz);
        cz = dot3(f[2].x, f[2].y, f[2].z, ox, oy, oz);
    } else {
        float px, py, pz = 0.0f;
        MFast::sincos((e.type == RF_CYLINDER ? r[0] : r[1]) * k2PiF, py, px);
        if (e.type == RF_FRUSTUM) {
            pz = 1.0f - e.util1;
        } else if (e.type == RF_SPHERE) {
            pz = fmaf(2.0f, r[0], -1.0f);
            const float rho = MFast::sqrt(fmaf(-pz, pz, 1.0f));
            px *= rho;
            py *= rho;
        }
        float nx = dot3(e.invm[0], e.invm[4], e.invm[8], px, py, pz);
        float ny = dot3(e.invm[1], e.invm[5], e.invm[9], px, py, pz);
        float nz = dot3(e.invm[2], e.invm[6], e.invm[10], px, py, pz);
        const float il = MFast::rsqrt(dot3(nx, ny, nz, nx, ny, nz)) * e.util2;
        nx *= il;
        ny *= il;
        nz *= il;
        const float d = MFast::rcp(fmaxf(1.0f + nz, 1e-6f));
        const float k = d * fmaf(ny, ox, -nx * oy);
        cx = fmaf(nz, ox, fmaf(ny, k, nx * oz));
        cy = fmaf(nz, oy, fmaf(-nx, k, ny * oz));
        cz = fmaf(nz, oz, -fmaf(nx, ox, ny * oy));
    }
    return (direction_cell(cx, cy, cz) << 4) | ((int)(r[0] * 4.0f) << 2) | (int)(r[1] * 4.0f);
}

// Rotation rows of alignRayDirection (RayFactorGPU.cl:87-97) for a planar
// emitter's normal, to the accuracy a sort key needs.
__device__ __forceinline__ void quick_frame(const rf_primitive &e, float4 *f)
{
    float x = e.invm[8], y = e.invm[9], z = e.invm[10];
    const float il = MFast::rsqrt(dot3(x, y, z, x, y, z));
    x *= il;
    y *= il;
    z *= il;
    const float d = MFast::rcp(fmaxf(1.0f + z, 1e-6f));
    f[0] = make_float4(fmaf(d * y, y, z), -d * x * y, x, 0.0f);
    f[1] = make_float4(-d * x * y, fmaf(d * x, x, z), y, 0.0f);
    f[2] = make_float4(-x, -y, z, 0.0f);
}

// As reaches (rf_batched.cuh), for the ray's points up to the nearest hit so far, beyond which no hit
// counts: the distance from the centre at the nearest parameter t of those, oc2 - 2 t
// bb + t^2 cc, rounded by a few u reach^2 (the spheres allow for 64, rf_bounds.cu:
// check_w).  For FP64, whose tests cost 70 times a gate: 1e6 rays 48 surfaces 1.37 ->
// 1.33 ms, 400 surfaces 7.6 -> 5.6.  In FP32 the three more instructions a gate cost
// more than the tests they save below 200 surfaces (EXACT 1e8 rays, 64: 5.83 -> 5.94
// ms; 2e7 rays, 400: 5.53 -> 5.25).
__device__ __forceinline__ bool reaches_before(const Ray<float> &r, float cc, float idd, const float4 b, double tb)
{
    const float ox = b.x - r.sx, oy = b.y - r.sy, oz = b.z - r.sz;
    const float oc2 = dot3(ox, oy, oz, ox, oy, oz);
    const float bb = dot3(ox, oy, oz, r.cx, r.cy, r.cz);
    const float t = fminf(fmaxf(bb * idd, 0.0f), __double2float_ru(tb));
    return fmaf(t, fmaf(t, cc, -bb) - bb, oc2) <= fabsf(b.w);
}

// As packet_bounds and packet_may_hit of the batched kernel, fused like reaches.
__device__ __forceinline__ Packet bounds_of(const Ray<float> &r, float idd)
{
    Packet pk;
    pk.ox = 0.5f * (warp_min(r.sx) + warp_max(r.sx));
    pk.oy = 0.5f * (warp_min(r.sy) + warp_max(r.sy));
    pk.oz = 0.5f * (warp_min(r.sz) + warp_max(r.sz));
    const float dx = r.sx - pk.ox, dy = r.sy - pk.oy, dz = r.sz - pk.oz;
    pk.rho = fmaf(MFast::sqrt(warp_max(dot3(dx, dy, dz, dx, dy, dz))), 1.0001f, 1e-30f);
    const float il = MFast::sqrt(idd);
    const float nx = r.cx * il, ny = r.cy * il, nz = r.cz * il;
    const float ax = 0.5f * (warp_min(nx) + warp_max(nx));
    const float ay = 0.5f * (warp_min(ny) + warp_max(ny));
    const float az = 0.5f * (warp_min(nz) + warp_max(nz));
    const float al2 = dot3(ax, ay, az, ax, ay, az);
    const bool ok = al2 > 1e-6f;
    const float ial = ok ? MFast::rsqrt(al2) : 0.0f;
    pk.ax = ax * ial;
    pk.ay = ay * ial;
    pk.az = az * ial;
    const float c = warp_min(dot3(nx, ny, nz, pk.ax, pk.ay, pk.az)) - 1e-4f;  // for rounding
    pk.cull = ok && c > 0.0f;
    pk.cos_t = c;
    pk.sin_t = MFast::sqrt(fmaxf(0.0f, fmaf(-c, c, 1.0f))) * 1.0001f;
    return pk;
}

__device__ __forceinline__ bool packet_reaches(const Packet &pk, const float4 b)
{
    const float vx = b.x - pk.ox, vy = b.y - pk.oy, vz = b.z - pk.oz;
    const float L2 = dot3(vx, vy, vz, vx, vy, vz);
    const float R = fmaf(MFast::sqrt(fabsf(b.w)), 1.0001f, pk.rho);
    const float R2 = R * R;
    const float va = dot3(vx, vy, vz, pk.ax, pk.ay, pk.az);
    return !(L2 > R2) || va >= fmaf(pk.cos_t, MFast::sqrt(L2 - R2), -pk.sin_t * R);
}

// c^T N c of a cone's A for direction c, N in q0.xyz (diagonal) and q1.xyz
// (yz, xz, xy, doubled).
__device__ __forceinline__ float cone_A(const float4 q0, const float4 q1, float x, float y, float z)
{
    return fmaf(x, fmaf(q0.x, x, q1.z * y), fmaf(y, fmaf(q0.y, y, q1.x * z), z * fmaf(q0.z, z, q1.y * x)));
}

// A ray along which the frustum's A nearly vanishes (its roots then carry
// unbounded rounding): q0.w is the threshold for a unit direction.
__device__ __forceinline__ bool band(const float4 *quad, int j, const Ray<float> &r, float cc)
{
    const float4 q0 = __ldg(quad + 2 * j), q1 = __ldg(quad + 2 * j + 1);
    return !(fabsf(cone_A(q0, q1, r.cx, r.cy, r.cz)) > q0.w * cc);
}

// The same for some direction of the packet's cone.  With c = a cos f + e sin f (a
// the axis, e square to it, f up to the half-angle), c^T N c differs from
// a^T N a cos^2 f by at most 2 sin f cos f |(N a) square to a| + sin^2 f |N|; q1.w = |N|.
__device__ __forceinline__ bool packet_band(const float4 *quad, int j, const Packet &pk)
{
    const float4 q0 = __ldg(quad + 2 * j), q1 = __ldg(quad + 2 * j + 1);
    const float nx = fmaf(q0.x, pk.ax, 0.5f * fmaf(q1.z, pk.ay, q1.y * pk.az));
    const float ny = fmaf(q0.y, pk.ay, 0.5f * fmaf(q1.z, pk.ax, q1.x * pk.az));
    const float nz = fmaf(q0.z, pk.az, 0.5f * fmaf(q1.y, pk.ax, q1.x * pk.ay));
    const float A = dot3(nx, ny, nz, pk.ax, pk.ay, pk.az);
    const float side = MFast::sqrt(fmaxf(0.0f, fmaf(-A, A, dot3(nx, ny, nz, nx, ny, nz))) + 1e-6f * q1.w * q1.w);
    const float c2 = pk.cos_t * pk.cos_t;
    return !(fabsf(A) * c2 > fmaf(2.0f * pk.sin_t, side, fmaf(pk.sin_t * pk.sin_t, q1.w, q0.w)));
}

// Surface j's FP64 record (tab64: invm row by row, 12 doubles a surface, then the
// bounding surfaces').  48 surfaces, 1e6 rays: 1.27 -> 1.03 ms, 400 surfaces 4.78 -> 3.61,
// with the emitter's matrices converted once a row.
__device__ __forceinline__ HitRec64 load_rec64(const double *tab64, int j, const float4 aux)
{
    const double2 *q = reinterpret_cast<const double2 *>(tab64 + 12 * (size_t)j);
    HitRec64 h;
    double2 a = __ldg(q), b = __ldg(q + 1);
    h.r0 = {a.x, a.y, b.x, b.y};
    a = __ldg(q + 2);
    b = __ldg(q + 3);
    h.r1 = {a.x, a.y, b.x, b.y};
    a = __ldg(q + 4);
    b = __ldg(q + 5);
    h.r2 = {a.x, a.y, b.x, b.y};
    h.aux = aux;
    return h;
}

// An emitter's record in FP64, one element a thread.
__device__ __forceinline__ void fill_emit64(Emit64 &q, const rf_primitive &e, int tid)
{
    if (tid < 12) {
        q.m[tid] = e.m[tid];
        q.invm[tid] = e.invm[tid];
    }
    if (tid == 12) {
        q.util1 = e.util1;
        q.util2 = e.util2;
        q.type = e.type;
    }
}

// Nearest hit among the rings [a, a + m) of a cylinder stack: the tests of the
// rings that the stack's own roots leave possible, each lane its own, with the
// plain kernel's arithmetic.  In the first ring's frame every point that a ring's
// test can accept has |x^2 + y^2 - 1| <= mg.x and z in its ring to within mg.y
// (rf_bounds.cu: ring_stack), so t lies between (B -+ sqrt(D + A mg.x)) / A and
// (B -+ sqrt(D - A mg.x)) / A; mg.z / sqrt(A) covers the rounding of these roots.
// Such an interval names one or two rings; NaN and overflow widen it to all.
template <class M>
__device__ __forceinline__ void ring_hits(const HitRec *tab, bool resident, const double *tab64, int a, int m, const float4 mg,
                                          const Ray<typename M::T> &ray, const Ray<float> &w, typename M::T eps,
                                          bool odd, typename M::T &tb, int &bi)
{
    using T = typename M::T;
    int k1 = 0, e1 = m - 1, k2 = 0, e2 = -1;
    if (!odd) {
        const HitRec h = resident ? tab[a] : load_rec(tab, a);
        const Ray<float> o = xfrm_ray<MFast>(h, w);
        const float A = fmaf(o.cx, o.cx, o.cy * o.cy);
        const float B = -fmaf(o.sx, o.cx, o.sy * o.cy);
        const float wz = fmaf(o.sx, o.cy, -o.sy * o.cx);
        const float D = fmaf(-wz, wz, A);
        const float dk = A * mg.x;
        const float ra = MFast::rcp(A), isa = MFast::rsqrt(A);
        const float hi = MFast::sqrt(fmaxf(D + dk, 0.0f)), lo = MFast::sqrt(fmaxf(D - dk, 0.0f));
        const float te = mg.z * isa, zs = fmaf(fabsf(o.cz), te, mg.y);
        const float t1a = (B - hi) * ra, t1b = (B - lo) * ra, t2a = (B + lo) * ra, t2b = (B + hi) * ra;
        const float z1a = fmaf(o.cz, t1a, o.sz), z1b = fmaf(o.cz, t1b, o.sz);
        const float z2a = fmaf(o.cz, t2a, o.sz), z2b = fmaf(o.cz, t2b, o.sz);
        const float feps = (float)eps, ftb = (float)tb, last = (float)(m - 1);
        k1 = (int)fmaxf(0.0f, floorf(fminf(z1a, z1b) - zs));
        e1 = (int)fminf(last, floorf(fmaxf(z1a, z1b) + zs));
        k2 = (int)fmaxf(0.0f, floorf(fminf(z2a, z2b) - zs));
        e2 = (int)fminf(last, floorf(fmaxf(z2a, z2b) + zs));
        const float s1 = fmaf(8e-6f, fabsf(t1a) + fabsf(t1b), te), s2 = fmaf(8e-6f, fabsf(t2a) + fabsf(t2b), te);
        const bool miss = D + dk < 0.0f;
        if (miss || t1b + s1 < feps || t1a - s1 > ftb) e1 = -1;  // behind the threshold, or farther than a hit found
        if (miss || t2b + s2 < feps || t2a - s2 > ftb) e2 = -1;
        if (!(A > 0.0f) || !(te < 1e30f)) {
            k1 = 0;
            e1 = m - 1;
            e2 = -1;
        }
    }
    bool second = false;
    for (;;) {
        if (k1 > e1 && !second) {
            k1 = k2;
            e1 = e2;
            second = true;
        }
        const bool have = k1 <= e1;
        if (!__any_sync(0xffffffffu, have)) break;
        if (have) {
            const int j = a + k1;
            T t;
            if constexpr (M::kF64)
                t = cylinder_hit<M>(load_rec64(tab64, j, make_float4(0.f, 0.f, 0.f, 0.f)), ray, eps);
            else
                t = cylinder_hit<M>(resident ? tab[j] : load_rec(tab, j), ray, eps);
            if (t < tb || (t == tb && j < bi)) {  // the rings do not come in index order
                tb = t;
                bi = j;
            }
            ++k1;
        }
    }
}

// FP32 looks at a surface whose FP64 test costs fifty times as much (16 clocks of an SM
// an instruction): false only when no point of the ray with eps < t < tb, as the FP64
// test finds them, can be a hit.  sl: rf_bounds.cu, look_slack; NaN anywhere keeps the
// test.  1e6 rays: 48 surfaces 1.33 -> 1.27 ms, 201 (5e5 rays) 2.10 -> 1.85, 400 5.65 ->
// 4.78; what is left is emission (20 surfaces 0.91).
__device__ __forceinline__ bool root_may(const Ray<float> &o, float t0, float t1, float te, float zslack, float eps,
                                         float tb)
{
    const float lo = fminf(t0, t1), hi = fmaxf(t0, t1);
    const float s = fmaf(8e-6f, fabsf(lo) + fabsf(hi), te), zs = fmaf(fabsf(o.cz), s, zslack);
    const float z0 = fmaf(o.cz, lo, o.sz), z1 = fmaf(o.cz, hi, o.sz);
    return !(hi + s < eps || lo - s > tb || fmaxf(z0, z1) + zs < 0.0f || fminf(z0, z1) - zs > 1.0f);
}

__device__ __forceinline__ bool cylinder_may(const HitRec &h, const float4 sl, const Ray<float> &w, float eps, float tb)
{
    const Ray<float> o = xfrm_ray<MFast>(h, w);  // as ring_hits
    const float A = fmaf(o.cx, o.cx, o.cy * o.cy);
    const float B = -fmaf(o.sx, o.cx, o.sy * o.cy);
    const float wz = fmaf(o.sx, o.cy, -o.sy * o.cx);
    const float D = fmaf(-wz, wz, A), dk = A * sl.x;
    if (D + dk < 0.0f) return false;
    const float ra = MFast::rcp(A), te = sl.z * MFast::rsqrt(A);
    if (!(A > 0.0f) || !(te < 1e30f)) return true;
    const float hi = MFast::sqrt(D + dk), lo = MFast::sqrt(fmaxf(D - dk, 0.0f));
    return root_may(o, (B - hi) * ra, (B - lo) * ra, te, sl.y, eps, tb) ||
           root_may(o, (B + lo) * ra, (B + hi) * ra, te, sl.y, eps, tb);
}

// A frustum, for rays out of its band (A then keeps 1e-3 of its terms or more).  D
// by Lagrange's identity is off by 32 u S^2 a, a the squared length of c over the
// quadric's coordinates; B by 8 u S sqrt(a).
__device__ __forceinline__ bool cone_may(const HitRec &h, const float4 sl, const Ray<float> &w, float eps, float tb)
{
    const Ray<float> o = xfrm_ray<MFast>(h, w);
    const float f = h.aux.y - 1.0f, fd = f * o.cz, fs = fmaf(f, o.sz, 1.0f);
    const float a2 = fmaf(o.cx, o.cx, o.cy * o.cy), A = fmaf(-fd, fd, a2), a = fmaf(fd, fd, a2);
    const float B = -fmaf(o.sx, o.cx, fmaf(o.sy, o.cy, -fs * fd));
    const float u = fmaf(o.cx, fs, -o.sx * fd), v = fmaf(o.cy, fs, -o.sy * fd), wz = fmaf(o.sx, o.cy, -o.sy * o.cx);
    const float D = fmaf(u, u, fmaf(v, v, -wz * wz));
    const float dk = fmaf(fabsf(A), sl.x, 0x1p-19f * sl.z * sl.z * a);
    if (D + dk < 0.0f) return false;
    const float ra = MFast::rcp(A), te = 0x1p-19f * sl.z * MFast::sqrt(a) * fabsf(ra);
    if (!(te < 1e30f)) return true;
    const float hi = MFast::sqrt(D + dk), lo = MFast::sqrt(fmaxf(D - dk, 0.0f));
    return root_may(o, (B - hi) * ra, (B - lo) * ra, te, sl.y, eps, tb) ||
           root_may(o, (B + lo) * ra, (B + hi) * ra, te, sl.y, eps, tb);
}

__device__ __forceinline__ bool plane_may(const HitRec &h, int type, const float4 sl, const Ray<float> &w, float eps,
                                          float tb)
{
    const Ray<float> o = xfrm_ray<MFast>(h, w);
    const float rz = MFast::rcp(o.cz), th = -o.sz * rz;
    const float dt = fmaf(sl.y, fabsf(rz), 1e-6f * fabsf(th));
    if (!(dt < 1e30f)) return true;
    const float hx = fmaf(o.cx, th, o.sx), hy = fmaf(o.cy, th, o.sy);
    const float m = 2.0f * fmaf(fabsf(o.cx) + fabsf(o.cy), dt, sl.x);
    if (th + dt < eps || th - dt > tb) return false;
    if (type == RF_RECTANGLE) return !(fabsf(hx) > 1.0f + m || fabsf(hy) > 1.0f + m);
    const float e = MFast::sqrt(fmaf(hx, hx, hy * hy));
    if (type == RF_DISC) return !(e > 1.00001f + m);
    return !(e > fmaf(MFast::sqrt(h.aux.z), 1.00001f, m) || e < fmaf(MFast::sqrt(h.aux.y), 0.99999f, -m));
}

// Nearest hit among the annuli [a, a + m) of a plate: one plane, one radius.
template <class M>
__device__ __forceinline__ void plate_hits(const HitRec &h, const HitRec *tab, bool resident, const double *tab64, int a, int m,
                                           const Ray<typename M::T> &w, typename M::T eps, typename M::T &tb, int &bi)
{
    using T = typename M::T;  // annulus_hit's operations
    Ray<T> o;
    if constexpr (M::kF64)
        o = xfrm_ray<M>(load_rec64(tab64, a, h.aux), w);
    else
        o = xfrm_ray<M>(h, w);
    const T th = -o.sz * M::rcp(o.cz);
    const T hx = o.sx + o.cx * th;
    const T hy = o.sy + o.cy * th;
    const T e = M::fma(hx, hx, hy * hy);
    auto util2 = [&](int k) { return T(resident ? tab[a + k].aux.z : __ldg(&tab[a + k].aux.z)); };
    int base = 0, len = m;  // lowest k with util2_k >= e (uniform trip count)
    while (len > 1) {
        const int half = len >> 1;
        base = util2(base + half - 1) < e ? base + half : base;
        len -= half;
    }
    const T lo = T(resident ? tab[a].aux.y : __ldg(&tab[a].aux.y));
    if (e >= lo && e <= util2(base) && th > eps && th < tb) {
        tb = th;
        bi = a + base;
    }
}

// The mixed-precision arithmetic (emit_mixed, test_mixed with FP64 for an
// ill-conditioned quadric at once) over the mixed tables; used for scenes with
// bounding surfaces, and for those that are nearly all segment stacks.
struct MMixed : MFast {};
template <class M> constexpr bool kIsMixed = false;
template <> constexpr bool kIsMixed<MMixed> = true;

// A bounding surface's test, out of line: one call or two per packet, and a second
// inlined set of the six tests overflows the instruction cache.
template <class M>
static __device__ __noinline__ typename M::T shell_hit(const HitRec *rec, Ray<typename M::T> w, typename M::T eps,
                                                       bool sc)
{
    const HitRec h = *rec;
    const int type = __float_as_int(h.aux.x);
    if constexpr (kIsMixed<M>) {
        bool defer = false;
        float t = hit_mixed(type, h, w, eps, sc, defer);
        if (defer) t = hit_f64(h, w, eps, sc);
        return t;
    } else {
        return hit_any<M>(type, h, w, eps, sc, M::inf());
    }
}

// BV: runBVGPU's walk (RayFactorGPU.cl:530-626) over at most kBatchMaxBV
// bounding surfaces; RESIDENT: the surfaces stay in shared memory (n <=
// kBatchTile; always so with BV); REC: write hit indices instead of tallying;
// COUNT: also the work counters (p.work: tests by type, candidates, packets).
template <class M, int THREADS, bool BV, bool REC, bool RESIDENT, bool COUNT>
__global__ void __launch_bounds__(THREADS, 1) culled_kernel(const TraceParams p)
{
    using T = typename M::T;
    constexpr bool kMixed = kIsMixed<M>;
    constexpr int kPer = kCells / THREADS;                 // buckets per thread of the scan
    constexpr int kMaxG = kChunkDraws / THREADS;           // draws per thread of the largest chunk
    static_assert(THREADS % 32 == 0 && kPer % 4 == 0, "scan shape");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ rf_primitive s_emit;
    __shared__ Emit64 s_emit64;  // FP64
    __shared__ float4 s_frame[3];
    __shared__ float4 s_mframe[kMixed ? kFrameWords : 1];  // mixed: the planar emitter's FP64 frame
    __shared__ int s_wsum[THREADS / 32];
    __shared__ int64_t s_chunk;
    __shared__ int s_next, s_nvalid, s_nlive;

    const int n = p.n, cd = p.chunk_draws;
    const bool hist = !REC && p.use_smem_hist;
    const CulledLayout lay(cd, RESIDENT ? n : 0, hist ? n : 0, BV ? p.nbv : 0);
    int *cnt = reinterpret_cast<int *>(smem_raw + lay.cnt);
    uint16_t *perm = reinterpret_cast<uint16_t *>(smem_raw + lay.perm);
    uint32_t *unif = reinterpret_cast<uint32_t *>(smem_raw + lay.unif);
    HitRec *s_tab = reinterpret_cast<HitRec *>(smem_raw + lay.tab);
    float4 *s_bs = reinterpret_cast<float4 *>(smem_raw + lay.bs);
    HitRec *s_bvtab = reinterpret_cast<HitRec *>(smem_raw + lay.bvtab);
    int4 *s_bvinfo = reinterpret_cast<int4 *>(smem_raw + lay.bvinfo);
    float4 *s_bvbs = reinterpret_cast<float4 *>(smem_raw + lay.bvbs);
    int *s_hist = reinterpret_cast<int *>(smem_raw + lay.hist);
    uint16_t *s_live = reinterpret_cast<uint16_t *>(smem_raw + lay.live);
    const HitRec *tab = RESIDENT ? s_tab : p.tab;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool sc = (p.compat & RF_COMPAT_SPHERE) != 0;
    const T eps = T(p.eps);

    if (RESIDENT) {
        for (int i = tid; i < 4 * n; i += THREADS)
            reinterpret_cast<float4 *>(s_tab)[i] = __ldg(reinterpret_cast<const float4 *>(p.tab) + i);
        if (warp == 0) {
            int m = 0;
            for (int i0 = 0; i0 < n; i0 += 32) {
                const int i = i0 + lane;
                float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < n) {
                    b = __ldg(p.bsph + i);
                    if (kMixed) {  // (the plain arithmetics' tables have w = 0 for a stack's later members)
                        const float4 aux = __ldg(&p.tab[i].aux);
                        if (is_stack(__float_as_int(aux.x)) && (__float_as_int(aux.w) & 0xffff)) b.w = 0.0f;
                    }
                }
                const unsigned on = __ballot_sync(0xffffffffu, b.w != 0.0f);
                if (b.w != 0.0f) {
                    const int k = m + __popc(on & ((1u << lane) - 1u));
                    s_live[k] = (uint16_t)i;
                    s_bs[k] = b;
                }
                m += __popc(on);
            }
            if (lane == 0) s_nlive = m;
        }
        __syncthreads();
    }
    const int nc = RESIDENT ? s_nlive : n;  // candidate positions
    auto surface = [&](int q) { return RESIDENT ? (int)s_live[q] : q; };
    if (BV) {
        for (int i = tid; i < 4 * p.nbv; i += THREADS)
            reinterpret_cast<float4 *>(s_bvtab)[i] = __ldg(reinterpret_cast<const float4 *>(p.bvtab) + i);
        for (int i = tid; i < p.nbv; i += THREADS) {
            int4 info = __ldg(p.bvinfo + i);  // children as positions
            int lo = 0, hi = 0;
            for (int q = 0; q < nc; ++q) {
                lo += s_live[q] < info.y;
                hi += s_live[q] < info.z;
            }
            info.y = lo;
            info.z = hi;
            s_bvinfo[i] = info;
            s_bvbs[i] = __ldg(p.bvsph + i);
        }
    }
    if (hist)
        for (int i = tid; i < n; i += THREADS) s_hist[i] = 0;

    int emitter = -1;
    int skip = -1;       // mixed: a planar emitter, which its own rays cannot hit
    int nref = 0;        // mixed: FP64 evaluations
    uint32_t tcount = 0; // COUNT: lane t < 6 tests of type t, lane 6 candidates, lane 7 packets (this chunk)
    int row_chunks = 0;  // chunks in the shared-memory row since its last flush
    auto flush = [&]() {
        __syncthreads();
        if (hist && emitter >= 0) {
            unsigned long long *row = p.hits + (int64_t)emitter * n;
            for (int i = tid; i < n; i += THREADS) {
                const int v = s_hist[i];
                if (v) {
                    atomicAdd(row + i, (unsigned long long)v);
                    s_hist[i] = 0;
                }
            }
        }
        __syncthreads();
    };

    for (;;) {
        if (tid == 0) s_chunk = (int64_t)atomicAdd(p.queue, 1ull);
        __syncthreads();
        const int64_t c = s_chunk;
        if (c >= p.total_chunks) break;  // block-uniform
        const Segment sg = p.seg[find_segment(p.seg, p.nseg, c)];
        if (sg.emitter != emitter || ++row_chunks >= 32768) {  // (32-bit bins: at most 32768 hits per chunk)
            flush();
            row_chunks = 0;
            if (sg.emitter != emitter) {
                if (tid < (int)(sizeof(rf_primitive) / 4))
                    reinterpret_cast<float *>(&s_emit)[tid] = reinterpret_cast<const float *>(p.emit + sg.emitter)[tid];
                if constexpr (M::kF64) fill_emit64(s_emit64, p.emit[sg.emitter], tid);
                if (tid == 32 % THREADS) quick_frame(p.emit[sg.emitter], s_frame);
                if (kMixed && tid < kFrameWords) s_mframe[tid] = p.frame[(int64_t)sg.emitter * kFrameWords + tid];
                emitter = sg.emitter;
                // (a plate's first member stands for all of it: the others are tested through it)
                if (kMixed)
                    skip = planar(p.emit[emitter].type) && !is_stack(__float_as_int(__ldg(&p.tab[emitter].aux.x))) ? emitter : -1;
            }
        }
        for (int i = tid; i < kCells; i += THREADS) cnt[i] = 0;
        if (tid == 0) s_next = 0;
        __syncthreads();
        const int64_t gid0 = (sg.ray_begin >> 2) + (c - sg.chunk_begin) * (int64_t)cd;
        const uint32_t sid = (p.compat & RF_COMPAT_STREAMS) ? 0u : p.scene_id;

        // 1. uniforms and sort keys; a ray's key waits in perm[] until the sort
#pragma unroll 1
        for (int d = tid; d < cd; d += THREADS) {
            const int64_t gid = gid0 + d;
            uint2 kk = make_uint2(kCells | (kCells << 16), kCells | (kCells << 16));  // no valid ray
            if (gid * 4 + 3 >= sg.ray_begin && gid * 4 < sg.ray_end) {
                const uint4 u = stream_bits(p.compat, p.key1, sid, sg.emitter, gid);
                pack_uniforms(u, unif[d], unif[cd + d], unif[2 * cd + d]);
                const float uf[4] = {u01(u.x), u01(u.y), u01(u.z), u01(u.w)};
                int key4[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    float r[4];
                    rotate_uniforms(uf, v, r);
                    const int64_t rid = gid * 4 + v;
                    const bool valid = rid >= sg.ray_begin && rid < sg.ray_end;
                    key4[v] = valid ? quick_key(s_emit, s_frame, r) : kCells;
                    if (valid) atomicAdd(&cnt[key4[v]], 1);
                }
                kk = make_uint2((uint32_t)key4[0] | ((uint32_t)key4[1] << 16),
                                (uint32_t)key4[2] | ((uint32_t)key4[3] << 16));
            }
            *reinterpret_cast<uint2 *>(&perm[4 * d]) = kk;
        }
        __syncthreads();
        uint2 mykeys[kMaxG];
#pragma unroll
        for (int g = 0; g < kMaxG; ++g)
            if (g * THREADS + tid < cd) mykeys[g] = *reinterpret_cast<const uint2 *>(&perm[4 * (g * THREADS + tid)]);
        // 2. counting sort: exclusive scan of the bucket sizes, kPer per thread
        {
            int sum = 0;
#pragma unroll
            for (int q = 0; q < kPer; ++q) sum += cnt[kPer * tid + q];
            int incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (lane == 31) s_wsum[warp] = incl;
            __syncthreads();
            if (warp == 0) {
                const int x = lane < THREADS / 32 ? s_wsum[lane] : 0;
                int xi = x;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, xi, o);
                    if (lane >= o) xi += t;
                }
                if (lane < THREADS / 32) s_wsum[lane] = xi - x;
                if (lane == 31) s_nvalid = xi;
            }
            __syncthreads();
            int run = s_wsum[warp] + incl - sum;
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const int v = cnt[kPer * tid + q];
                cnt[kPer * tid + q] = run;
                run += v;
            }
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < kMaxG; ++g) {
            const int d = g * THREADS + tid;
            if (d < cd) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const uint32_t w = (v < 2) ? mykeys[g].x : mykeys[g].y;
                    const int key = (int)((w >> (16 * (v & 1))) & 0xffffu);
                    if (key < kCells) perm[atomicAdd(&cnt[key], 1)] = (uint16_t)(4 * d + v);
                }
            }
        }
        __syncthreads();

        // 3. packets of 32 sorted rays
        const int n_valid = s_nvalid;
        const int n_packets = (n_valid + 31) >> 5;
        for (;;) {
            int k = 0;
            if (lane == 0) k = atomicAdd(&s_next, 1);
            k = __shfl_sync(0xffffffffu, k, 0);
            if (k >= n_packets) break;  // warp-uniform
            const int pos = k * 32 + lane;
            const bool valid = pos < n_valid;
            const int l = perm[valid ? pos : k * 32];  // (an idle lane repeats the packet's first ray)
            Ray<T> ray;
            {
                const int d = l >> 2;
                float r[4];
                unpack_rotated(unif[d], unif[cd + d], unif[2 * cd + d], l & 3, r);
                if constexpr (kMixed)
                    ray = emit_mixed(s_emit, s_mframe, r);
                else if constexpr (M::kF64)
                    ray = emit_ray<M>(s_emit64, r);
                else
                    ray = emit_ray<M>(s_emit, r);
            }
            const int nvalid = COUNT ? __popc(__ballot_sync(0xffffffffu, valid)) : 0;  // every lane
            if (COUNT && lane == 7) ++tcount;
            const Ray<float> rf = to_f32(ray);
            const float cc = dot3(rf.cx, rf.cy, rf.cz, rf.cx, rf.cy, rf.cz);
            // a ray the bounds do not speak for: its packet tests everything (mixed: a ray's
            // own sphere checks always speak for it)
            const bool odd = !kMixed && __any_sync(0xffffffffu, !(fabsf(rf.sx) + fabsf(rf.sy) + fabsf(rf.sz) < 1e15f) ||
                                                                    !(cc > 1e-6f && cc < 1e6f));
            const float idd = MFast::rcp(cc);
            Packet pk = bounds_of(rf, idd);
            pk.cull = pk.cull && !odd;

            // candidate words of the 1024 positions from q0 on, lane w holding word w: by
            // sphere (cmask), and frusta in whose band some ray of the packet lies (bmask; a
            // packet too wide for packet_band looks at the band of every frustum)
            unsigned cmask = 0u, bmask = 0u;
            auto candidates = [&](int q0) {
                const int nwords = min(32, (nc - q0 + 31) >> 5);
#pragma unroll 1
                for (int w = 0; w < nwords; ++w) {
                    const int qw = q0 + (w << 5), q = qw + lane;
                    bool cand = false, banded = false;
                    if (q < nc) {
                        const float4 b = RESIDENT ? s_bs[q] : __ldg(p.bsph + q);
                        cand = (RESIDENT || b.w != 0.0f) && (!pk.cull || packet_reaches(pk, b));
                        if (kMixed) cand = cand && surface(q) != skip;
                        if (!kMixed && b.w < 0.0f) banded = !pk.cull || packet_band(p.cquad, surface(q), pk);
                    }
                    const unsigned cm = __ballot_sync(0xffffffffu, cand);
                    unsigned bm = kMixed ? 0u : __ballot_sync(0xffffffffu, banded);
                    for (unsigned todo = bm; todo; todo &= todo - 1) {  // warp-uniform
                        const int b_ = __ffs(todo) - 1;
                        if (!__any_sync(0xffffffffu, band(p.cquad, surface(qw + b_), rf, cc))) bm &= ~(1u << b_);
                    }
                    if (lane == w) {
                        cmask = cm;
                        bmask = bm;
                    }
                }
            };
            // can the lane's ray be hit by the surface at q (a packet's sphere candidate)
            auto gate = [&](int q, T tb) {
                const float4 b = RESIDENT ? s_bs[q] : __ldg(p.bsph + q);
                if constexpr (M::kF64)  // (RF_COMPAT_SPHERE's hits need not lie on the sphere)
                    return odd || reaches_before(rf, cc, idd, b, sc ? M::inf() : tb);
                else
                    return odd || reaches(rf, idd, b);
            };
            // the surface at q, every lane the same.  In mixed arithmetic a hit counts only if
            // the lane's own gate admits the surface: the mixed spheres follow its m, its hits
            // its invm, and a result must not depend on what else the packet tests.  (The gate is
            // formed again for a nearer hit.  Furnace, bounding surfaces, 5e7 rays: 2.48 ms; the
            // first one kept as a flag 2.60; the winner held against it after each search, with
            // a search of the lane's own where it fails, 2.84.)
            auto test = [&](int q, T &tb, int &bi) {
                const int j = surface(q);
                const HitRec h = RESIDENT ? s_tab[j] : load_rec(p.tab, j);
                const int type = __float_as_int(h.aux.x);
                if (COUNT) tcount += lane == (kMixed ? stat_type(type) : type) ? nvalid : 0;
                if constexpr (kMixed) {
                    bool defer = false;
                    int idx;
                    float t = test_mixed<true>(type, h, j, tab, RESIDENT, ray, eps, sc, defer, idx);
                    if (__any_sync(0xffffffffu, defer) && defer) {
                        const float2 q = deferred_f64(tab + j, j, ray, eps, sc);
                        t = q.x;
                        idx = __float_as_int(q.y);
                        nref += valid;
                    }
                    if (t < tb && gate(q, tb)) {
                        tb = t;
                        bi = idx;
                    }
                    return;
                }
                const unsigned m = (unsigned)__float_as_int(h.aux.w);
                if (m) {  // the first of a stack of m surfaces: one search for all of them
                    if (type == RF_ANNULUS)
                        plate_hits<M>(h, tab, RESIDENT, p.tab64, j, (int)m, ray, eps, tb, bi);
                    else
                        ring_hits<M>(tab, RESIDENT, p.tab64, j, (int)m, __ldg(p.cstack + j), ray, rf, eps, odd, tb, bi);
                } else {
                    if constexpr (M::kF64) {  // FP32 first: half the tests find a hit for no ray
                        const float4 sl = __ldg(p.cstack + j);
                        bool may = odd || sl.w == 0.0f;
                        if (!may) {
                            const float feps = __double2float_rd(eps), ftb = __double2float_ru(tb);
                            may = type == RF_FRUSTUM ? band(p.cquad, j, rf, cc) || cone_may(h, sl, rf, feps, ftb)
                                  : type == RF_CYLINDER ? cylinder_may(h, sl, rf, feps, ftb)
                                                        : plane_may(h, type, sl, rf, feps, ftb);
                        }
                        if (!__any_sync(0xffffffffu, may)) return;
                    }
                    T t;
                    if constexpr (M::kF64)
                        t = hit_any<M>(type, load_rec64(p.tab64, j, h.aux), ray, eps, sc, M::inf());
                    else
                        t = hit_any<M>(type, h, ray, eps, sc, M::inf());
                    if (t < tb) {
                        tb = t;
                        bi = j;
                    }
                }
            };
            // nearest hit among the candidates of positions [lo, hi) within the words of q0, in index order
            auto search = [&](int q0, int lo, int hi, T &tb, int &bi) {
#pragma unroll 1
                for (int w = (lo - q0) >> 5; w < 32 && q0 + (w << 5) < hi; ++w) {
                    const int qw = q0 + (w << 5);
                    const unsigned bm = kMixed ? 0u : __shfl_sync(0xffffffffu, bmask, w);
                    unsigned cm = (__shfl_sync(0xffffffffu, cmask, w) | bm) & keep_from(lo - qw);
                    if (hi < qw + 32) cm &= (1u << (hi - qw)) - 1u;
                    while (cm) {  // the same in every lane; two spheres per pass (independent chains)
                        const int ba_ = __ffs(cm) - 1;
                        cm &= cm - 1;
                        const int bb_ = cm ? __ffs(cm) - 1 : ba_;
                        const bool two = cm != 0u;
                        if (COUNT && lane == 6) tcount += two ? 2 : 1;
                        cm &= cm - 1;  // 0 stays 0
                        const bool ma = gate(qw + ba_, tb), mb = gate(qw + bb_, tb);
                        unsigned go = (__any_sync(0xffffffffu, ma) || ((bm >> ba_) & 1u)) ? 1u : 0u;
                        if (two && (__any_sync(0xffffffffu, mb) || ((bm >> bb_) & 1u))) go |= 2u;
                        if constexpr (kMixed) {  // one copy of the tests: two spill (furnace 2.55 -> 2.60 ms)
#pragma unroll 1
                            for (; go; go &= go - 1) test(qw + ((go & 1u) ? ba_ : bb_), tb, bi);
                        } else {  // two: no loop to step (64 surfaces FAST 5.03 -> 4.95 ms)
                            if (go & 1u) test(qw + ba_, tb, bi);
                            if (go & 2u) test(qw + bb_, tb, bi);
                        }
                    }
                }
            };

            int bi = -1;
            if constexpr (BV) {  // RayFactorGPU.cl:580-619, the children's hit found when a lane needs it
                candidates(0);  // n <= kBatchTile
                T tbest = M::inf();
                int bvi = -1, obj = -1, nb = -1;  // nb: children's nearest hit of the current winner bvi
                for (int w = 0; w < p.nbv; ++w) {
                    const bool may = odd || reaches(rf, idd, s_bvbs[w]);
                    if (!__any_sync(0xffffffffu, may)) continue;
                    T t;
                    if constexpr (M::kF64)  // (registers to spare, and no code to share it with)
                        t = hit_any<M>(__float_as_int(s_bvtab[w].aux.x), load_rec64(p.tab64, n + w, s_bvtab[w].aux), ray, eps,
                                       sc, M::inf());
                    else
                        t = shell_hit<M>(s_bvtab + w, ray, eps, sc);
                    const bool nearer = t < tbest && (!kMixed || reaches(rf, idd, s_bvbs[w]));
                    if (!__any_sync(0xffffffffu, nearer)) continue;
                    const int4 info = s_bvinfo[w];
                    T tn = M::inf();
                    int nw = -1;
                    search(0, info.y, info.z, tn, nw);
                    if (nearer) {
                        if (info.x == 1) {  // counts only if a child is hit
                            obj = nw;
                            if (nw != -1) {
                                tbest = t;
                                bvi = w;
                                nb = nw;
                            }
                        } else {
                            tbest = t;
                            bvi = w;
                            nb = nw;
                            if (!(p.compat & RF_COMPAT_BV_STALE)) obj = -1;
                        }
                    }
                }
                bi = (bvi != -1 && obj == -1) ? nb : obj;
            } else {
                T tb = M::inf();
#pragma unroll 1
                for (int q0 = 0; q0 < nc; q0 += 1024) {
                    candidates(q0);
                    search(q0, q0, min(nc, q0 + 1024), tb, bi);
                }
            }
            if (REC) {
                if (valid) p.rec[gid0 * 4 + l - p.rec_base] = bi;
            } else if (hist) {
                warp_tally(s_hist, valid ? bi : -1);
            } else {
                warp_tally_global(p.hits + (int64_t)emitter * n, valid ? bi : -1);
            }
        }
        if (COUNT) {
            if (lane < 8 && tcount) atomicAdd(p.work + lane, (unsigned long long)tcount);
            tcount = 0;
        }
        __syncthreads();
    }
    if (!REC) flush();
    if (kMixed) {
#pragma unroll
        for (int o = 16; o; o >>= 1) nref += __shfl_xor_sync(0xffffffffu, nref, o);
        if (lane == 0 && nref) atomicAdd(p.refined, (unsigned long long)nref);
    }
}

template <class M, bool BV, bool REC, bool RES, bool COUNT = false>
static cudaError_t launch_culled_k(const TraceParams &p, int blocks, cudaStream_t st)
{
    // one block per SM: 1024 threads of 64 registers, in FP64 512 of 128 (two blocks of
    // 512 or four of 256 threads with shorter chunks sort into less similar packets:
    // 64 surfaces EXACT, 1e8 rays, 5.9 / 6.4 / 7.6 ms)
    constexpr int THREADS = M::kF64 ? 512 : 1024;
    auto k = culled_kernel<M, THREADS, BV, REC, RES, COUNT>;
    const int smem = CulledLayout(p.chunk_draws, RES ? p.n : 0, !REC && p.use_smem_hist ? p.n : 0, BV ? p.nbv : 0).bytes;
    // the largest launch's size always: the attribute is the function's on the device, and
    // another thread's context may launch it between this call and ours
    constexpr CulledLayout most(kChunkDraws, RES ? kBatchTile : 0, REC ? 0 : kBatchHist, BV ? kBatchMaxBV : 0);
    static_assert(most.bytes <= 225 * 1024, "shared memory of a block, with 2 KB for the static arrays");
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most.bytes);
    if (e != cudaSuccess) return e;
    const int grid = (int)max((int64_t)1, min((int64_t)blocks, p.total_chunks));
    k<<<grid, THREADS, smem, st>>>(p);
    return cudaGetLastError();
}

static bool culled_fits(const TraceParams &p, bool bv)
{
    return p.chunk_draws > 0 && p.chunk_draws <= kChunkDraws && p.chunk_draws % 4 == 0 &&
           (!bv || (p.n <= kBatchTile && p.nbv > 0 && p.nbv <= kBatchMaxBV)) && (!p.use_smem_hist || p.n <= kBatchHist);
}

template <class M>
cudaError_t launch_culled(const TraceParams &p, bool bv, bool rec, int sms, cudaStream_t st)
{
    if (!culled_fits(p, bv)) return cudaErrorInvalidValue;
    if (bv)
        return rec ? launch_culled_k<M, true, true, true>(p, sms, st) : launch_culled_k<M, true, false, true>(p, sms, st);
    if (p.n <= kBatchTile)
        return rec ? launch_culled_k<M, false, true, true>(p, sms, st) : launch_culled_k<M, false, false, true>(p, sms, st);
    return rec ? launch_culled_k<M, false, true, false>(p, sms, st) : launch_culled_k<M, false, false, false>(p, sms, st);
}

}  // namespace rf
