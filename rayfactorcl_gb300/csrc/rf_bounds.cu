// rf_bounds.cu -- host geometry (FP64): bounding spheres of surfaces under a
// transform, and the tables of the culled kernel (rf_culled.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "rf_internal.h"

namespace rf {
namespace {

struct Ball {
    double c[3];
    double r;
};

double dot(const double a[3], const double b[3]) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }

// Largest length of c0 cos + c1 sin.
double ellipse_radius(const double c0[3], const double c1[3])
{
    const double g0 = dot(c0, c0), g1 = dot(c1, c1), g = dot(c0, c1);
    return std::sqrt(0.5 * (g0 + g1 + std::sqrt((g0 - g1) * (g0 - g1) + 4 * g * g)));
}

// Largest singular value of the 3x3 matrix with columns c0, c1, c2: the largest
// root of the characteristic polynomial of its Gram matrix (Smith, "Eigenvalues
// of a symmetric 3 x 3 matrix", CACM 1961).
double ellipsoid_radius(const double c0[3], const double c1[3], const double c2[3])
{
    const double a = dot(c0, c0), b = dot(c1, c1), c = dot(c2, c2);
    const double d = dot(c0, c1), e = dot(c1, c2), f = dot(c0, c2);
    const double q = (a + b + c) / 3.0;
    const double p1 = d * d + e * e + f * f;
    const double p = std::sqrt(((a - q) * (a - q) + (b - q) * (b - q) + (c - q) * (c - q) + 2 * p1) / 6.0);
    if (!(p > 1e-9 * q)) return std::sqrt(q + 2 * p) * (1.0 + 1e-9);  // a scaled rotation: roots within 2 p of q
    const double A = (a - q) / p, B = (b - q) / p, C = (c - q) / p, D = d / p, E = e / p, F = f / p;
    const double r = 0.5 * (A * (B * C - E * E) - D * (D * C - E * F) + F * (D * E - B * F));
    const double phi = std::acos(std::max(-1.0, std::min(1.0, r))) / 3.0;
    return std::sqrt(std::max(0.0, q + 2 * p * std::cos(phi))) * (1.0 + 1e-9);
}

// A surface's object-space extent: a stack of circles about z, radius r0 at z0 to
// r1 at z1 (discs, annuli, cylinders, frusta), a ball of radius r0 (spheres) or a
// box [-r0, r0] x [-r1, r1] x [z0, z1] (rectangles).
struct Extent {
    enum { kRound, kBall, kBox } shape;
    double r0, r1, z0, z1;
};

Extent extent_of(int type, float util1, float util2)
{
    switch (type) {
    case RF_CYLINDER: return {Extent::kRound, 1.0, 1.0, 0.0, 1.0};
    case RF_FRUSTUM: return {Extent::kRound, 1.0, std::fabs((double)util1), 0.0, 1.0};
    case RF_SPHERE: return {Extent::kBall, 1.0, 1.0, 0.0, 0.0};
    case RF_ANNULUS: {
        const double r = std::sqrt(std::max(0.0, (double)util2));
        return {Extent::kRound, r, r, 0.0, 0.0};
    }
    case RF_DISC: return {Extent::kRound, 1.0, 1.0, 0.0, 0.0};
    default: return {Extent::kBox, 1.0, 1.0, 0.0, 0.0};
    }
}

// Bounding ball of the image of an extent under x -> M x + t (M row-major 3x3).
Ball image_ball(const double M[9], const double t[3], const Extent &x)
{
    const double c0[3] = {M[0], M[3], M[6]}, c1[3] = {M[1], M[4], M[7]}, Z[3] = {M[2], M[5], M[8]};
    Ball b;
    if (x.shape == Extent::kBall) {
        for (int k = 0; k < 3; ++k) b.c[k] = t[k];
        b.r = x.r0 * ellipsoid_radius(c0, c1, Z);
        return b;
    }
    double zc = 0.5 * (x.z0 + x.z1);
    const double L2 = dot(Z, Z), len = x.z1 - x.z0;
    if (x.shape == Extent::kRound) {
        const double rmax = ellipse_radius(c0, c1);
        if (L2 * len > 0.0)  // equal distances to both rims, if that lies between them
            zc = std::max(x.z0, std::min(x.z1, zc + (x.r1 * x.r1 - x.r0 * x.r0) * rmax * rmax / (2 * L2 * len)));
        const double lean = std::hypot(dot(c0, Z), dot(c1, Z));  // 0 when the axis is square to the rims
        b.r = 0.0;
        for (int s = 0; s < 2; ++s) {
            const double r = s ? x.r1 : x.r0, dz = std::fabs((s ? x.z1 : x.z0) - zc);
            b.r = std::max(b.r, std::sqrt(r * r * rmax * rmax + dz * dz * L2 + 2 * dz * r * lean));
        }
    } else {
        b.r = 0.0;
        const double dz = 0.5 * len;
        for (int s = 0; s < 4; ++s) {
            const double px = (s & 1) ? x.r0 : -x.r0, py = (s & 2) ? x.r1 : -x.r1;
            double v[3];
            for (int k = 0; k < 3; ++k) v[k] = c0[k] * px + c1[k] * py + Z[k] * dz;
            b.r = std::max(b.r, std::sqrt(dot(v, v)));  // the other four corners mirror these
        }
    }
    for (int k = 0; k < 3; ++k) b.c[k] = t[k] + Z[k] * zc;
    return b;
}

// M, t of the inverse of a row-major 3x4 world -> object transform; false when
// it is singular.
bool inverse_of(const float *im, double M[9], double t[3])
{
    const double A[9] = {im[0], im[1], im[2], im[4], im[5], im[6], im[8], im[9], im[10]};
    const double c0 = A[4] * A[8] - A[5] * A[7], c1 = A[5] * A[6] - A[3] * A[8], c2 = A[3] * A[7] - A[4] * A[6];
    const double det = A[0] * c0 + A[1] * c1 + A[2] * c2;
    const double i = 1.0 / det;
    if (det == 0.0 || !std::isfinite(i)) return false;
    M[0] = c0 * i;
    M[1] = (A[2] * A[7] - A[1] * A[8]) * i;
    M[2] = (A[1] * A[5] - A[2] * A[4]) * i;
    M[3] = c1 * i;
    M[4] = (A[0] * A[8] - A[2] * A[6]) * i;
    M[5] = (A[2] * A[3] - A[0] * A[5]) * i;
    M[6] = c2 * i;
    M[7] = (A[1] * A[6] - A[0] * A[7]) * i;
    M[8] = (A[0] * A[4] - A[1] * A[3]) * i;
    for (int k = 0; k < 3; ++k) t[k] = -(M[3 * k] * im[3] + M[3 * k + 1] * im[7] + M[3 * k + 2] * im[11]);
    for (int k = 0; k < 9; ++k)
        if (!std::isfinite(M[k])) return false;
    return std::isfinite(t[0] + t[1] + t[2]);
}

// The ball around the points that surface (type, invm) can return as hits to rays
// that start within `from` (and |s| <= smax), in FP32, given its true extent x.
// u = 2^-24; the object-space ray (s, c) as computed is taken as given: it differs
// from the true one by a few u (S + M) at every point up to the hit, S_k bounding
// |s_k| and |c_k t|, M_k the terms s_k is summed from; `lin` covers that.
//
// * Planar: the returned t has |z| and the error of (x, y) within lin.
// * Quadrics, Q(t) = A t^2 - 2 B t + C: the rounding of A, B and C changes Q(t) by
//   at most 12 u S^2 (S^2: squared length over the quadric's coordinates, at the
//   origin or the hit).  The computed root of the rounded A, B, C leaves a residual
//   of at most 28 u S^2 + 16 u B^2 / |A| (the last covers a hardware square root).
//   With a = |c|^2 over the quadric's coordinates, B^2 <= S^2 a.
//   - Cylinder, sphere: |A| = a, so |Q| <= 64 u S^2: the radius grows, z does not.
//   - Cone, where A may vanish: if |A t| >= |B| / 2 then B^2 / |A| <= 4 |A| t^2 <=
//     4 S^2 and again |Q| <= 128 u S^2.  Else the slope of Q at t is at least |B|,
//     so a point with |Q| <= 128 u S^2 lies within dt = 32 u |B| / |A| along the
//     ray, |c_z| dt <= 32 u S a / |A| = m beyond the rims (a with c_z^2 itself added).
//     m is chosen here; rays with |A| below the alpha a that it implies are let
//     through by the band (quad: N of A = c^T N c and the threshold).
Ball hit_ball(const float *im, int type, float util1, Extent x, const Ball &from, double smax, float4 *quad)
{
    constexpr double u = 1.0 / (1 << 24), lin = 32.0 / (1 << 24);
    Ball none{{0, 0, 0}, INFINITY};
    double M[9], t[3];
    if (!inverse_of(im, M, t)) return none;
    const Ball b = image_ball(M, t, x);
    double off[3], L[3], S[3], Mk[3];
    for (int k = 0; k < 3; ++k) off[k] = b.c[k] - from.c[k];
    const double reach = 1.25 * (std::sqrt(dot(off, off)) + from.r + b.r);  // longest ray to a grown hit point
    for (int k = 0; k < 3; ++k) {
        const double r[3] = {im[4 * k], im[4 * k + 1], im[4 * k + 2]};
        L[k] = std::sqrt(dot(r, r));
        // |s_k| <= |L| (distance to the ball) + the object's own extent about its centre
        const double own = k == 2 ? std::max(std::fabs(x.z0), std::fabs(x.z1)) : std::max(x.r0, x.r1);
        S[k] = L[k] * reach + std::max(own, x.shape == Extent::kBall ? x.r0 : 0.0);
        Mk[k] = L[k] * smax + std::fabs((double)im[4 * k + 3]) + own;  // (a stack's members: up to own off)
    }
    Extent g = x;
    double over = 0.0;  // beyond the rims
    if (type == RF_CYLINDER || type == RF_FRUSTUM || type == RF_SPHERE) {
        const double slope = type == RF_FRUSTUM ? (double)util1 - 1.0 : 0.0;
        const double w2 = type == RF_SPHERE ? 1.0 : slope * slope;
        const double fS = std::sqrt(w2) * S[2] + (type == RF_FRUSTUM ? 1.0 : 0.0);  // f(z) = slope z + 1
        const double S2 = S[0] * S[0] + S[1] * S[1] + fS * fS + 1.0;
        const double dQ = 128 * u * S2;
        if (type == RF_FRUSTUM) {
            const double Z = std::sqrt(M[2] * M[2] + M[5] * M[5] + M[8] * M[8]);
            over = std::max(0.1, std::max(0.1 * b.r, 0.01 * reach) / Z);  // the ball grows by about a tenth
            const double alpha = 32 * u * std::sqrt(S2) / over;
            if (!(alpha < 0.25)) return none;
            double n[6];  // xx, yy, zz, yz, xz, xy
            for (int q = 0; q < 6; ++q) {
                const int i = q < 3 ? q : (q == 3 ? 1 : 0), j = q < 3 ? q : (q == 5 ? 1 : 2);
                n[q] = (double)im[i] * im[j] + (double)im[4 + i] * im[4 + j] - w2 * (double)im[8 + i] * im[8 + j];
            }
            const double trace = L[0] * L[0] + L[1] * L[1] + (1.0 + w2) * L[2] * L[2];  // a <= trace |c|^2
            const double norm = std::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2] + 2 * (n[3] * n[3] + n[4] * n[4] + n[5] * n[5]));
            quad[0] = make_float4((float)n[0], (float)n[1], (float)n[2], (float)((alpha + 2e-6) * trace * 1.001));
            quad[1] = make_float4((float)(2 * n[3]), (float)(2 * n[4]), (float)(2 * n[5]), (float)(1.001 * norm));
        }
        g.r0 = std::sqrt(x.r0 * x.r0 + dQ);
        g.r1 = std::sqrt(x.r1 * x.r1 + dQ);
    }
    const double exy = lin * (std::max(S[0], S[1]) + std::max(Mk[0], Mk[1])), ez = lin * (S[2] + Mk[2]);
    if (type == RF_FRUSTUM) {  // the radius where z passes the rims
        const double more = std::fabs((double)util1 - 1.0) * (ez + over);
        g.r0 += more;
        g.r1 += more;
    }
    g.r0 += exy + (x.shape == Extent::kBall ? ez : 0.0);
    g.r1 += exy;
    g.z0 -= ez + over;
    g.z1 += ez + over;
    const Ball grown = image_ball(M, t, g);
    if (!(grown.r - b.r + 16 * lin * (smax + reach) <= 0.2 * (reach / 1.25))) return none;  // (reach assumes that much)
    return grown;
}

// Squared radius for the kernel's FP32 check of a ball: its own rounding, of
// coordinates up to size and distances up to reach.
float check_w(const Ball &b, double size, double reach)
{
    constexpr double u = 1.0 / (1 << 24);
    double c = 0.0;
    for (int k = 0; k < 3; ++k) c = std::max(c, std::fabs(b.c[k]));
    const double r = b.r * (1 + 1e-5) + 16 * u * (size + c + reach);
    const double w = r * r + 64 * u * reach * reach;
    return w < 1e30 ? (float)(w * (1 + 1e-6)) : INFINITY;
}

// What the FP64 kernel's FP32 look at a surface (rf_culled.cuh: cone_may, plane_may,
// ring_hits) must allow for, given the surface's true extent x; w = 0: no look.  The
// FP64 test's own rounding is nothing here; the FP32 ray in object space is off by at
// most 8 u of the terms S_k it is summed from, at every point up to the hit.
// * Planar: x, y = 32 u S of the hit's place and of its height.
// * Quadrics: a true root t leaves |Q(t)| <= x = 128 u S^2 (cones 256) in the FP32
//   coordinates (2 S times their error, and the rounding of A and B); y: z's slack; z:
//   of a cylinder 64 u S, which over sqrt(A) is the rounding of its roots, of a cone S.
float4 look_slack(const float *im, int type, float util1, const Extent &x, const Ball &b, const Ball &from, double smax)
{
    constexpr double u = 1.0 / (1 << 24);
    double off[3], S[3];
    for (int k = 0; k < 3; ++k) off[k] = b.c[k] - from.c[k];
    const double reach = 1.25 * (std::sqrt(dot(off, off)) + from.r + b.r);
    for (int k = 0; k < 3; ++k) {
        const double l[3] = {im[4 * k], im[4 * k + 1], im[4 * k + 2]};
        S[k] = std::sqrt(dot(l, l)) * (smax + reach) + std::fabs((double)im[4 * k + 3]) + std::max(1.0, std::max(x.r0, x.r1));
    }
    const double Sxy = std::max(S[0], S[1]), sz = 128 * u * S[2] + 1e-6;
    double S2 = S[0] * S[0] + S[1] * S[1] + 1.0;
    float4 sl = make_float4(0.f, 0.f, 0.f, 0.f);
    if (type == RF_CYLINDER) {
        sl = make_float4((float)(128 * u * S2), (float)sz, (float)(64 * u * Sxy), 1.f);
    } else if (type == RF_FRUSTUM) {
        const double fS = std::fabs((double)util1 - 1.0) * S[2] + 1.0;
        S2 += fS * fS;
        sl = make_float4((float)(256 * u * S2), (float)sz, (float)std::sqrt(S2), 1.f);
    } else if (type != RF_SPHERE) {  // (a sphere's ball is all there is to look at)
        sl = make_float4((float)(32 * u * Sxy), (float)(32 * u * S[2]), 0.f, 1.f);
    }
    if (!(sl.x < 0.25f) || !(sl.y < 0.25f)) sl.w = 0.f;
    return sl;
}

constexpr double kStackDrift = 0.01;  // of a stack's axis, in radii

// Rings [i, i + m) that one cylinder search finds (ring_hits): cylinders that tile
// a longer one.  Returns m (1: none); x becomes the stack's extent in the first
// ring's frame, sl its slack.  Ring k's object coordinates along a ray, with z
// raised by k, are the first ring's to within dev for every point of the ray up to
// its reach; its test accepts points with |x^2 + y^2 - 1| <= dQ (as in hit_ball),
// so in the first ring's frame |x^2 + y^2 - 1| <= dQ + 2 dev + dev^2 = sl.x, and z
// is known to sl.y.  sl.z: rounding of the search's own FP32 roots.
int ring_stack(const rf_primitive *prims, int n, int i, const std::vector<char> &cut, const Ball &from, double smax,
               Extent &x, float4 &sl)
{
    constexpr double u = 1.0 / (1 << 24);
    const float *a = prims[i].invm;
    double M[9], t[3];
    if (!inverse_of(a, M, t)) return 1;
    auto tiles = [&](int m) {  // do the rings [i, i + m) pass; x and sl if so
        Extent s = {Extent::kRound, 1.0, 1.0, 0.0, (double)m};
        const Ball b = image_ball(M, t, s);
        double d[3];
        for (int k = 0; k < 3; ++k) d[k] = b.c[k] - from.c[k];
        const double reach = 1.25 * (std::sqrt(dot(d, d)) + from.r + b.r);
        double dev[3] = {0, 0, 0}, S[3];
        for (int k = 0; k < 3; ++k) {
            double w = 0.0;
            for (int r = 0; r < m; ++r) {
                const float *g = prims[i + r].invm + 4 * k, *h = a + 4 * k;
                const double e[3] = {(double)g[0] - h[0], (double)g[1] - h[1], (double)g[2] - h[2]};
                const double shift = (double)g[3] - h[3] + (k == 2 ? r : 0);
                dev[k] = std::max(dev[k], std::sqrt(dot(e, e)) * (smax + reach) + std::fabs(shift));
                w = std::max(w, std::fabs((double)g[3]));
            }
            const double l[3] = {a[4 * k], a[4 * k + 1], a[4 * k + 2]};
            S[k] = std::sqrt(dot(l, l)) * (smax + reach) + w + (k == 2 ? m : 1);
        }
        const double dxy = std::hypot(dev[0], dev[1]), S2 = S[0] * S[0] + S[1] * S[1] + 1.0;
        const float4 q = make_float4((float)(128 * u * S2 + 2.5 * dxy), (float)(std::ldexp(S[2], -17) + dev[2] + 1e-6),
                                     (float)(std::ldexp(std::max(S[0], S[1]), -18)), 0.f);
        if (!(dxy < kStackDrift && q.x < 0.1f && q.y < 0.25f)) return false;
        s.r0 = s.r1 = 1.0 + 1.5 * dxy;
        s.z0 -= dev[2];
        s.z1 += dev[2];
        x = s;
        sl = q;
        return true;
    };
    // a first guess; four that fail end it at once: with every ring of a long run (far from the
    // origin, or leaning) going through all the rest, 3000 rings took 107 ms, now 1
    int m = 1;
    for (; i + m < n && m < 4096 && !cut[i + m] && prims[i + m].type == RF_CYLINDER; ++m) {
        const float *b = prims[i + m].invm;
        double d = 0.0;
        for (int k = 0; k < 3; ++k)
            for (int q = 0; q < 3; ++q)
                d = std::max(d, std::fabs((double)b[4 * k + q] - a[4 * k + q]) / (1e-30 + std::fabs(a[4 * k]) +
                                                                              std::fabs(a[4 * k + 1]) + std::fabs(a[4 * k + 2])));
        if (d > 1e-5 || std::fabs((double)b[11] - ((double)a[11] - m)) > 0.02) break;
        if (!(std::hypot((double)b[3] - a[3], (double)b[7] - a[7]) < kStackDrift)) break;
        if (m == 3 && !tiles(4)) return 1;
    }
    const bool four = m >= 4;
    for (; m >= 4; m /= 2)  // (fewer are tested one by one as cheaply)
        if (tiles(m)) return m;
    return four && tiles(4) ? 4 : 1;
}

// The share of an emitter's packets that reach ball b, roughly: rays start within 0.4 of
// the emitter's radius of each other and span 0.15 about their axis (a sort cell), which
// points anywhere.
double packet_share(const Ball &e, const Ball &b)
{
    if (!std::isfinite(b.r)) return 1.0;
    double d[3];
    for (int k = 0; k < 3; ++k) d[k] = b.c[k] - e.c[k];
    const double L = std::sqrt(dot(d, d)), R = b.r + 0.4 * e.r;
    if (!(L > R)) return 1.0;
    const double s = R / L;
    return 0.5 * (1.0 - (std::sqrt(1.0 - s * s) * std::cos(0.15) - s * std::sin(0.15)));
}

}  // namespace

float4 tight_sphere(const rf_primitive &e, float4 box, int rings, float outer2, double reach, bool loose_balls)
{
    if (loose_balls && e.type == RF_SPHERE) return box;
    const double M[9] = {e.m[0], e.m[1], e.m[2], e.m[4], e.m[5], e.m[6], e.m[8], e.m[9], e.m[10]};
    const double t[3] = {e.m[3], e.m[7], e.m[11]};
    Extent x = extent_of(e.type, e.util1, e.type == RF_ANNULUS ? outer2 : e.util2);
    if (rings > 1) x.z1 = rings;
    if (e.type == RF_FRUSTUM) {
        double L2 = 0.0;
        for (int k = 0; k < 3; ++k)
            L2 = std::max(L2, (double)e.invm[4 * k] * e.invm[4 * k] + (double)e.invm[4 * k + 1] * e.invm[4 * k + 1] +
                                  (double)e.invm[4 * k + 2] * e.invm[4 * k + 2]);
        const double over = 16.0 * 4096.0 / (1 << 24) * std::sqrt(3.0 * L2) * reach;
        const double grow = std::fabs((double)e.util1 - 1.0) * over;
        x.z0 -= over;
        x.z1 += over;
        x.r0 += grow;
        x.r1 += grow;
    }
    const Ball b = image_ball(M, t, x);
    const double cn = std::sqrt(dot(b.c, b.c));
    const double r = b.r * (1.0 + 1e-5) + 1e-6 * (cn + b.r) + 1e-7;
    if (!(r < (double)box.w)) return box;
    // the hits follow invm: where it places the surface elsewhere than m does (half of the
    // check's own widening is allowed for), the box's sphere as well as it can
    // (at once where invm m differs from 1 by so little that no point of the surface moves far)
    const double far = 2 * std::max(x.r0, x.r1) + std::max(std::fabs(x.z0), std::fabs(x.z1)) + 1.0;
    double moved = 0.0;
    for (int i = 0; i < 3; ++i) {
        const float *p = e.invm + 4 * i;
        double off = std::fabs(p[0] * t[0] + p[1] * t[1] + p[2] * t[2] + p[3]);
        for (int k = 0; k < 3; ++k)
            off = std::max(off, std::fabs(p[0] * M[k] + p[1] * M[3 + k] + p[2] * M[6 + k] - (i == k ? 1.0 : 0.0)));
        moved += off * std::sqrt(M[i] * M[i] + M[3 + i] * M[3 + i] + M[6 + i] * M[6 + i]);
    }
    const float4 tight = make_float4((float)b.c[0], (float)b.c[1], (float)b.c[2], (float)r);
    if (moved * far <= 0.002 * r) return tight;
    double Mi[9], ti[3], d[3];
    if (!inverse_of(e.invm, Mi, ti)) return box;
    const Ball h = image_ball(Mi, ti, x);
    for (int k = 0; k < 3; ++k) d[k] = h.c[k] - b.c[k];
    return std::sqrt(dot(d, d)) + h.r <= 1.005 * r ? tight : box;
}

bool cull_tables(const rf_primitive *prims, int n, const rf_bounding_volume *bvs, int nbv, bool stacks, HitRec *tab,
                 float4 *sph, float4 *quad, float4 *slack, float4 *bvsph, CullReach *reach)
{
    // where rays start: the emitters' surfaces under m (a frustum's z from its own
    // formula, RayFactorGPU.cl:369-393, which loses digits as util1 nears 1)
    Ball from{{0, 0, 0}, 0.0};
    std::vector<Ball> emit(n);
    for (int i = 0; i < n; ++i) {
        const rf_primitive &p = prims[i];
        const double M[9] = {p.m[0], p.m[1], p.m[2], p.m[4], p.m[5], p.m[6], p.m[8], p.m[9], p.m[10]};
        const double t[3] = {p.m[3], p.m[7], p.m[11]};
        Extent x = extent_of(p.type, p.util1, p.util2);
        if (p.type == RF_FRUSTUM) {
            const double gap = std::fabs((double)p.util1 - 1.0);
            if (gap > 0.0) {
                const double e = 1e-6 / gap;
                x.z0 -= e;
                x.z1 += e;
                x.r0 = x.r1 = std::max(x.r0, x.r1) + 1e-6;
            }
        }
        emit[i] = image_ball(M, t, x);
        for (int k = 0; k < 3; ++k) from.c[k] += emit[i].c[k] / n;
    }
    double smax = 0.0;
    for (int i = 0; i < n; ++i) {
        double d[3];
        for (int k = 0; k < 3; ++k) d[k] = emit[i].c[k] - from.c[k];
        from.r = std::max(from.r, std::sqrt(dot(d, d)) + emit[i].r);
        smax = std::max(smax, std::sqrt(dot(emit[i].c, emit[i].c)) + emit[i].r);
    }
    from.r *= 1.0 + 1e-5;
    smax *= 1.0 + 1e-5;
    if (!std::isfinite(from.r + smax) || smax > 1e12) return false;

    std::vector<char> cut(n + 1, 0);  // stacks stay inside a bounding surface's children
    for (int b = 0; b < nbv; ++b) cut[bvs[b].objStartIndex] = cut[bvs[b].objEndIndex] = 1;

    auto ball_out = [&](const Ball &b, bool frustum) {
        double d[3];
        for (int k = 0; k < 3; ++k) d[k] = b.c[k] - from.c[k];
        const float w = std::isfinite(b.r) ? check_w(b, smax, 1.25 * (std::sqrt(dot(d, d)) + from.r + b.r)) : INFINITY;
        if (std::isinf(w)) return make_float4(0.f, 0.f, 0.f, w);
        return make_float4((float)b.c[0], (float)b.c[1], (float)b.c[2], frustum ? -w : w);
    };

    const int nsample = std::min(n, 16);
    *reach = CullReach{};
    int bounded = 0;
    for (int i = 0; i < n;) {
        const rf_primitive &p = prims[i];
        Extent x = extent_of(p.type, p.util1, p.util2);
        int m = 1;
        float4 sl = make_float4(0.f, 0.f, 0.f, 0.f);
        if (stacks && p.type == RF_CYLINDER) {
            m = ring_stack(prims, n, i, cut, from, smax, x, sl);
        } else if (stacks && p.type == RF_ANNULUS && p.util1 < p.util2) {
            while (i + m < n && m < 4096 && !cut[i + m] && prims[i + m].type == RF_ANNULUS &&
                   std::memcmp(prims[i + m].invm, p.invm, sizeof p.invm) == 0 &&
                   prims[i + m].util1 == prims[i + m - 1].util2 && prims[i + m].util1 < prims[i + m].util2)
                ++m;
            x.r0 = x.r1 = std::sqrt((double)prims[i + m - 1].util2);
        }
        quad[2 * i] = quad[2 * i + 1] = make_float4(0.f, 0.f, 0.f, INFINITY);
        const Ball b = hit_ball(p.invm, p.type, p.util1, x, from, smax, quad + 2 * i);
        const float4 s = ball_out(b, p.type == RF_FRUSTUM);
        double share = 0.0;
        for (int q = 0; q < nsample; ++q) share += packet_share(emit[(size_t)q * n / nsample], b) / nsample;
        if (p.type == RF_CYLINDER || p.type == RF_SPHERE || p.type == RF_FRUSTUM) {
            (p.type == RF_FRUSTUM ? reach->cones : reach->round) += (float)(m > 1 ? 3.0 * share : share);
            reach->ncurved += m;
        } else {
            reach->planar += (float)(m > 1 ? 2.0 * share : share);
            reach->nplanar += m;
        }
        if (std::isfinite(s.w)) bounded += m;
        double M[9], t[3];
        if (m == 1 && std::isfinite(s.w) && inverse_of(p.invm, M, t))
            sl = look_slack(p.invm, p.type, p.util1, x, image_ball(M, t, x), from, smax);
        for (int k = 0; k < m; ++k) {
            sph[i + k] = s;
            slack[i + k] = sl;
            if (k) quad[2 * (i + k)] = quad[2 * (i + k) + 1] = quad[2 * i];
            const int32_t w = m > 1 && k == 0 ? m : 0;
            std::memcpy(&tab[i + k].aux.w, &w, 4);
            if (k) sph[i + k].w = 0.f;  // found through the first
        }
        i += m;
    }
    for (int b = 0; b < nbv; ++b) {
        const rf_bounding_volume &v = bvs[b];
        float4 q[2];
        bvsph[b] = v.type == RF_FRUSTUM ? make_float4(0.f, 0.f, 0.f, INFINITY)
                                        : ball_out(hit_ball(v.invm, v.type, v.util1, extent_of(v.type, v.util1, v.util2),
                                                            from, smax, q), false);
    }
    return 4 * bounded >= 3 * n;  // else too little is left out for the sort to pay
}

}  // namespace rf
