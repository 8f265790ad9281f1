// Jacobi rotation parameters shared by the FP32 SIMT sweep kernels (jacobi.cu,
// gramsweep.cu) and the tensor-core block sweep (tcjacobi.cu).
#pragma once

#include "common.cuh"

namespace mps {

// Columns whose squared norm is below this (theta's is in [1, 4)) count as zero:
// nothing rotates them, and the isometric factor is completed where they stand
// (kZeroSigma).  A pair that rotates has |gamma| of 1e-7 sqrt(a b) or more, and
// make_rot's sigma / conj(gamma), up to 1 / |gamma|, has to stay a float: 1e-31 at
// least.  Columns of an exactly dependent set shrink by 1e-7 a sweep, and were
// followed down to 1e-18 and below, where squares underflow and a cosine comes out
// too large for ever: sweeps up to the cap, or NaN.
constexpr float kZeroNorm2 = 1e-30f;

// Squared cosine of the angle between two columns, |gamma|^2 / (a b).  A pair
// rotates when it exceeds tol^2, and the per-job maximum of the same value
// decides convergence, so a sweep that rotates nothing always ends the job.
// Zero columns give 0; when g2 = |gamma|^2 is below the smallest normal float, the
// cosine is formed from |gamma| and the square roots of the norms with IEEE
// operations instead.
__device__ __forceinline__ float pair_cos2(cf gam, float g2, float a, float b) {
    const float kMinNormal = 1.17549435e-38f;
    if (!(a >= kZeroNorm2 && b >= kZeroNorm2)) return 0.f;
    if (g2 >= kMinNormal) return __fdividef(__fdividef(g2, a), b);
    // |gamma|^2 underflows once the columns are below ~1e-10 in norm (graded
    // columns, as the L factor has from the start): take |gamma| itself.
    const float r = (hypotf(gam.x, gam.y) / sqrtf(a)) / sqrtf(b);
    return r * r;
}

// The rotation of a pair in the form
//   x <- x - (tp x + sigma q),   q <- q + (conj(sigma) x - tp q),
// sigma = s conj(gamma)/|gamma|, tp = 1 - c = s^2 / (1 + c): the complex
// Jacobi rotation [[c, -sigma], [conj(sigma), c]], with c kept implicit as
// 1 - tp (see the file comment).  It equals the rotation with the unit phase
// e = conj(gamma)/|gamma| applied to q (q <- e q + ...) followed by conj(e)
// on the new q, which changes no norm and no orthogonality.  dn = t |gamma|
// is the norm transfer: |x'|^2 = a - dn, |q'|^2 = b + dn.
struct Rot {
    float tp, dn;
    cf sigma;
};

// Rotation parameters for gamma != 0 from quantities scaled by u = 1/(a+b)
// (gamma u is squared, not gamma: no overflow or underflow for a + b >= kZeroNorm2):
// t = sign(b-a) 2|gamma| / (|b-a| + sqrt((b-a)^2 + 4|gamma|^2)),
// c = 1/sqrt(1+t^2) (approximate reciprocal square root refined by one
// Newton step), s = c t.  |sigma|^2 and tp come from the same c^2 t^2, so
// rounding perturbs a rotated column's norm by a few ulps times s^2 only.
__device__ __forceinline__ Rot make_rot(float a, float b, cf gam) {
    const float ab = a + b;
    const float u = ab >= 1e-30f ? __fdividef(1.f, ab) : 1.f / ab;
    const float p = b - a;
    const float ph = p * u;                              // in [-1, 1]
    const float gx = gam.x * u, gy = gam.y * u;
    const float gh = fmaf(gx, gx, gy * gy);              // |gamma|^2 u^2, in (0, 1/4]
    const float h = fmaf(ph, ph, 4.f * gh);
    const float th = __fdividef(2.f, fabsf(ph) + h * rsqrtf(h));   // |t| / (|gamma| u)
    const float t2 = gh * th * th;                       // t^2 <= 1
    const float x = 1.f + t2;
    float c = rsqrtf(x);
    c = c * fmaf(-0.5f * x * c, c, 1.5f);                // Newton step for 1/sqrt(x)
    const float sg = p >= 0.f ? 1.f : -1.f;
    const float k = c * sg * u * th;                     // sigma = k conj(gamma)
    Rot r;
    r.sigma = cmake(k * gam.x, -k * gam.y);
    r.tp = __fdividef(c * c * t2, 1.f + c);
    r.dn = sg * gh * th * ab;                            // = sg |gamma|^2 u th
    return r;
}

__device__ __forceinline__ void apply_rot(const Rot& r, cf& x, cf& q) {
    const float sr = r.sigma.x, si = r.sigma.y, tp = r.tp;
    float nxr = fmaf(-tp, x.x, x.x), nxi = fmaf(-tp, x.y, x.y);
    float nqr = fmaf(-tp, q.x, q.x), nqi = fmaf(-tp, q.y, q.y);
    nxr = fmaf(-sr, q.x, nxr);
    nxi = fmaf(-sr, q.y, nxi);
    nqr = fmaf(sr, x.x, nqr);
    nqi = fmaf(sr, x.y, nqi);
    nxr = fmaf(si, q.y, nxr);
    nxi = fmaf(-si, q.x, nxi);
    nqr = fmaf(si, x.y, nqr);
    nqi = fmaf(-si, x.x, nqi);
    x = cmake(nxr, nxi);
    q = cmake(nqr, nqi);
}

// The same rotation for the two-sided steps on a Gram matrix (one pair a lane,
// where the chain of dependent operations is what a step waits for): tp, sigma
// and dn from one chain of three approximate reciprocals: with u = 1 / sqrt(p^2 + 4
// |gamma|^2), p = b - a, the double angle gives c^2 = (1 + |p| u) / 2 and
// s = |gamma| u / c; tp = s^2 / (1 + c).  Both reciprocal square roots take a
// Newton step, and tp comes from s^2, so a rotation changes no norm by more
// than a few ulps of s^2.  A pair whose squared cosine is not above thr gets the
// identity; in a careful visit (one with tiny columns), pairs whose squares could
// leave FP32's range take the scaled form above.
// Within a visit the norms are carried along, and those of columns that cancel against
// each other (equal columns) end as noise that need not agree with gamma.  Whatever
// they are, the rotation has to be a rotation: a pair whose p^2 + 4 |gamma|^2 is too
// small for u, or whose gamma is too large for its norms (the scaled form would
// square their ratio), stays as it is until its products are formed afresh.
// Squared norms above this (theta's is in [1, 4)) keep every product that a
// rotation is decided on within FP32's normal range.
constexpr float kTinyNorm2 = 1e-9f;
__device__ __forceinline__ float newton_rsqrt(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r * fmaf(-0.5f * x * r, r, 1.5f);
}
// 1 / x to about an ulp (x near 1).
__device__ __forceinline__ float recip(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fmaf(fmaf(-x, r, 1.f), r, r);
}
struct PairRot {
    float tp, sr, si, dn, c, ic;             // (c and 1 / c: 1 where it does not rotate)
    bool rot;
};
__device__ __forceinline__ PairRot pair_rotation(float a, float b, cf gam, float thr,
                                                 bool careful) {
    const float g2 = cabs2(gam), ab = a * b, p = b - a;
    const bool small = careful && (g2 < 1e-30f || ab < 1e-30f);
    PairRot o;
    const float x = fmaf(p, p, 4.f * g2);
    o.rot = !small && g2 > thr * ab && x >= 1e-37f;
    // (a pair of zero columns stays finite)
    const float u = newton_rsqrt(fmaxf(x, 1e-37f));
    const float c2 = fmaf(0.5f * fabsf(p), u, 0.5f);
    const float ic = newton_rsqrt(c2);
    const float k = o.rot ? u * ic : 0.f;                // s = |gamma| k
    const float ks = p >= 0.f ? k : -k;
    float rc;
    o.sr = ks * gam.x;
    o.si = -ks * gam.y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(fmaf(c2, ic, 1.f)));
    o.tp = g2 * k * k * rc;
    o.dn = g2 * ks * ic;                                 // t |gamma| = s |gamma| / c
    o.c = o.rot ? c2 * ic : 1.f;
    o.ic = o.rot ? ic : 1.f;
    if (careful) {
        if (small && fabsf(gam.x) + fabsf(gam.y) <= a + b && pair_cos2(gam, g2, a, b) > thr) {
            const Rot r = make_rot(a, b, gam);
            o.tp = r.tp;
            o.sr = r.sigma.x;
            o.si = r.sigma.y;
            o.dn = r.dn;
            o.c = 1.f - r.tp;
            o.ic = recip(o.c);
            o.rot = true;
        }
    }
    return o;
}
}  // namespace mps
