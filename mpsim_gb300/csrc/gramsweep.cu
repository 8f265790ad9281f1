// One Jacobi sweep per launch with the rotations of a block pair taken from its
// Gram matrix (FP32 SIMT).
//
// Replaces the same computation as the sweep kernel of jacobi.cu (one-sided
// Jacobi in TensorNetwork's split_node_full_svd, mpsim/core.py:1132-1137), and
// keeps its protocol: column blocks, circle-method rounds, items (round, job,
// block pair) claimed from one counter in round-major order, bounded waits on
// the blocks' previous round, visit stamps.  What differs is the visit.  There,
// a warp meets one column after another and each meeting is a chain -- hand-off,
// 512-row dot product, five-step warp reduction, rotation angle, rotation.  Here
// the visit of blocks (I, J) of 8 columns, Y = [X_I X_J] (L x 16 complex) in
// shared memory, is
//   1. Gram:  the 8 x 8 inter-block products X_I^H X_J and the 16 squared
//             norms, fresh from the columns; four lanes cover all 64 products
//             (4 x 4 a lane) for their share of the rows, so a product costs
//             no reduction until the end.  The products within a block
//             (X_I^H X_I, needed to carry X_I^H X_J through the rotations) are
//             kept beside the columns from visit to visit (gblk): rotations
//             update them exactly as they update the columns, and round 0 of
//             every sweep (full visits) computes them afresh.
//   2. Test:  a visit none of whose fresh pairs exceeds the tolerance changes
//             nothing; one with work marks the job as not converged.
//   3. Solve: one warp runs the two-sided Jacobi on G (16 x 16, shared
//             memory), 8 disjoint pairs a step: the 64 inter-block pairs in 8
//             steps, or all 120 in 15 steps on a full visit.  A lane holds one
//             2 x 2 block of G (pair i x pair j, i < j: 28 of them) and lane k
//             computes pair k's rotation, so the angle chain is paid once per
//             8 pairs instead of once per pair.  A pair over kInnerTol2 tol^2
//             rotates: pairs left just above the tolerance by the visit's
//             rounding are settled in it.
//   4. Apply: a warp holds 64 whole rows of Y in registers (16 columns of two
//             rows a lane) and applies each step's 8 rotations as the solver
//             publishes them: no reduction, no exchange, and in lifting form 8
//             FMAs a row and pair instead of 12 (see solve).  The rows of V
//             (jobs that accumulate it) go through the same code.
//
// Each of these is a chain of dependent latencies (a solver step ~330 cycles, a
// claim or a wait for a block ~700 each), so an SM works on several visits at
// once: one CTA per SM whose warps are specialised -- a loader (claims items,
// waits for their blocks, brings the columns in by bulk copies), Gram warps, one
// solver warp per visit slot, and apply warps -- and pass S visit slots round in
// order through mbarriers.  The columns themselves lie in B <= S buffers of their
// own: once the apply warps hold a visit's rows in registers its buffer takes the
// next visit's columns, while the rotations and the write-back go on.
//
// Measured (GB300): 31 theta of 512 x 512, mean sweep 1.16 ms against 1.76 of the
// column-by-column kernel (59% of the issue slots busy at four warps a scheduler;
// L2 27%).  Buffers apart from the slots, against a slot that kept its columns to
// the end: layers of 40 sites chi=420 (one buffer of 1024 rows) 58.3 -> 51.7 ms, of
// 32 qutrits chi=192 14.75 -> 14.3, of 64 sites chi=256 19.8 -> 19.4; slots of up to
// 256 rows have a buffer each (sharing them measured 1-3% slower).  24
// of 256 x 256, 0.26 against 0.29 ms; wide or right-canonical jobs of 200
// columns (V rows included), 0.24 against 0.35 ms.  Variants measured on the
// same case (512 x 512): 16-column blocks with four solver warps, 1.9 ms; three
// CTAs of five warps each doing every step of its own visit, 1.7 ms; packed
// (f32x2) rotations, 1.4 ms (their longer latency shows, and they need the
// parameters twice).
#include <limits.h>

#include "presort.cuh"
#include "rot.cuh"
#include "tc.cuh"
#include "twoq.cuh"

namespace mps {
namespace {

constexpr int GS_BC = kGramBlock;            // columns per block
constexpr int GS_W = 2 * GS_BC;              // columns per visit
constexpr int GS_GST = GS_W + 1;             // row stride of G in shared memory
constexpr int GS_FULL = GS_W - 1;            // steps of a full visit
constexpr int GS_NP = GS_BC * GS_BC;         // products of two blocks
constexpr int GS_NBLK = GS_BC * (GS_BC - 1) / 2;   // 2 x 2 blocks off the diagonal
constexpr int GS_LEAD = 3;                   // step the solver has taken when a warp starts
                                             // (1 where each slot has its own buffer)
constexpr int GS_ACT = 256;                  // jobs left that a CTA keeps in shared memory
constexpr unsigned GS_SUSPEND_NS = 1000;
constexpr float kInnerTol2 = 0.25f;
static_assert(GS_BC == 8 && GS_NBLK <= 32, "one solver warp, one 2 x 2 block a lane");

// One rotation in lifting form, (alpha, beta): x -= alpha y, then y += beta x,
// on columns that carry a scale each (see solve).
typedef float4 Lift;

// A visit slot: what the roles pass on beside the columns.
template <int NG>
struct Slot {
    union {
        Lift prm[GS_FULL * GS_BC];        // rotations of every step
        struct {
            cf part[3][NG][GS_NP];           // Gram partial sums of every warp
            float pnrm[NG][GS_W];            // partial squared norms
        } gr;                                // (summed before the first rotation)
    };
    cf G[GS_W * GS_GST];                     // products of the columns, both triangles
    float dg[GS_W];                          // squared norms
    float scale[GS_W];                       // the columns' scales at the end, less 1
    alignas(8) unsigned mask[GS_W];          // pairs that rotate in a step
    int col[GS_W];                           // physical columns
    int buf;                                 // the column buffer
    int job, I, J, full, L, vrows;
    float tol2;        // the visit (job < 0: no more)
    int time, changedI, changedJ;            // its time, when its blocks last changed
    int* qst;                                // its quiet stamp
    int work;
    // claimed, columns arrived, products formed, rotations decided (or none),
    // rows written, slot free; then one barrier a step
    uint64_t b_info, b_full, b_gram, b_work, b_done, b_free;
    uint64_t b_ring[GS_BC], b_circle[GS_FULL];
};

template <int LW, int B, int S, int NG>
constexpr size_t gs_smem() {
    return B * ((size_t)GS_W * (LW + 2) * sizeof(cf) + sizeof(uint64_t) * 2) + S * sizeof(Slot<NG>) +
           GS_ACT * sizeof(int4);
}

// Column blocks of a job of C columns: an even number, two at least.
__host__ __device__ __forceinline__ int block_count(int C) {
    const int nb = (C + GS_BC - 1) / GS_BC;
    return nb < 2 ? 2 : nb + (nb & 1);
}

// Columns of pair k at step s: of the ring (index k of block I against
// k + s of block J), or of the circle method over all 16.
template <bool FULL>
__device__ __forceinline__ void step_pair(int s, int k, int& p, int& q) {
    if (!FULL) {
        p = k;
        q = GS_BC + ((k + s) & (GS_BC - 1));
    } else {
        p = k + s;
        if (p >= GS_FULL) p -= GS_FULL;
        q = GS_FULL - k + s;
        if (q >= GS_FULL) q -= GS_FULL;
        if (k == 0) q = GS_FULL;
    }
}

// Columns x, y of a row times R = [[1 - tp, conj(sg)], [-sg, 1 - tp]].
__device__ __forceinline__ void rotate(cf& x, cf& y, float tp, float sr, float si) {
    const float xr = x.x, xi = x.y, yr = y.x, yi = y.y;
    x.x = fmaf(-sr, yr, fmaf(si, yi, fmaf(-tp, xr, xr)));
    x.y = fmaf(-sr, yi, fmaf(-si, yr, fmaf(-tp, xi, xi)));
    y.x = fmaf(sr, xr, fmaf(si, xi, fmaf(-tp, yr, yr)));
    y.y = fmaf(sr, xi, fmaf(-si, xr, fmaf(-tp, yi, yi)));
}

// Packed pairs of floats.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// Two rows of a column.
struct Row2 {
    cf a, b;
};
__device__ __forceinline__ Row2 make_row2(float4 v) {
    Row2 x;
    x.a = cmake(v.x, v.y);
    x.b = cmake(v.z, v.w);
    return x;
}
__device__ __forceinline__ float4 from_row2(const Row2& x) {
    return make_float4(x.a.x, x.a.y, x.b.x, x.b.y);
}
// Both steps of a rotation, in place: 8 FMAs a row.
__device__ __forceinline__ void lift(cf& x, cf& y, const Lift& p) {
    x.x = fmaf(-p.x, y.x, fmaf(p.y, y.y, x.x));
    x.y = fmaf(-p.x, y.y, fmaf(-p.y, y.x, x.y));
    y.x = fmaf(p.z, x.x, fmaf(-p.w, x.y, y.x));
    y.y = fmaf(p.z, x.y, fmaf(p.w, x.x, y.y));
}
__device__ __forceinline__ void rotate2(Row2& x, Row2& y, const Lift& p) {
    lift(x.a, y.a, p);
    lift(x.b, y.b, p);
}
// A column times 1 + e.
__device__ __forceinline__ void rescale2(Row2& x, float e) {
    x.a = cmake(fmaf(e, x.a.x, x.a.x), fmaf(e, x.a.y, x.a.y));
    x.b = cmake(fmaf(e, x.b.x, x.b.x), fmaf(e, x.b.y, x.b.y));
}

// The partial products of columns a0.. and b0.. over this lane group's row
// pairs, summed over the warp into part[64] (and the columns' partial norms
// into pn[16]).  A group of four lanes (ti, tj) covers the 8 x 8 product, 4 x 4
// a lane, in an order rotated by 2 tj (rows) and 2 ti (columns): the eight lanes
// of a quarter-warp then read eight different 16-byte banks, and slots 0 and 1
// of the four lanes are together every column once (the norms).
// The two products of a complex pair are packed as (xr yr, xi yi) and
// (xr yi, xi yr), whose sum and difference are its real and imaginary part.
template <int XST, int NG>
__device__ __forceinline__ void gram_partial(const cf* Xs, int a0, int b0, int L, cf* part,
                                             float* pn, int warp, int lane) {
    const int grp = lane >> 2, ti = (lane >> 1) & 1, tj = lane & 1;
    constexpr int CST = XST / 2;              // a column in row pairs
    const float4* x4 = reinterpret_cast<const float4*>(Xs);
    const float4* xa0 = x4 + (a0 + 4 * ti + 2 * tj) * CST;
    const float4* xa2 = x4 + (a0 + 4 * ti + 2 - 2 * tj) * CST;
    const float4* xb0 = x4 + (b0 + 4 * tj + 2 * ti) * CST;
    const float4* xb2 = x4 + (b0 + 4 * tj + 2 - 2 * ti) * CST;
    f2 s1[16], s2[16], na[2], nb[2];
#pragma unroll
    for (int e = 0; e < 16; ++e) s1[e] = s2[e] = 0ull;
    na[0] = na[1] = nb[0] = nb[1] = 0ull;
    const int nrp = (L + 1) >> 1;
#pragma unroll 1
    for (int rp = 8 * warp + grp; rp < nrp; rp += 8 * NG) {
        float4 y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) y[c] = (c < 2 ? xb0 + c * CST : xb2 + (c - 2) * CST)[rp];
        f2 ya[4], yb[4], yas[4], ybs[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            ya[c] = pack2(y[c].x, y[c].y);
            yb[c] = pack2(y[c].z, y[c].w);
            yas[c] = pack2(y[c].y, y[c].x);
            ybs[c] = pack2(y[c].w, y[c].z);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(
                (c < 2 ? xa0 + c * CST : xa2 + (c - 2) * CST) + rp);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s1[4 * c + e] = fma2(x.x, ya[e], s1[4 * c + e]);
                s2[4 * c + e] = fma2(x.x, yas[e], s2[4 * c + e]);
                s1[4 * c + e] = fma2(x.y, yb[e], s1[4 * c + e]);
                s2[4 * c + e] = fma2(x.y, ybs[e], s2[4 * c + e]);
            }
            if (c < 2) na[c] = fma2(x.x, x.x, fma2(x.y, x.y, na[c]));
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) nb[c] = fma2(ya[c], ya[c], fma2(yb[c], yb[c], nb[c]));
    }
    cf acc[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
        float u, v, w, z;
        unpack2(s1[e], u, v);
        unpack2(s2[e], w, z);
        acc[e] = cmake(u + v, w - z);
    }
    __syncwarp();
    // the eight groups' sums by recursive halving: 16 -> 8 -> 4 -> 2 products a lane
    const bool h4 = (lane & 16) != 0, h3 = (lane & 8) != 0, h2 = (lane & 4) != 0;
    cf r8[8], r4[4], r2[2];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const cf send = h4 ? acc[e] : acc[8 + e], mine = h4 ? acc[8 + e] : acc[e];
        r8[e] = cmake(mine.x + __shfl_xor_sync(0xffffffffu, send.x, 16),
                      mine.y + __shfl_xor_sync(0xffffffffu, send.y, 16));
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const cf send = h3 ? r8[e] : r8[4 + e], mine = h3 ? r8[4 + e] : r8[e];
        r4[e] = cmake(mine.x + __shfl_xor_sync(0xffffffffu, send.x, 8),
                      mine.y + __shfl_xor_sync(0xffffffffu, send.y, 8));
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const cf send = h2 ? r4[e] : r4[2 + e], mine = h2 ? r4[2 + e] : r4[e];
        r2[e] = cmake(mine.x + __shfl_xor_sync(0xffffffffu, send.x, 4),
                      mine.y + __shfl_xor_sync(0xffffffffu, send.y, 4));
        // slot 4 c + f with f = 2 h2 + e, c = 2 h4 + h3
        const int c = (h4 ? 2 : 0) + (h3 ? 1 : 0), f = (h2 ? 2 : 0) + e;
        part[(4 * ti + ((c + 2 * tj) & 3)) * GS_BC + 4 * tj + ((f + 2 * ti) & 3)] = r2[e];
    }
    float n[4];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        float u, v;
        unpack2(na[c], u, v);
        n[c] = u + v;
        unpack2(nb[c], u, v);
        n[2 + c] = u + v;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        n[c] += __shfl_xor_sync(0xffffffffu, n[c], 16);
        n[c] += __shfl_xor_sync(0xffffffffu, n[c], 8);
        n[c] += __shfl_xor_sync(0xffffffffu, n[c], 4);
    }
    if (lane < 4 && pn) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            pn[4 * ti + ((c + 2 * tj) & 3)] = n[c];
            pn[GS_BC + 4 * tj + ((c + 2 * ti) & 3)] = n[2 + c];
        }
    }
}

// Whether a pair's squared cosine exceeds tol2 (pair_cos2 without its divisions
// where nothing can leave FP32's range).
__device__ __forceinline__ bool pair_over(cf gam, float a, float b, float tol2) {
    const float g2 = cabs2(gam), ab = a * b;
    if (g2 < 1e-30f || ab < 1e-30f) return pair_cos2(gam, g2, a, b) > tol2;
    return g2 > tol2 * ab;
}

// One step of the circle method for values of the pairs' columns (lane k: those
// of positions k and 15 - k): positions 0..14 move on by one.
__device__ __forceinline__ void circle_move(float& a, float& b, int k) {
    const float a0 = __shfl_sync(0xffffffffu, a, 0);
    const float an = __shfl_sync(0xffffffffu, a, (k + 1) & (GS_BC - 1));
    const float bp = __shfl_sync(0xffffffffu, b, k == 0 ? 0 : k - 1);
    a = k == GS_BC - 1 ? b : an;
    b = k == 1 ? a0 : bp;
}
// Arrives from lane 0, predicated.
__device__ __forceinline__ void lane0_arrive(uint64_t* bar, int lane) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile(
        "{\n\t.reg .b64 st;\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(a), "r"(lane)
        : "memory");
}

// The solver warp: rotations of every step, published one by one.  Lane t < 28
// holds the 2 x 2 block of G of pairs bi < bj, read at the step's start and
// written back (both triangles) at its end; lane l keeps the squared norm of
// position l & 15: pair k is positions k and 8 + k of the ring (the upper half
// moves on by one each step), k and 15 - k of the circle method (positions
// 0..14 move).  A step's own products come by shuffle from the lanes whose
// blocks held them in the step before, so nothing reads the entries a step
// annihilates.
//
// What it publishes for the columns themselves is the same rotation in lifting
// form: with x = d_x X, y = d_y Y, the rotation x' = c x - sigma y,
// y' = conj(sigma) x + c y is X' = X - alpha Y, Y' = Y + beta X' with
// alpha = sigma d_y / (c d_x), beta = conj(sigma) c d_x / d_y, and scales
// d_x' = c d_x, d_y' = d_y / c: two thirds of the arithmetic, in place.  The
// scales start at 1 in every visit and multiply the columns at its end; they
// are kept as e = d - 1 (d_x' - 1 = e - tp d_x), because a c that rounds to 1
// must still undo the growth of t^2 / 2 in the norm (see rot.cuh).
template <bool FULL, int NG>
__device__ __forceinline__ void solve(Slot<NG>& sm, float tol2, bool careful, int lane) {
    cf* G = sm.G;
    int bi = 0, bj = 1;
    {
        int t = lane < GS_NBLK ? lane : 0, row = 0;
        while (t >= GS_BC - 1 - row) {
            t -= GS_BC - 1 - row;
            ++row;
        }
        bi = row;
        bj = row + 1 + t;
    }
    const auto lane_of = [](int i, int j) { return i * (GS_BC - 1) - i * (i - 1) / 2 + j - i - 1; };
    const int k = lane & (GS_BC - 1);
    // the block holding pair k's next product, and which of its entries a
    // lane's block gives (1 pp, 2 pq, 3 qp, 4 qq; all but pq conjugated)
    int src, pick = 0;
    if (!FULL) {
        src = k < GS_BC - 1 ? lane_of(k, k + 1) : lane_of(0, GS_BC - 1);
        pick = bj == bi + 1 ? 2 : 3;
    } else {
        src = k == 0 ? lane_of(0, 1) : k == 1 ? lane_of(0, 2)
              : k == GS_BC - 1 ? lane_of(GS_BC - 2, GS_BC - 1) : lane_of(k - 1, k + 1);
        pick = bi == 0 && bj == 2 ? 1 : (bi == GS_BC - 2 ? 4 : 3);
    }
    constexpr int steps = FULL ? GS_FULL : GS_BC;
    uint64_t* bars = FULL ? sm.b_circle : sm.b_ring;
    // lane k: the squared norms of pair k's columns
    float na = sm.dg[k], nb = sm.dg[FULL ? GS_FULL - k : GS_BC + k];
    float ea = 0.f, eb = 0.f;                 // and their scales, less 1
    cf gam;
    {
        int p, q;
        step_pair<FULL>(0, k, p, q);
        gam = G[p * GS_GST + q];
    }
    const float thr = kInnerTol2 * tol2;
    cf pp = G[bi * GS_GST + bj];
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        int pi, qi, pj, qj;
        step_pair<FULL>(s, bi, pi, qi);
        step_pair<FULL>(s, bj, pj, qj);
        // (of the ring's blocks the first products stay with the lane, and the
        // inter-block ones are kept in the upper triangle only)
        if (FULL) pp = G[pi * GS_GST + pj];
        cf pq = G[pi * GS_GST + qj], qq = G[qi * GS_GST + qj];
        cf qp = FULL ? G[qi * GS_GST + pj] : cconj(G[pj * GS_GST + qi]);
        const float dx = 1.f + ea, dy = 1.f + eb;
        const float yx = dy * recip(dx), xy = dx * recip(dy);
        const PairRot o = pair_rotation(na, nb, gam, thr, careful);
        // what the next step's rotations wait for comes first
        const float tpi = __shfl_sync(0xffffffffu, o.tp, bi), tpj = __shfl_sync(0xffffffffu, o.tp, bj);
        const float sri = __shfl_sync(0xffffffffu, o.sr, bi), srj = __shfl_sync(0xffffffffu, o.sr, bj);
        const float sii = __shfl_sync(0xffffffffu, o.si, bi), sij = __shfl_sync(0xffffffffu, o.si, bj);
        // R_i^H B R_j (the identity where neither pair rotates)
        rotate(pp, pq, tpj, srj, sij);
        rotate(qp, qq, tpj, srj, sij);
        rotate(pp, qp, tpi, sri, -sii);
        rotate(pq, qq, tpi, sri, -sii);
        cf v = pick == 2 ? pq : (pick == 3 ? qp : (pick == 1 ? pp : qq));
        if (pick != 2) v.y = -v.y;
        gam.x = __shfl_sync(0xffffffffu, v.x, src);
        gam.y = __shfl_sync(0xffffffffu, v.y, src);
        // the columns' rotation in lifting form
        const float ka = o.ic * yx, kb = o.c * xy;
        const float4 lf = make_float4(o.sr * ka, o.si * ka, o.sr * kb, -o.si * kb);
        ea = fmaf(-o.tp, dx, ea);
        eb = fmaf(o.tp * o.ic, dy, eb);
        const unsigned mask = __ballot_sync(0xffffffffu, o.rot) & ((1u << GS_BC) - 1u);
        // (lanes that hold the same pair or block store the same values: a
        // branch would cost more)
        sm.prm[s * GS_BC + k] = lf;
        sm.mask[s] = mask;
        int p, q;
        step_pair<FULL>(s, k, p, q);
        if (s == steps - 1) {
            sm.scale[p] = ea;
            sm.scale[q] = eb;
        }
        G[pi * GS_GST + qj] = pq;
        G[pj * GS_GST + qi] = cconj(qp);
        G[qi * GS_GST + qj] = qq;
        G[qj * GS_GST + qi] = cconj(qq);
        if (FULL) {
            G[qi * GS_GST + pj] = qp;
            G[qj * GS_GST + pi] = cconj(pq);
            G[pi * GS_GST + pj] = pp;
            G[pj * GS_GST + pi] = cconj(pp);
        }
        // a rotated pair's own product (else the unused column 16 of row 0)
        G[o.rot ? p * GS_GST + q : GS_W] = cmake(0.f, 0.f);
        if (FULL) G[o.rot ? q * GS_GST + p : GS_W] = cmake(0.f, 0.f);
        __syncwarp();
        lane0_arrive(bars + s, lane);
        // the norms and scales move to the lanes of their next pairs
        na -= o.dn;
        nb += o.dn;
        if (!FULL) {
            nb = __shfl_sync(0xffffffffu, nb, (k + 1) & (GS_BC - 1));
            eb = __shfl_sync(0xffffffffu, eb, (k + 1) & (GS_BC - 1));
        } else {
            circle_move(na, nb, k);
            circle_move(ea, eb, k);
        }
    }
    if (!FULL) G[bi * GS_GST + bj] = pp;
    sm.dg[k] = na;
    sm.dg[FULL ? GS_FULL - k : GS_BC + k] = nb;
    __syncwarp();
}

// A block's progress word (time it last ended a visit, time it last changed):
// read with acquire and written with release order, so that whoever sees a time
// sees the columns and products of every visit up to it.
__device__ __forceinline__ int2 ld_state(const int2* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return make_int2((int)(unsigned)v, (int)(unsigned)(v >> 32));
}
// (lane 0 writes block I's word, lane 1 block J's, behind one fence)
__device__ __forceinline__ void st_states(int2* bst, int I, int J, int t, int cI, int cJ, int lane) {
    if (lane < 2) {
        const unsigned long long v = (unsigned long long)(unsigned)t |
                                     ((unsigned long long)(unsigned)(lane ? cJ : cI) << 32);
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(bst + (lane ? J : I)), "l"(v)
                     : "memory");
    }
}

// Waits for a barrier's phase; gives up for good after limit suspended tries
// (SweepSync::slot_limit; the call then reports an expired wait).
__device__ __forceinline__ void slot_wait(uint64_t* bar, unsigned parity, int limit, bool& expired) {
    if (expired) return;
    int tries = 0;
    while (!mbar_try_wait(bar, parity, GS_SUSPEND_NS)) {
        if (++tries > limit) {
            expired = true;
            break;
        }
    }
    expired = __any_sync(0xffffffffu, expired);
}

// Every step's rotations on this thread's two rows: y[c] are the 16 columns.
// Two steps a pass of the loop (fully unrolled, the kernel's code outgrows the
// instruction cache), after which the visitors move on by two.  The solver's
// steps are waited for two at a time, unless the last one is there already.
template <int NG>
__device__ __forceinline__ void apply_ring(Row2 (&y)[GS_W], Slot<NG>& sm, unsigned parity,
                                           int limit, bool& expired) {
    const bool ready = __all_sync(0xffffffffu, mbar_test_wait(sm.b_ring + GS_BC - 1, parity));
#pragma unroll 1
    for (int s = 0; s < GS_BC; s += 2) {
        if (!ready) slot_wait(sm.b_ring + s + 1, parity, limit, expired);
        const uint2 m = *reinterpret_cast<const uint2*>(sm.mask + s);
        if (m.x) {
#pragma unroll
            for (int k = 0; k < GS_BC; ++k) rotate2(y[k], y[GS_BC + k], sm.prm[s * GS_BC + k]);
        }
        if (m.y) {
#pragma unroll
            for (int k = 0; k < GS_BC; ++k)
                rotate2(y[k], y[GS_BC + ((k + 1) & (GS_BC - 1))], sm.prm[(s + 1) * GS_BC + k]);
        }
        const Row2 t0 = y[GS_BC], t1 = y[GS_BC + 1];
#pragma unroll
        for (int k = GS_BC; k < GS_W - 2; ++k) y[k] = y[k + 2];
        y[GS_W - 2] = t0;
        y[GS_W - 1] = t1;
    }
}

// The same for a full visit: positions 0..7 hold the pairs' first columns,
// 15 - k the second one of pair k; after every step the 15 columns other than
// column 15 (which stays in place) move one pair on (step_pair).  In these
// positions a move is a shift by one of positions 0..14, so that after 15
// steps every column is back at its own.
template <int NG>
__device__ __forceinline__ void apply_full(Row2 (&y)[GS_W], Slot<NG>& sm, unsigned parity,
                                           int limit, bool& expired) {
#pragma unroll 1
    for (int s = 0; s < GS_FULL; ++s) {
        slot_wait(sm.b_circle + s, parity, limit, expired);
        if (sm.mask[s] != 0) {
#pragma unroll
            for (int k = 0; k < GS_BC; ++k) rotate2(y[k], y[GS_FULL - k], sm.prm[s * GS_BC + k]);
        }
        const Row2 t = y[0];
#pragma unroll
        for (int k = 0; k < GS_FULL - 1; ++k) y[k] = y[k + 1];
        y[GS_FULL - 1] = t;
    }
}

// The visit slots in turn: visit n takes slot n mod S, its (n / S)-th use.
template <int S>
struct Turn {
    int slot = 0;
    unsigned use = 0;
    __device__ __forceinline__ unsigned parity() const { return use & 1u; }
    __device__ __forceinline__ void next() {
        if (++slot == S) {
            slot = 0;
            ++use;
        }
    }
};

// Claims items, waits for their blocks and brings their columns in.  Every step
// of this is a round trip to L2 (the visit slots leave L1 next to nothing), so
// the next item is claimed and its job looked up while the present one is on
// its way.
template <int LW, int B, int S, int NG>
__device__ __forceinline__ void loader(const TwoQGeom& g, float tol2, const SweepSync& sync,
                                       int tbase, cf* Xs, uint64_t* b_read, const int4* act,
                                       Slot<NG>* slots, int lane) {
    constexpr int XST = LW + 2;
    const int4 head = __ldcg(g.gact);         // jobs left, their rounds and pairs
    const int rounds = head.y, pairs = head.z, per_round = head.x * pairs;
    const int total = rounds * per_round;
    volatile int* err = sync.error;
    Turn<S> t;
    Turn<B> tb;
    bool expired = false;
    int left = S;                             // end markers to post
    const auto claim = [&]() {                // lane 0: the next item, lane 1: the stop flag
        int v = 0;
        if (lane == 0) v = atomicAdd(sync.next_item, 1);
        else if (lane == 1) v = *err;
        return v;
    };
    // Claiming ahead keeps an item waiting behind the present one: only where a
    // round gives every SM more visits than it has slots (up to 6.5 an SM, 31
    // theta of 512 x 512: 18.8 ms a layer with it down to 3 an SM, 19.35 down to 6;
    // 3.8, 16 of 576 x 576: 14.4 ms with it, 14.1 without).
    const bool ahead = per_round > 4 * (int)gridDim.x;
    int claimed = 0, item = 0;
    int round = 0, round_at = 0, pair = 0;    // the item's round, that round's first item, its pair
    const float per_pair = 1.f / (float)pairs;
    int4 info = make_int4(0, 0, 0, 0);
    bool more = true;
    const auto take = [&]() {
        if (!ahead) claimed = claim();
        item = __shfl_sync(0xffffffffu, claimed, 0);
        more = item < total && __shfl_sync(0xffffffffu, claimed, 1) == 0;
        if (more) {
            // (this warp's items come in order; below 2^24 a round, so the quotient
            // is off by one at most)
            while (item - round_at >= per_round) {
                round_at += per_round;
                ++round;
            }
            int i = (int)((float)(item - round_at) * per_pair);
            pair = item - round_at - i * pairs;
            if (pair < 0) {
                --i;
                pair += pairs;
            } else if (pair >= pairs) {
                ++i;
                pair -= pairs;
            }
            info = i < GS_ACT ? act[i] : __ldcg(g.gact + 1 + i);
        }
    };
    if (ahead) {
        claimed = claim();
        take();
    }
    while (left > 0 && !expired) {
        Slot<NG>& sl = slots[t.slot];
        // ---- the next item that needs a visit -----------------------------
        int j = -1, I = 0, J = 0, L = 0, vrows = 0, r = 0, cI = 0, cJ = 0, col = 0;
        int* qst = nullptr;
        if (!ahead && more) take();
        while (more) {
            const int now_item = item;
            if (ahead) claimed = claim();     // on its way during what follows
            r = round;
            const int p = pair, jj = info.x, C = info.z;
            L = info.y;
            vrows = info.w;
            const int nb = block_count(C);
            const bool active = r < nb - 1 && p < nb / 2;
            bool visit = active;
            if (active) {
                tournament_pair(nb, r, p, I, J);
                int2* bst = g.gstate + (size_t)jj * g.nbmax;
                qst = g.qstamp + (size_t)jj * g.qstride + r * (nb / 2) + p;
                // A block's last finished time and the time it last changed are
                // one 8-byte word, so one read gives both; the quiet stamp of
                // this (round, pair) changes only when this item runs, and the
                // column map not at all during a sweep.
                const int q = *reinterpret_cast<volatile int*>(qst);
                const int c = lane & (GS_W - 1);
                col = __ldcg(g.cmap + (size_t)jj * g.cslot + (c < GS_BC ? I : J - 1) * GS_BC + c);
                // the test hook waits for a round no block ever reaches
                const int need = (sync.stall_test && now_item == per_round) ? INT_MAX : tbase + r;
                int2 st = ld_state(bst + (lane & 1 ? J : I));     // even lanes I, odd lanes J
                int polls = 0;
                bool ok = true;
                while (r > 0 && __any_sync(0xffffffffu, st.x < need)) {
                    ++polls;
                    if (polls > sync.wait_limit && lane == 0) atomicExch(sync.error, 1);
                    // (the stop flag is another round trip: looked at now and then)
                    if (polls > sync.wait_limit ||
                        ((polls & 15) == 0 && __any_sync(0xffffffffu, *err != 0))) {
                        ok = false;
                        break;
                    }
                    st = ld_state(bst + (lane & 1 ? J : I));
                }
                if (!ok) {
                    more = false;
                    break;
                }
                cI = __shfl_sync(0xffffffffu, st.y, 0);
                cJ = __shfl_sync(0xffffffffu, st.y, 1);
                // a visit that last rotated nothing and whose blocks have not
                // changed since would rotate nothing again; no pair lies between
                // a block and padding (round 0 has the pairs inside I)
                const bool quiet = __shfl_sync(0xffffffffu, q >= 0 && q > cI && q > cJ, 0) && nb > 2;
                if (quiet || (r > 0 && J * GS_BC >= C)) {
                    visit = false;
                    st_states(bst, I, J, tbase + r + 1, cI, cJ, lane);
                }
            }
            if (visit) j = jj;
            if (visit && !ahead) break;
            take();
            if (visit) break;
        }
        // ---- into the slot ---------------------------------------------------
        if (t.use > 0) slot_wait(&sl.b_free, t.parity() ^ 1u, sync.slot_limit, expired);
        if (j < 0) {
            --left;
            if (lane == 0) {
                sl.job = -1;
                sl.work = 0;
                mbar_arrive(&sl.b_info);
                mbar_arrive(&sl.b_full);
            }
        } else {
            if (B < S && tb.use > 0) slot_wait(b_read + tb.slot, tb.parity() ^ 1u, sync.slot_limit, expired);
            const uint32_t bytes = (uint32_t)((L + 63) >> 6) * 64u * (uint32_t)sizeof(cf);
            if (lane < GS_W) sl.col[lane] = col;
            if (lane == 0) {
                sl.job = j;
                sl.buf = B < S ? tb.slot : t.slot;
                sl.I = I;
                sl.J = J;
                sl.full = r == 0 ? 1 : 0;
                sl.L = L;
                sl.vrows = vrows;
                sl.tol2 = tol2 > 0.f ? tol2 : default_tol2(slot_rows(L));
                sl.time = tbase + r + 1;
                sl.changedI = cI;
                sl.changedJ = cJ;
                sl.qst = qst;
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sl.b_info);
                tc::mbar_arrive_expect_tx(&sl.b_full, GS_W * bytes);
            }
            __syncwarp();
            // other SMs' (generic) writes of the columns, acquired above, before
            // the bulk copies' (async) reads
            asm volatile("fence.proxy.async;" ::: "memory");
            if (lane < GS_W)
                tc::bulk_g2s(Xs + ((size_t)(B < S ? tb.slot : t.slot) * GS_W + lane) * XST,
                             g.X + (size_t)j * g.lslot * g.cslot + (size_t)col * g.lslot, bytes,
                             &sl.b_full);
            tb.next();
        }
        t.next();
    }
    if (expired && lane == 0) atomicExch(sync.error, 1);
}

template <int LW, int S, int NG>
__device__ __forceinline__ void gram_role(const SweepSync& sync, const cf* Xs, Slot<NG>* slots,
                                          int gw, int lane) {
    constexpr int XST = LW + 2;
    Turn<S> t;
    bool expired = false;
    for (;; t.next()) {
        Slot<NG>& sl = slots[t.slot];
        slot_wait(&sl.b_full, t.parity(), sync.slot_limit, expired);
        if (sl.job < 0 || expired) break;
        const int L = sl.L, np = sl.full ? 3 : 1;
        const cf* X = Xs + (size_t)sl.buf * GS_W * XST;
        // inter-block, then (full visits) the two blocks' own
#pragma unroll 1
        for (int ps = 0; ps < np; ++ps)
            gram_partial<XST, NG>(X, ps == 2 ? GS_BC : 0, ps == 1 ? 0 : GS_BC, L, sl.gr.part[ps][gw],
                                  ps == 0 ? sl.gr.pnrm[gw] : nullptr, gw, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sl.b_gram);
    }
    if (expired && lane == 0) atomicExch(sync.error, 1);
}

template <int LW, int S, int NG>
__device__ __forceinline__ void solver_role(const TwoQGeom& g, const SweepSync& sync, Slot<NG>& sl,
                                            int lane) {
    bool expired = false;
    for (unsigned par = 0u;; par ^= 1u) {
        slot_wait(&sl.b_info, par, sync.slot_limit, expired);
        const int j = sl.job;
        if (j < 0 || expired) {
            if (lane == 0) {
                sl.work = 0;
                mbar_arrive(&sl.b_work);
            }
            break;
        }
        const int I = sl.I, J = sl.J;
        const bool full = sl.full != 0;
        const float tol2 = sl.tol2;
        cf* GI = g.gblk + ((size_t)j * (g.cslot / GS_BC) + I) * GS_NP;
        cf* GJ = g.gblk + ((size_t)j * (g.cslot / GS_BC) + J) * GS_NP;
        if (!full) {
            // the products within the blocks, as the last visits left them
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = lane + 32 * h, a = e / GS_BC, b = e % GS_BC;
                if (a < b) {
                    const cf x = __ldcg(GI + e), y = __ldcg(GJ + e);
                    sl.G[a * GS_GST + b] = x;
                    sl.G[b * GS_GST + a] = cconj(x);
                    sl.G[(GS_BC + a) * GS_GST + GS_BC + b] = y;
                    sl.G[(GS_BC + b) * GS_GST + GS_BC + a] = cconj(y);
                }
            }
        }
        slot_wait(&sl.b_gram, par, sync.slot_limit, expired);
        // the squared norms (lane l: column l & 15), then every product against
        // them as it is summed
        float nrm = 0.f;
#pragma unroll
        for (int w = 0; w < NG; ++w) nrm += sl.gr.pnrm[w][lane & (GS_W - 1)];
        if (lane < GS_W) sl.dg[lane] = nrm;
        const bool careful = __any_sync(0xffffffffu, nrm > 0.f && nrm < kTinyNorm2);
        bool over = false;
#pragma unroll 1
        for (int ps = 0; ps < (full ? 3 : 1); ++ps) {
            const int a0 = ps == 2 ? GS_BC : 0, b0 = ps == 1 ? 0 : GS_BC;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = lane + 32 * h;
                const int a = a0 + e / GS_BC, b = b0 + e % GS_BC;
                cf s = sl.gr.part[ps][0][e];
#pragma unroll
                for (int w = 1; w < NG; ++w) s = cadd(s, sl.gr.part[ps][w][e]);
                const float na = __shfl_sync(0xffffffffu, nrm, a), nb = __shfl_sync(0xffffffffu, nrm, b);
                if (a < b) {
                    sl.G[a * GS_GST + b] = s;
                    sl.G[b * GS_GST + a] = cconj(s);
                    over |= pair_over(s, na, nb, tol2);
                }
            }
        }
        const bool work = __any_sync(0xffffffffu, over);
        if (lane == 0) {
            sl.work = work ? 1 : 0;
            mbar_arrive(&sl.b_work);
            // (the record only says whether the job has a pair over the tolerance)
            if (work) g.offmax[j] = 1.f;
        }
        __syncwarp();
        if (work) {
            if (full) solve<true>(sl, tol2, careful, lane);
            else solve<false>(sl, tol2, careful, lane);
        }
        if (work || full) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int e = lane + 32 * h, a = e / GS_BC, b = e % GS_BC;
                if (a < b) {
                    GI[e] = sl.G[a * GS_GST + b];
                    GJ[e] = sl.G[(GS_BC + a) * GS_GST + GS_BC + b];
                }
            }
        }
        if (lane < GS_W) g.cnrm[(size_t)j * g.cslot + sl.col[lane]] = sl.dg[lane];
        const int now = sl.time, cI = sl.changedI, cJ = sl.changedJ;
        int* qst = sl.qst;
        __syncwarp();
        slot_wait(&sl.b_done, par, sync.slot_limit, expired);
        if (lane == 0) {
            mbar_arrive(&sl.b_free);
            if (!work) *reinterpret_cast<volatile int*>(qst) = now;
        }
        st_states(g.gstate + (size_t)j * g.nbmax, I, J, now, work ? now : cI, work ? now : cJ, lane);
        __syncwarp();
    }
    if (expired && lane == 0) atomicExch(sync.error, 1);
}

template <int LW, int B, int S, int NG, int NA>
__device__ __forceinline__ void apply_role(const TwoQGeom& g, const SweepSync& sync, const cf* Xs,
                                           uint64_t* b_read, Slot<NG>* slots, int aw, int lane) {
    constexpr int XST = LW + 2;
    Turn<S> t;
    bool expired = false;
    unsigned par_ring = 0u, par_circle = 0u;  // step barriers' parities, a bit a slot
    int first = aw;                           // this warp's first task of the visit
    for (;; t.next()) {
        Slot<NG>& sl = slots[t.slot];
        slot_wait(&sl.b_work, t.parity(), sync.slot_limit, expired);
        const int j = sl.job;
        if (j < 0 || expired) break;
        bool reading = B < S;                 // the visit's column buffer
        if (sl.work) {
            // tasks of 64 rows, dealt to the warps in turn across visits: the
            // rows of X, then (where the job accumulates it) those of V
            const bool full = sl.full != 0;
            const unsigned par = ((full ? par_circle : par_ring) >> t.slot) & 1u;
            const int xp = (sl.L + 63) >> 6, np = xp + ((sl.vrows + 63) >> 6);
            cf* X = g.X + (size_t)j * g.lslot * g.cslot;
            cf* V = g.V + (size_t)j * g.cslot * g.cslot;
            const cf* Y = Xs + (size_t)sl.buf * GS_W * XST;
            int q = first;
            // A warp that followed the solver from its first step would spend
            // the whole solve on one visit; from here on it keeps up with the
            // steps as they come.  (Where a buffer waits for it, the warp takes
            // the columns first.)
            uint64_t* start = full ? sl.b_circle + GS_FULL / 2 : sl.b_ring + (B < S ? GS_LEAD : 1);
            if (B == S && q < np) slot_wait(start, par, sync.slot_limit, expired);
#pragma unroll 1
            for (; q < np; q += NA) {
                const bool in_x = q < xp;
                const int r = (in_x ? q : q - xp) * 64 + lane * 2;
                const int ld = in_x ? g.lslot : g.cslot;
                const bool live = r < ld;
                cf* base = (in_x ? X : V) + r;
                Row2 y[GS_W];
                if (in_x) {
#pragma unroll
                    for (int c = 0; c < GS_W; ++c)
                        y[c] = make_row2(*reinterpret_cast<const float4*>(Y + (size_t)c * XST + r));
                } else {
#pragma unroll
                    for (int c = 0; c < GS_W; ++c)
                        y[c] = make_row2(__ldcg(reinterpret_cast<const float4*>(
                            base + (size_t)sl.col[c] * ld - (live ? 0 : r))));
                }
                // this warp's last rows of X are in registers: the buffer's next
                // columns may come
                if (reading && q + NA >= xp) {
                    __syncwarp();
                    lane0_arrive(b_read + sl.buf, lane);
                    reading = false;
                }
                if (B < S && q == first) slot_wait(start, par, sync.slot_limit, expired);
                if (full) apply_full(y, sl, par, sync.slot_limit, expired);
                else apply_ring(y, sl, par, sync.slot_limit, expired);
#pragma unroll
                for (int c = 0; c < GS_W; ++c) rescale2(y[c], sl.scale[c]);
                if (live) {
#pragma unroll
                    for (int c = 0; c < GS_W; ++c)
                        *reinterpret_cast<float4*>(base + (size_t)sl.col[c] * ld) = from_row2(y[c]);
                }
            }
            first = q - np;
            if (full) par_circle ^= 1u << t.slot;
            else par_ring ^= 1u << t.slot;
        }
        __syncwarp();
        if (lane == 0) {
            if (reading) mbar_arrive(b_read + sl.buf);
            mbar_arrive(&sl.b_done);
        }
    }
    if (expired && lane == 0) atomicExch(sync.error, 1);
}

template <int LW, int B, int S, int NG, int NA>
__global__ void __launch_bounds__((NA + NG + S + 1) * 32, 1)
gram_sweep_kernel(TwoQGeom g, float tol2, SweepSync sync, int tbase) {
    extern __shared__ __align__(16) float2 gs_sm[];
    const int left = __ldcg(&g.gact[0].x);
    if (left == 0) return;                    // no job left to sweep here
    cf* Xs = gs_sm;
    int4* act = reinterpret_cast<int4*>(Xs + (size_t)B * GS_W * (LW + 2));
    Slot<NG>* slots = reinterpret_cast<Slot<NG>*>(act + GS_ACT);
    uint64_t* b_read = reinterpret_cast<uint64_t*>(slots + S);       // buffers read out
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < S) {
        Slot<NG>& sl = slots[warp];
        if (lane < GS_BC) mbar_init(sl.b_ring + lane, 1);
        if (lane < GS_FULL) mbar_init(sl.b_circle + lane, 1);
        if (lane == 0) {
            mbar_init(&sl.b_info, 1);
            mbar_init(&sl.b_full, 1);
            mbar_init(&sl.b_gram, NG);
            mbar_init(&sl.b_work, 1);
            mbar_init(&sl.b_done, NA);
            mbar_init(&sl.b_free, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    for (int i = threadIdx.x; i < min(left, GS_ACT); i += blockDim.x) act[i] = __ldcg(g.gact + 1 + i);
    if (B < S && warp == S && lane < B) {
        mbar_init(b_read + lane, NA);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int role = (int)(blockDim.x >> 5) - 1 - warp;          // apply warps first
    if (role == 0) loader<LW, B, S, NG>(g, tol2, sync, tbase, Xs, b_read, act, slots, lane);
    else if (role <= S) solver_role<LW, S, NG>(g, sync, slots[role - 1], lane);
    else if (role <= S + NG) gram_role<LW, S, NG>(sync, Xs, slots, role - 1 - S, lane);
    else apply_role<LW, B, S, NG, NA>(g, sync, Xs, b_read, slots, role - 1 - S - NG, lane);
}

// The jobs left (not done, and not the tensor-core sweeps' in a mixed call), in
// order, into gact; the sweep's counters cleared.  One block -- or, where the
// columns are sorted, a block a job, which ends the job's sweep and sorts it, and
// the last block to finish goes on to the list (a kernel of its own for the sort
// cost a launch, ~5 us, a sweep).
constexpr int GS_BEGIN_T = PRESORT_T;

__global__ void __launch_bounds__(GS_BEGIN_T)
gram_begin_kernel(const mps_2q_job* __restrict__ jobs, TwoQGeom g, int njobs, SweepSync sync,
                  GramBegin b) {
    __shared__ int s_warp[GS_BEGIN_T / 32];
    __shared__ int s_nb, s_flag;
    extern __shared__ __align__(16) float s_sort[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (b.sort_cols) {
        const int j = blockIdx.x;
        if (tid == 0) {
            bool open = !g.done[j];
            if (open && b.end_sweep) {
                if (!(g.offmax[j] > b.tol2)) {
                    g.done[j] = 1;
                    open = false;
                }
                g.offmax[j] = 0.f;
            }
            s_flag = open ? 1 : 0;
        }
        __syncthreads();
        if (s_flag) presort_job(jobs[j], g, j, s_sort, GS_BC, b.tpre);
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            s_flag = atomicAdd(g.counter + 7, 1) == njobs - 1;
            __threadfence();
        }
        __syncthreads();
        if (!s_flag) return;
    }
    if (tid == 0) {
        s_nb = 0;
        g.counter[7] = 0;
        g.counter[0] = 0;
        *sync.next_item = 0;
        if (g.tc_mode) g.counter[4] = g.counter[5] = 0;
        if (b.clear_error) *sync.error = 0;
        // an expired wait also marks every job's status
        else if (b.end_sweep && *sync.error) g.counter[3] = 1;
    }
    __syncthreads();
    int base = 0;
    for (int j0 = 0; j0 < njobs; j0 += GS_BEGIN_T) {
        const int j = j0 + tid;
        bool live = false;
        int4 e = make_int4(j, 0, 0, 0);
        bool open = j < njobs && !__ldcg(g.done + j);
        if (open && b.end_sweep && !b.sort_cols) {
            if (!(g.offmax[j] > b.tol2)) {
                g.done[j] = 1;
                open = false;
            }
            g.offmax[j] = 0.f;
        }
        if (open) {
            const int m = jobs[j].chi_l * g.d, n = jobs[j].chi_r * g.d;
            const int lc = jobs[j].keep_left_canonical;
            e.y = max(m, n);
            e.z = min(m, n);
            e.w = job_tracks_v(m, n, lc) ? e.z : 0;
            live = e.z >= 2 && !(g.tc_mode && tc_job(m, n, lc));
        }
        const unsigned mask = __ballot_sync(0xffffffffu, live);
        if (lane == 0) s_warp[warp] = __popc(mask);
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < GS_BEGIN_T / 32; ++w) {
            if (w < warp) before += s_warp[w];
            all += s_warp[w];
        }
        if (live) {
            g.gact[1 + base + before + __popc(mask & ((1u << lane) - 1u))] = e;
            atomicMax(&s_nb, block_count(e.z));
        }
        base += all;
        __syncthreads();
    }
    if (tid == 0) {
        g.gact[0] = make_int4(base, s_nb - 1, s_nb / 2, 0);
        if (b.record) {
            volatile int* rec = b.record;
            rec[0] = base;
            rec[1] = g.counter[1];
            rec[2] = *sync.error;
            __threadfence_system();
            rec[3] = b.seq;
        }
    }
}

template <int LW, int B, int S, int NG, int NA>
int launch(int njobs, int rounds, int pairs, const TwoQGeom& g, float tol2, const SweepSync& sync,
           int tbase, cudaStream_t s) {
    static KernelSetup ks;
    constexpr size_t smem = gs_smem<LW, B, S, NG>();
    constexpr int threads = (NA + NG + S + 1) * 32;
    static_assert(smem <= 227 * 1024, "visit slots exceed shared memory");
    int dev = 0;
    MPS_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(MPS_ERR_ARG, "device index beyond 63");
    std::call_once(ks.once[dev], [&] {
        int rc = MPS_OK, sms = 0;
        auto kernel = gram_sweep_kernel<LW, B, S, NG, NA>;
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) rc = cuda_fail(e, "setup of gram_sweep_kernel");
        ks.ctas[dev] = sms;
        ks.rc[dev] = rc;
    });
    if (ks.rc[dev] != MPS_OK) return fail(ks.rc[dev], "setup of gram_sweep_kernel failed on this device");
    const int items = njobs * pairs;          // a round's visits
    const int grid = items < ks.ctas[dev] ? items : ks.ctas[dev];
    if (grid <= 0 || rounds <= 0) return MPS_OK;
    gram_sweep_kernel<LW, B, S, NG, NA><<<grid, threads, smem, s>>>(g, tol2, sync, tbase);
    MPS_LAUNCH_CHECK("gram_sweep_kernel");
    return MPS_OK;
}

}  // namespace

int gram_begin_launch(const mps_2q_job* jobs, int njobs, const TwoQGeom& g, const SweepSync& sync,
                      const GramBegin& b, cudaStream_t s) {
    gram_begin_kernel<<<b.sort_cols ? njobs : 1, GS_BEGIN_T, presort_smem(b.sort_cols), s>>>(
        jobs, g, njobs, sync, b);
    MPS_LAUNCH_CHECK("gram_begin_kernel");
    return MPS_OK;
}

int gram_sweep_launch(int njobs, int rounds, int pairs, const TwoQGeom& g,
                      float tol2, const SweepSync& sync, int tbase, cudaStream_t s) {
    if (!g.gblk || !g.gstate || !g.gact || !g.qstamp) return fail(MPS_ERR_ARG, "gram sweeps: no block products");
    // (three Gram warps everywhere: a product's partial sums, and so its rounding,
    // do not depend on the slot a job happens to share with others)
    switch (g.lslot) {
        case 64: return launch<64, 4, 4, 3, 4>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        case 128: return launch<128, 4, 4, 3, 8>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        case 256: return launch<256, 4, 4, 3, 8>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        case 512: return launch<512, 3, 4, 3, 8>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        case 576: return launch<576, 2, 3, 3, 9>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        case 1024: return launch<1024, 1, 2, 3, 10>(njobs, rounds, pairs, g, tol2, sync, tbase, s);
        default: return fail(MPS_ERR_ARG, "gram sweeps: unsupported slot size");
    }
}

}  // namespace mps
