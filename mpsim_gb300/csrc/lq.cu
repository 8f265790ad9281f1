// lq.cu -- LQ preconditioning of the Jacobi SVD (sm_103a).
//
// For a job whose isometric factor is read off the final Jacobi columns (X =
// theta or theta^T, L x C with L >= C, column-major in the X slot: job_tracks_v),
// X is replaced by its L factor before the sweeps:
//
//     X = L Q,  Q (C x C) unitary,  L (L x C) lower trapezoidal.
//
// Q changes neither the singular values nor the left singular vectors, so
// the sweeps' final columns L V = U S still give U, and S V^H is formed as
// U'^H theta from the untouched copy of theta in g.T, exactly as without the
// factorisation.  One-sided Jacobi needs markedly fewer sweeps on the
// triangular factor than on theta itself: the QR-preconditioned Jacobi SVD
// of Drmac and Veselic (SIAM J. Matrix Anal. Appl. 29, 2008), here applied to
// the rows (theta^H = Q^H L^H is the QR factorisation of theta^H).  On the
// chi=256 brickwork layers the sorted ring needs about 10 sweeps on L
// against 14-15 on theta.
//
// Algorithm: blocked Householder reflectors applied from the right.  For
// each panel of LQ_B rows k0 .. k0+kb-1:
//   lq_panel_kernel (one CTA per job), row i's reflector H_i = I - tau_i v_i v_i^H
//     with x_i H_i = beta_i e_i (x_i the row, beta_i real; the textbook complex
//     Householder vector of y = x_i^H: beta = -sign(Re y0) |y|,
//     tau = (beta - y0) / beta, v = (1, y_1.. / (y0 - beta))), applied at once
//     to the panel rows below; and the compact WY factor
//     H_0 ... H_{kb-1} = I - V T V^H (T upper triangular,
//     T[0:i, i] = -tau_i T[0:i, 0:i] V[:, 0:i]^H v_i).
//   lq_trail_kernel (job x 64-row tiles): the rows below the panel,
//     R <- R (I - V T V^H) = R - ((R V) T) V^H.
// V (nc x LQ_B) and T (LQ_B x LQ_B) of the current panel live in the job's
// V slot, which jobs of this kind do not otherwise use before the Gram step
// after the sweeps.
#include <mutex>

#include "gemm.cuh"
#include "twoq.cuh"

namespace mps {
namespace {

constexpr int LQ_B = 32;        // rows per panel
constexpr int LQ_RW = 16;       // warps of the panel kernel, two rows each
constexpr int LQ_T = LQ_RW * 32;
constexpr int LQ_TR = 64;       // rows per trailing-update CTA
constexpr int LQ_TC = 64;       // columns of one step of the trailing update's second product
constexpr int LQ_MIN_C = 64;    // narrower jobs converge in a few cheap sweeps anyway
constexpr int LQ_MAX_C = 768;   // the panel (LQ_B x (C+1)) must fit in shared memory
// V (C x LQ_B) and T (LQ_B x LQ_B, at offset LQ_B * cslot) must fit in the
// job's cslot x cslot V slot; cslot >= C >= LQ_MIN_C
static_assert(LQ_MIN_C * LQ_MIN_C >= LQ_B * (LQ_MIN_C + LQ_B), "V slot too small for V and T");

// Jobs that are factorised, and their shape (X is L x C).
__device__ __forceinline__ bool lq_job(const mps_2q_job& job, int d, int& L, int& C) {
    const int m = job.chi_l * d, n = job.chi_r * d;
    if (job_tracks_v(m, n, job.keep_left_canonical)) return false;
    L = max(m, n);
    C = min(m, n);
    return C >= LQ_MIN_C && C <= LQ_MAX_C;
}

// Shared memory of the panel kernel for nc columns, in units of cf.
__host__ __device__ constexpr int panel_stride(int nc) { return nc | 1; }   // odd: no bank conflicts
__host__ __device__ constexpr size_t panel_elems(int nc, int nt) {
    return (size_t)LQ_B * panel_stride(nc) + 2 * 32 * nt + LQ_B * LQ_B + LQ_B * (LQ_B + 1) +
           4 * LQ_B;
}

// The four values' sums over the warp, in every lane: halves of the warp take two
// of them each, then quarters one each (10 shuffles instead of 20).
__device__ __forceinline__ void warp_sum4(float& v0, float& v1, float& v2, float& v3, int lane) {
    const bool h = lane & 16, q = lane & 8;
    const float a = (h ? v2 : v0) + __shfl_xor_sync(0xffffffffu, h ? v0 : v2, 16);
    const float b = (h ? v3 : v1) + __shfl_xor_sync(0xffffffffu, h ? v1 : v3, 16);
    float c = (q ? b : a) + __shfl_xor_sync(0xffffffffu, q ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    v0 = __shfl_sync(0xffffffffu, c, 0);
    v1 = __shfl_sync(0xffffffffu, c, 8);
    v2 = __shfl_sync(0xffffffffu, c, 16);
    v3 = __shfl_sync(0xffffffffu, c, 24);
}

// A panel of at most 32 NT columns.  Its 32 reflectors are a serial chain, so the
// kernel is bound by a reflector's latency and, beyond ~300 columns, by the FMAs of
// one SM.  The rows therefore stay in registers (warp w: rows w and w + 16, lane l:
// columns l, l + 32, ...) and only the pivot row's u_i = v_i (y0 - beta) goes through
// shared memory, conjugated; one barrier a reflector.  Every row r takes the same
// product a = x_r u_i: a row below becomes x_r - tau a conj(u_i) / |y0 - beta|^2, and
// for a row above it is (V^H V)[r][i] up to conj(inv_r) inv_i, which T needs.  The
// warp of the next pivot row computes its scalars, that of the last one T's column.
// Mean panel of a 512-column job: 38 us (before, with the rows in shared memory, a
// warp a row, and T afterwards: 94 us).  Beyond 512 columns a part of the rows spills
// (60 bytes a thread in the kernel for 640, 444 in that for 768); it is still ahead: calls of
// 16 jobs of 768 columns 52 ms with the factorised start, 57 without it, 104 with it before.
template <int NT>
__global__ void __launch_bounds__(LQ_T, 1)
lq_panel_kernel(const mps_2q_job* __restrict__ jobs, TwoQGeom g, int k0) {
    extern __shared__ float2 lq_sm[];
    const int j = blockIdx.x;
    int L, C;
    if (!lq_job(jobs[j], g.d, L, C) || k0 >= C) return;
    const int kb = min(LQ_B, C - k0), nc = C - k0, ps = panel_stride(nc);
    cf* P = lq_sm;                              // [kb][ps]: the panel, row-major
    cf* xs = P + (size_t)LQ_B * ps;             // [2][32 NT]: conj(u) of the pivot row
    cf* zz = xs + 2 * 32 * NT;                  // [LQ_B][LQ_B]: (V^H V)[a][b], a < b (0 else)
    cf* Ts = zz + LQ_B * LQ_B;                  // [LQ_B][LQ_B + 1]: T, row-major
    cf* tau = Ts + LQ_B * (LQ_B + 1);           // [LQ_B]
    cf* invs = tau + LQ_B;                      // [LQ_B]: 1 / (y0 - beta)
    cf* taun = invs + LQ_B;                     // [LQ_B]: tau / |y0 - beta|^2
    float* betas = reinterpret_cast<float*>(taun + LQ_B);   // [LQ_B]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cf* X = g.X + (size_t)j * g.lslot * g.cslot;

    const uint32_t pbase = (uint32_t)__cvta_generic_to_shared(P);
    for (int c = warp; c < nc; c += LQ_RW)
        if (lane < kb)
            copy8_async(pbase + (uint32_t)(lane * ps + c) * 8u,
                        X + (size_t)(k0 + c) * g.lslot + k0 + lane, 8u);
    for (int e = tid; e < LQ_B * (2 * LQ_B + 1); e += LQ_T) zz[e] = cmake(0.f, 0.f);   // and T
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // Row i of this warp's two: its scalars and u.
    cf z[2][NT];
    const auto publish = [&](int i) {
        const int h = i / LQ_RW;
        float s = 0.f;
        cf* x = xs + (i & 1) * 32 * NT + lane;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            cf v = h ? z[1][t] : z[0][t];
            if (t == 0 && lane <= i) v = cmake(0.f, 0.f);
            s += cabs2(v);
            x[32 * t] = v;
        }
        s = warp_sum(s);
        const cf y = h ? z[1][0] : z[0][0];
        if (lane == i) {
            const cf y0 = cconj(y);
            const float n2 = cabs2(y0) + s;
            cf t = cmake(0.f, 0.f), inv = cmake(0.f, 0.f), tn = cmake(0.f, 0.f);
            float beta = y0.x;
            // (a row whose square is no normal number has no reflector: 1 / |y0 - beta|^2
            // would overflow)
            if ((s > 0.f || y0.y != 0.f) && !(n2 < 4.8e-38f)) {
                const float nrm = sqrtf(n2);
                beta = y0.x >= 0.f ? -nrm : nrm;
                const cf u = cmake(y0.x - beta, y0.y);
                const float rb = 1.f / beta, q = 1.f / cabs2(u);
                t = cmake(-u.x * rb, -u.y * rb);
                inv = cmake(u.x * q, -u.y * q);
                tn = cscale(t, q);
                *x = cconj(u);
            }
            tau[i] = t;
            invs[i] = inv;
            taun[i] = tn;
            betas[i] = beta;
        }
    };
    // T[a][b] for all a, from column b of V^H V
    const auto t_column = [&](int b) {
        cf s0 = cmake(0.f, 0.f), s1 = cmake(0.f, 0.f);
        for (int q0 = 0; q0 < b; q0 += 8) {
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                cfma(s0, Ts[lane * (LQ_B + 1) + q0 + q], zz[(q0 + q) * LQ_B + b]);
                cfma(s1, Ts[lane * (LQ_B + 1) + q0 + q + 1], zz[(q0 + q + 1) * LQ_B + b]);
            }
        }
        const cf tb = tau[b], ts = cmul(tb, cadd(s0, s1));
        __syncwarp();
        if (lane <= b) Ts[lane * (LQ_B + 1) + b] = lane == b ? tb : cmake(-ts.x, -ts.y);
        __syncwarp();
    };

#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = warp + LQ_RW * h;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int c = lane + 32 * t;
            z[h][t] = r < kb && c < nc ? P[r * ps + c] : cmake(0.f, 0.f);
        }
    }
    if (warp == 0) publish(0);
    for (int i = 0; i < kb; ++i) {
        __syncthreads();
        const cf* x = xs + (i & 1) * 32 * NT + lane;
        cf a0 = cmake(0.f, 0.f), a1 = cmake(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const cf xv = x[32 * t];
            cfma_conj(a0, xv, z[0][t]);
            cfma_conj(a1, xv, z[1][t]);
        }
        warp_sum4(a0.x, a0.y, a1.x, a1.y, lane);
        const cf mt = cmake(-taun[i].x, -taun[i].y);
        const cf w0 = cmul(mt, a0), w1 = cmul(mt, a1);
        if (warp > i) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const cf xv = x[32 * t];
                cfma(z[0][t], w0, xv);
                cfma(z[1][t], w1, xv);
            }
        } else if (warp + LQ_RW > i) {
#pragma unroll
            for (int t = 0; t < NT; ++t) cfma(z[1][t], w1, x[32 * t]);
        }
        if (i + 1 < kb && warp == (i + 1) % LQ_RW) publish(i + 1);
        if (lane == 0) {
            const cf inv = invs[i];
            if (warp < i) zz[warp * LQ_B + i] = cmul(cmul(cconj(invs[warp]), inv), a0);
            if (warp + LQ_RW < i)
                zz[(warp + LQ_RW) * LQ_B + i] = cmul(cmul(cconj(invs[warp + LQ_RW]), inv), a1);
        }
        if (i > 0 && warp == (i - 1) % LQ_RW) t_column(i - 1);
    }
    __syncthreads();
    // the rows to shared memory: L left of the diagonal, beta on it, v right of it
    if (warp == (kb - 1) % LQ_RW) t_column(kb - 1);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = warp + LQ_RW * h;
        if (r >= kb) continue;
        const cf inv = invs[r];
        const float beta = betas[r];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int c = lane + 32 * t;
            cf v = z[h][t];
            if (t > 0 || lane > r) v = cmul(cconj(v), inv);
            else if (lane == r) v = cmake(beta, 0.f);
            if (c < nc) P[r * ps + c] = v;
        }
    }
    __syncthreads();

    // V (nc x LQ_B, zero beyond kb) and T (LQ_B x LQ_B) to the V slot
    cf* Vg = g.V + (size_t)j * g.cslot * g.cslot;
    cf* Tg = Vg + (size_t)LQ_B * g.cslot;
    for (int e = tid; e < nc * LQ_B; e += LQ_T) {
        const int c = e / LQ_B, b = e % LQ_B;
        cf v = cmake(0.f, 0.f);
        if (b < kb) v = c < b ? cmake(0.f, 0.f) : (c == b ? cmake(1.f, 0.f) : P[b * ps + c]);
        Vg[e] = v;
    }
    for (int e = tid; e < LQ_B * LQ_B; e += LQ_T) {
        const int a = e / LQ_B, b = e % LQ_B;
        Tg[e] = a < kb && b < kb && b >= a ? Ts[a * (LQ_B + 1) + b] : cmake(0.f, 0.f);
    }
    // the panel's rows of L: zero right of the diagonal
    for (int c = warp; c < nc; c += LQ_RW)
        if (lane < kb)
            X[(size_t)(k0 + c) * g.lslot + k0 + lane] =
                c <= lane ? P[lane * ps + c] : cmake(0.f, 0.f);
}

// Rows k0+kb .. L-1 of the job, 64 per CTA: W = R V by the shared GEMM tile, W T
// in shared memory, then R - (W T) V^H in steps of 64 columns with V's rows and R's
// entries fetched a step ahead.  Both products read shared memory in 8 wavefronts
// for 64 FMAs a thread, so the FP32 pipes bound it: mean launch of 63 jobs of 512
// columns 47 us (73 us before, when the second product read 3 wavefronts for
// every 4 FMAs).
struct TrailSmem {
    using Tile = GemmTile<LQ_TR, LQ_B, 2>;
    static constexpr int VST = LQ_TC + 1;
    union {
        cf ab[Tile::ST * Tile::BUF];            // the first product's chunks
        cf vt[2][LQ_B][VST];                    // a step's 64 rows of V, transposed
    };
    cf w[LQ_B][LQ_TR + 1];                      // W, then W T
    cf t[LQ_B][LQ_B];
};

__global__ void __launch_bounds__(256, 2)
lq_trail_kernel(const mps_2q_job* __restrict__ jobs, TwoQGeom g, int k0) {
    extern __shared__ float2 lq_sm[];
    TrailSmem& sm = *reinterpret_cast<TrailSmem*>(lq_sm);
    const int j = blockIdx.y;
    int L, C;
    if (!lq_job(jobs[j], g.d, L, C) || k0 >= C) return;
    const int kb = min(LQ_B, C - k0), nc = C - k0;
    const int row0 = k0 + kb + blockIdx.x * LQ_TR;
    if (row0 >= L) return;
    const int tid = threadIdx.x, rows = L - row0;
    cf* R = g.X + (size_t)j * g.lslot * g.cslot + (size_t)k0 * g.lslot + row0;
    const cf* Vg = g.V + (size_t)j * g.cslot * g.cslot;
    const cf* Tg = Vg + (size_t)LQ_B * g.cslot;

    for (int e = tid; e < LQ_B * LQ_B; e += 256) (&sm.t[0][0])[e] = Tg[e];
    const GemmArgs a{min(rows, LQ_TR), LQ_B, nc, R, 1, g.lslot, 0, Vg, LQ_B, 1, 0, nullptr, 0, 0};
    for (int e = tid; e < LQ_B * (LQ_TR + 1); e += 256) (&sm.w[0][0])[e] = cmake(0.f, 0.f);
    __syncthreads();
    TrailSmem::Tile::run<false, false>(a, 0, 0, nullptr, sm.ab,
                                       [&](int r, int b, cf v) { sm.w[b][r] = v; });
    __syncthreads();
    const uint32_t vbase = (uint32_t)__cvta_generic_to_shared(&sm.vt[0][0][0]);
    const auto fetch_v = [&](int c0) {
        const uint32_t off = vbase + (uint32_t)((c0 / LQ_TC) & 1) * (LQ_B * TrailSmem::VST * 8);
#pragma unroll
        for (int q = 0; q < LQ_TC * LQ_B / 256; ++q) {
            const int e = tid + 256 * q, c = e / LQ_B, b = e % LQ_B;
            const bool in = c0 + c < nc;
            copy8_async(off + (uint32_t)(b * TrailSmem::VST + c) * 8u,
                        in ? Vg + (size_t)(c0 + c) * LQ_B + b : Vg, in ? 8u : 0u);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch_v(0);
    // W <- W T (T upper triangular): row r, columns q, q + 4, ...
    {
        const int r = tid & (LQ_TR - 1), q = tid / LQ_TR;
        cf w[LQ_B / 4];
#pragma unroll
        for (int e = 0; e < LQ_B / 4; ++e) w[e] = cmake(0.f, 0.f);
#pragma unroll 4
        for (int i = 0; i < LQ_B; ++i) {
            const cf x = sm.w[i][r];
#pragma unroll
            for (int e = 0; e < LQ_B / 4; ++e) cfma(w[e], x, sm.t[i][q + 4 * e]);
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < LQ_B / 4; ++e) sm.w[q + 4 * e][r] = cmake(-w[e].x, -w[e].y);
    }
    // this thread: rows tx + 16 i, columns ty + 16 j of a step
    const int tx = tid & 15, ty = tid >> 4;
    cf zr[4][4];
    const auto fetch_r = [&](int c0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = tx + 16 * i, c = c0 + ty + 16 * q;
                zr[i][q] = r < rows && c < nc ? R[(size_t)c * g.lslot + r] : cmake(0.f, 0.f);
            }
    };
    fetch_r(0);
    for (int c0 = 0; c0 < nc; c0 += LQ_TC) {
        cf acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][q] = zr[i][q];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (c0 + LQ_TC < nc) {
            fetch_v(c0 + LQ_TC);
            fetch_r(c0 + LQ_TC);
        }
        const cf (*vt)[TrailSmem::VST] = sm.vt[(c0 / LQ_TC) & 1];
#pragma unroll 8
        for (int b = 0; b < LQ_B; ++b) {
            cf wv[4], vv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) wv[i] = sm.w[b][tx + 16 * i];
#pragma unroll
            for (int q = 0; q < 4; ++q) vv[q] = vt[b][ty + 16 * q];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) cfma_conj(acc[i][q], vv[q], wv[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = tx + 16 * i, c = c0 + ty + 16 * q;
                if (r < rows && c < nc) R[(size_t)c * g.lslot + r] = acc[i][q];
            }
    }
}

// Column norms of the factorised jobs for the first sweep's sort.
__global__ void __launch_bounds__(256) lq_norm_kernel(const mps_2q_job* __restrict__ jobs,
                                                      TwoQGeom g) {
    const int j = blockIdx.y;
    int L, C;
    if (!lq_job(jobs[j], g.d, L, C)) return;
    const int lane = threadIdx.x & 31;
    const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (c >= C) return;
    const cf* col = g.X + (size_t)j * g.lslot * g.cslot + (size_t)c * g.lslot;
    float acc = 0.f;
    for (int r = lane; r < L; r += 32) acc += cabs2(col[r]);
    acc = warp_sum(acc);
    if (lane == 0) g.cnrm[(size_t)j * g.cslot + c] = acc;
}

}  // namespace

int lq_precondition(const mps_2q_job* jobs, int njobs, int max_m, int max_n, const TwoQGeom& g,
                    cudaStream_t s) {
    const int cmax = min(min(max_m, max_n), LQ_MAX_C);
    if (cmax < LQ_MIN_C) return MPS_OK;
    // the shared-memory opt-in is per device: set it once on every device used
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr[kMaxDevices];
    // kernels for panels of up to 64, 128, 256, 384, ... columns
    static constexpr int kNt[] = {2, 4, 8, 12, 16, 20, 24};
    static void (*const kPanel[])(const mps_2q_job*, TwoQGeom, int) = {
        lq_panel_kernel<2>,  lq_panel_kernel<4>,  lq_panel_kernel<8>, lq_panel_kernel<12>,
        lq_panel_kernel<16>, lq_panel_kernel<20>, lq_panel_kernel<24>};
    int dev = 0;
    MPS_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(MPS_ERR_ARG, "lq_precondition: device index beyond 63");
    std::call_once(once[dev], [&] {
        attr[dev] = cudaSuccess;
        for (int q = 0; q < 7 && attr[dev] == cudaSuccess; ++q)
            attr[dev] = cudaFuncSetAttribute(kPanel[q], cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(panel_elems(32 * kNt[q], kNt[q]) * sizeof(cf)));
        if (attr[dev] == cudaSuccess)
            attr[dev] = cudaFuncSetAttribute(lq_trail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(TrailSmem));
    });
    if (attr[dev] != cudaSuccess) return cuda_fail(attr[dev], "cudaFuncSetAttribute(lq_panel_kernel)");
    for (int k0 = 0; k0 < cmax; k0 += LQ_B) {
        int q = 0;
        while (32 * kNt[q] < cmax - k0) ++q;
        const size_t smem = panel_elems(cmax - k0, kNt[q]) * sizeof(cf);
        kPanel[q]<<<njobs, LQ_T, smem, s>>>(jobs, g, k0);
        MPS_LAUNCH_CHECK("lq_panel_kernel");
        const int rows = max(max_m, max_n) - k0;   // covers every job's rows below its panel
        if (rows > 0) {
            lq_trail_kernel<<<dim3((rows + LQ_TR - 1) / LQ_TR, njobs), 256, sizeof(TrailSmem), s>>>(
                jobs, g, k0);
            MPS_LAUNCH_CHECK("lq_trail_kernel");
        }
    }
    lq_norm_kernel<<<dim3((cmax + 7) / 8, njobs), 256, 0, s>>>(jobs, g);
    MPS_LAUNCH_CHECK("lq_norm_kernel");
    return MPS_OK;
}

}  // namespace mps
