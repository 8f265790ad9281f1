// Complex GEMM tile (FP32 SIMT) of the read-out contractions (contract.cu) and of
// the products that finish a two-qudit gate (jacobi.cu): C = op(A) op(B) with
// arbitrary element strides and optional conjugation.
//
// 256 threads form TM x TN outputs, 4 x 4 a thread (rows ty + TM/4 i, columns
// tx + TN/4 j), from K chunks copied into shared memory three ahead; KS groups of
// threads each take a share of every chunk and are summed at the end, so that a
// 32 x 32 tile keeps all eight warps busy.  A 64 x 64 tile reads shared memory
// in 8 wavefronts for 64 FMAs a thread, so the FP32 pipes bound it.
#pragma once

#include <limits.h>

#include "common.cuh"

namespace mps {

struct GemmArgs {
    int M, N, K;
    const cf* A;
    long long sam, sak;
    int conjA;
    const cf* B;
    long long sbk, sbn;
    int conjB;
    cf* C;
    long long scm, scn;
    int batch;                  // 0 or 1: one product
    long long bsa, bsb, bsc;
};

// acc += a b, or a conj(b).
template <bool CONJ>
__device__ __forceinline__ void cfma_op(cf& acc, cf a, cf b) {
    if (CONJ) {
        acc.x = fmaf(a.x, b.x, fmaf(a.y, b.y, acc.x));
        acc.y = fmaf(a.y, b.x, fmaf(-a.x, b.y, acc.y));
    } else {
        cfma(acc, a, b);
    }
}

__device__ __forceinline__ void copy8_async(uint32_t dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                 : "memory");
}

// The tile at (m0, n0) of g, every output handed to put(row, column, value).
// CONJ: the second factor is conjugated (conjA != conjB); a conjugated first
// factor is the conjugate of the product with the second one's conjugation
// flipped.  GATHER: row i of A (and the row given to put) is rows[i], negative:
// none.  PART > 0: the sum over K is taken in parts of PART chunks, so that its
// rounding error stays that of short sums where every term has the same sign (two
// columns of equal entries: a single sum of 512 terms is off by 1.5e-5).  All
// threads of the block call it.
template <int TM, int TN, int KS, int PART = 0>
struct GemmTile {
    static constexpr int KC = KS > 1 ? 16 : 8;                // K of a chunk
    static constexpr int ST = 4;                              // chunks in shared memory
    static constexpr int BUF = KC * (TM + 1 + TN + 1);
    static constexpr int GT = 256 / KS;                       // threads of a group
    static_assert(TM / 4 * (TN / 4) == GT, "4 x 4 outputs a thread");
    static_assert((KS - 1) * TM * TN <= ST * BUF, "the groups' sums fit");

    template <bool CONJ, bool GATHER, typename Put>
    static __device__ __forceinline__ void run(const GemmArgs& g, int m0, int n0, const int* rows,
                                               cf* sm, const Put& put) {
        constexpr int XN = TN / 4, XM = TM / 4;
        constexpr int NA = TM * KC / 256, NB = TN * KC / 256;     // loads a thread and chunk
        const int tid = threadIdx.x, grp = tid / GT, t = tid % GT, tx = t % XN, ty = t / XN;
        // this thread's elements of a chunk, along the unit stride of each operand:
        // source (of chunk 0), K index (beyond K for an absent row or column)
        const bool a_kfast = g.sak == 1, b_nfast = g.sbn == 1;
        int ak[NA], bk[NB];
        uint32_t ad[NA], bd[NB];
        const cf* ap[NA];
        const cf* bp[NB];
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
#pragma unroll
        for (int q = 0; q < NA; ++q) {
            const int e = tid + 256 * q;
            const int k = a_kfast ? e % KC : e / TM, r = a_kfast ? e / KC : e % TM;
            int row = m0 + r;
            bool in = row < g.M;
            if (GATHER && in) {
                row = rows[row];
                in = row >= 0;
            }
            ak[q] = in ? k : INT_MAX;
            ad[q] = base + (k * (TM + 1) + r) * (uint32_t)sizeof(cf);
            ap[q] = in ? g.A + row * g.sam + k * g.sak : g.A;
        }
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int e = tid + 256 * q;
            const int k = b_nfast ? e / TN : e % KC, c = b_nfast ? e % TN : e / KC;
            const int col = n0 + c;
            bk[q] = col < g.N ? k : INT_MAX;
            bd[q] = base + (KC * (TM + 1) + k * (TN + 1) + c) * (uint32_t)sizeof(cf);
            bp[q] = col < g.N ? g.B + k * g.sbk + col * g.sbn : g.B;
        }
        const long long da = KC * g.sak, db = KC * g.sbk;
        const int chunks = (g.K + KC - 1) / KC;
        // chunk c into buffer c mod ST by 8-byte asynchronous copies (zeros past K)
        const auto fetch = [&](int c) {
            if (c < chunks) {
                const int left = g.K - c * KC;
                const uint32_t off = (uint32_t)((c & (ST - 1)) * BUF) * (uint32_t)sizeof(cf);
#pragma unroll
                for (int q = 0; q < NA; ++q) {
                    const bool in = ak[q] < left;
                    copy8_async(ad[q] + off, in ? ap[q] : g.A, in ? 8u : 0u);
                    ap[q] += da;
                }
#pragma unroll
                for (int q = 0; q < NB; ++q) {
                    const bool in = bk[q] < left;
                    copy8_async(bd[q] + off, in ? bp[q] : g.B, in ? 8u : 0u);
                    bp[q] += db;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        cf acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = cmake(0.f, 0.f);
        cf sum[PART > 0 ? 4 : 1][4];
        if constexpr (PART > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) sum[i][j] = cmake(0.f, 0.f);
        }
#pragma unroll
        for (int c = 0; c < ST - 1; ++c) fetch(c);
        for (int c = 0; c < chunks; ++c) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncthreads();
            fetch(c + ST - 1);
            const cf* As = sm + (c & (ST - 1)) * BUF;
            const cf* Bs = As + KC * (TM + 1);
#pragma unroll
            for (int kk = 0; kk < KC / KS; ++kk) {
                const int k = kk * KS + grp;
                cf av[4], bv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) av[i] = As[k * (TM + 1) + ty + XM * i];
#pragma unroll
                for (int j = 0; j < 4; ++j) bv[j] = Bs[k * (TN + 1) + tx + XN * j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) cfma_op<CONJ>(acc[i][j], av[i], bv[j]);
            }
            if constexpr (PART > 0) {
                if (c % PART == PART - 1 || c == chunks - 1) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            sum[i][j] = cadd(sum[i][j], acc[i][j]);
                            acc[i][j] = cmake(0.f, 0.f);
                        }
                }
            }
        }
        if constexpr (PART > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = sum[i][j];
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (KS > 1) {
            if (grp > 0) {
                cf* dst = sm + (size_t)(grp - 1) * TM * TN;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) dst[(4 * i + j) * GT + t] = acc[i][j];
            }
            __syncthreads();
            if (grp > 0) return;
#pragma unroll
            for (int q = 0; q < KS - 1; ++q)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        acc[i][j] = cadd(acc[i][j], sm[(size_t)q * TM * TN + (4 * i + j) * GT + t]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int row = m0 + ty + XM * i;
            if (row >= g.M) continue;
            if (GATHER) {
                row = rows[row];
                if (row < 0) continue;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int col = n0 + tx + XN * j;
                if (col < g.N) put(row, col, g.conjA ? cconj(acc[i][j]) : acc[i][j]);
            }
        }
    }
};

}  // namespace mps
