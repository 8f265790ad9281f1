// Per-sweep column sort of the SIMT Jacobi jobs, for the kernels that begin a
// sweep (jacobi.cu, gramsweep.cu).
#pragma once

#include <float.h>
#include <math.h>

#include "twoq.cuh"

namespace mps {

constexpr int PRESORT_T = 512;

// Shared memory of presort_job: a key and an index for every column.
constexpr size_t presort_smem(int cslot) { return (size_t)cslot * (sizeof(float) + sizeof(int)); }

// The largest float below x (not NaN or -infinity).
__device__ __forceinline__ float float_below(float x) {
    const int b = __float_as_int(x);
    return __int_as_float(x > 0.f ? b - 1 : (x < 0.f ? b + 1 : (int)0x80000001));
}

// Sorts job j's column map by the squared norms in cnrm, descending, ties by
// column index (block-wide, PRESORT_T threads).  Every column counts the columns
// that come before it: P threads a column, four keys a load, no barrier inside.
// With it the kernel that begins a sweep takes 10.8 us at 256 columns and 14.9 at
// 512 (ncu, cold), against 14.7 and 16.3 for the two it replaced, one of them a
// bitonic network of 36 and 45 barriers, and a launch between.
__device__ __forceinline__ void presort_job(const mps_2q_job& job, const TwoQGeom& g, int j,
                                            float* key, int bc, int tpre) {
    int* idx = reinterpret_cast<int*>(key + g.cslot);         // cslot: a multiple of 32
    const int m = job.chi_l * g.d, n = job.chi_r * g.d;
    const int C = min(m, n);
    if (C < 2) return;
    // The tensor-core sweeps keep their columns in place: measured, their jobs
    // converge about a sweep sooner unsorted (the LQ factor's own column order,
    // and blocks that keep their columns keep their visits skippable), while
    // the SIMT sweeps gain from the sort.
    if (g.tc_mode && tc_job(m, n, job.keep_left_canonical)) return;
    const int tid = threadIdx.x;
    const float* cn = g.cnrm + (size_t)j * g.cslot;
    const int C4 = (C + 3) >> 2;
    for (int i = tid; i < 4 * C4; i += PRESORT_T) {
        // (padding is above nothing; a call with infinities goes on to its error
        // with a valid order)
        float k = -INFINITY;
        if (i < C) {
            k = __ldcg(cn + i);
            k = k == k ? fmaxf(k, -FLT_MAX) : 0.f;   // NaN sorts as zero
        }
        key[i] = k;
    }
    __syncthreads();
    int P = 1;
    while (P < 32 && 2 * P * C <= PRESORT_T) P <<= 1;
    const int part = tid & (P - 1);
    for (int i0 = 0; i0 < C; i0 += PRESORT_T / P) {
        const int i = i0 + tid / P;
        int rank = 0;
        if (i < C) {
            // an earlier column of the same key comes first: it counts against the
            // next float below
            const float ki = key[i], below = float_below(ki);
            const int qi = i >> 2;
            for (int q = part; q < C4; q += P) {
                const float4 k = reinterpret_cast<const float4*>(key)[q];
                const float t = q < qi ? below : ki;
                rank += (k.x > t ? 1 : 0) + (k.y > t ? 1 : 0) + (k.z > t ? 1 : 0) + (k.w > t ? 1 : 0);
            }
            // (of its own four, those before it that are equal are still missing)
            if (part == (qi & (P - 1)))
                for (int c = 4 * qi; c < i; ++c) rank += key[c] == ki ? 1 : 0;
        }
        for (int o = P >> 1; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
        if (part == 0 && i < C) idx[rank] = i;
    }
    __syncthreads();
    if (g.vstamp) {
        // a block whose set of columns changes counts as changed (its pairs
        // are not the ones last checked); moves inside a block do not, except
        // for the Gram sweeps, whose block products go by position
        int* oldpos = reinterpret_cast<int*>(key);     // the keys are no longer needed
        for (int i = tid; i < C; i += PRESORT_T) oldpos[__ldcg(g.cmap + (size_t)j * g.cslot + i)] = i;
        __syncthreads();
        int* vst = g.vstamp + (size_t)j * g.nbmax;
        int2* bst = g.gstate + (size_t)j * g.nbmax;
        for (int c = tid; c < C; c += PRESORT_T) {
            const int ob = oldpos[idx[c]] / bc, nb = c / bc;
            if (g.gstate) {
                if (oldpos[idx[c]] != c) bst[ob].y = bst[nb].y = tpre;
            } else if (ob != nb) {
                vst[ob] = tpre;
                vst[nb] = tpre;
            }
        }
    }
    for (int i = tid; i < C; i += PRESORT_T) g.cmap[(size_t)j * g.cslot + i] = idx[i];
}

}  // namespace mps
