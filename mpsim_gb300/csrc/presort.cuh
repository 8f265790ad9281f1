// Per-sweep column sort of the SIMT Jacobi jobs, for the kernels that begin a
// sweep (jacobi.cu, gramsweep.cu).
#pragma once

#include "twoq.cuh"

namespace mps {

constexpr int PRESORT_T = 512;

// Shared memory of presort_job: a key and an index for every column.
constexpr size_t presort_smem(int cslot) { return (size_t)cslot * (sizeof(float) + sizeof(int)); }

// Sorts job j's column map by the squared norms in cnrm, descending, ties by
// column index (block-wide, PRESORT_T threads).  Every column counts the columns
// that come before it: P threads a column, four keys a load, no barrier inside
// (a bitonic network's 28 to 55 barriers took 6 to 9 us a sweep of 128 to 512
// columns, this count 2 to 4).
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
        float k = -1.f;
        if (i < C) {
            k = __ldcg(cn + i);
            if (!(k == k)) k = 0.f;                  // NaN sorts as zero
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
            const float ki = key[i];
            for (int q = part; q < C4; q += P) {
                const float4 k = reinterpret_cast<const float4*>(key)[q];
                const int c = 4 * q;
                rank += (k.x > ki || (k.x == ki && c < i)) ? 1 : 0;
                rank += (k.y > ki || (k.y == ki && c + 1 < i)) ? 1 : 0;
                rank += (k.z > ki || (k.z == ki && c + 2 < i)) ? 1 : 0;
                rank += (k.w > ki || (k.w == ki && c + 3 < i)) ? 1 : 0;
            }
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
