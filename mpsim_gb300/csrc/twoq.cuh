// Workspace geometry shared by the two-qudit kernels (merge, Jacobi SVD,
// sort, regauge).  One slot per job; every job's slot has the same shape.
//
// For a job with theta of m x n (m = chi_l*d, n = d*chi_r), C = min(m, n) columns
// of length L = max(m, n) (see job_tall and job_tracks_v):
//   X = theta    X V = U S
//   X = theta^H  (wide, V tracked)   theta = V S (X/S)^H
//   X = theta^T  (wide or square, right-canonical, V not tracked)
//                X V = U S, theta = conj(V) S U^T
// X: lslot x cslot complex64, column-major (column c at X + c*lslot).
// V: cslot x cslot complex64, column-major, starts as the identity.
#pragma once

#include "common.cuh"

namespace mps {

struct TwoQGeom {
    int d;
    int lslot;        // rows per slot, multiple of 32
    int cslot;        // columns per slot, multiple of 32
    cf* X;            // njobs * lslot * cslot
    cf* V;            // njobs * cslot * cslot (only jobs that track V use theirs)
    cf* T;            // njobs * lslot * cslot: copy of theta for jobs that form
                      // S V^H as U^H theta instead of tracking V
    float* sig;       // njobs * cslot: sorted singular values
    int* perm;        // njobs * cslot: source column of each sorted value
    float* offmax;    // njobs: max relative off-diagonal seen this sweep
    int* done;        // njobs: 1 once a sweep made no rotation
    int* need;        // njobs: kept columns that need an orthonormal completion
    int* counter;     // [0] jobs still rotating, [1] jobs with NaN/Inf, [2] the tensor-core
                      // sweep's item counter, [3] an expired wait (MMA or round flag),
                      // [4] / [5] tensor-core / SIMT jobs left after a sweep (mixed
                      // calls), [6] SIMT jobs of a mixed call, [7] blocks of a
                      // Gram sweep's begin kernel that have sorted their job
    int* cmap;        // njobs * cslot: physical column at each sorted position
    float* cnrm;      // njobs * cslot: squared norm of each physical column
    int* scale;       // njobs: theta was multiplied by 2^scale[j] before the SVD
    double* nrm2;     // njobs: |theta|_F^2 (scratch of the scaling)
    // Visit skipping of the sweep kernel (null where unused).  Times count
    // t = sweep * (rounds + 1) + round + 1, and sweep * (rounds + 1) for the
    // sort before a sweep.
    int* vstamp;      // njobs * nbmax: last time a column block changed
    int* qstamp;      // njobs * qstride: last time visit (round, pair) rotated nothing
    int nbmax, qstride;
    // Products within each 8-column block (block b of job j: 8 x 8 complex at
    // gblk + (j * cslot / 8 + b) * 64, the entries above the diagonal), kept by
    // the Gram sweep kernel beside the columns; null where unused
    cf* gblk;
    // njobs * nbmax, the Gram sweeps' progress (null where unused): x, the last
    // time (as above) a visit of the block ended; y, the last time it changed
    int2* gstate;
    // The jobs the Gram sweeps have left, compacted before every sweep: entry 0
    // is (count, rounds, pairs, 0) over them, entry 1 + i job i's (index, L, C,
    // rows of V); njobs + 1 entries, null where unused
    int4* gact;
    // MPS_PRECISION_MIXED only (null otherwise): X split into three bf16
    // piece planes per job, plane i of job j at P + (3 j + i) * pplane, each
    // laid out like X (column c = 2 lslot bf16 at c * 2 lslot); during the
    // tensor-core sweeps the planes, not X, hold the columns
    uint16_t* P;
    size_t pplane;
    // 1 in MPS_PRECISION_MIXED calls: the jobs tc_job() accepts take the
    // tensor-core sweeps, the SIMT sweep kernel the others
    int tc_mode;
};

// Work distribution of the persistent sweep kernel.
struct SweepSync {
    int* next_item;   // atomic item counter (reset to 0 before each sweep)
    int* error;       // set to 1 when a dependency wait expires
    int* block_round; // [njobs][nbmax]: last round each block finished (-1)
    int nbmax;
    int wait_limit;
    // suspended tries of the Gram sweeps' waits inside a CTA: what they wait for may
    // itself be a wait of wait_limit polls
    int slot_limit;
    int stall_test;
};

// A job's X and whether it tracks the right rotations V.  The factor that must
// come out isometric is the left one (keep_left_canonical) or the right one;
// let Z = theta in the first case and theta^T in the second, so that it is
// the left factor of Z.  Where Z has at least as many rows as columns (every
// square theta, in both forms), X = Z, U = X/S of the final columns is all the
// Jacobi iteration must produce, and the other factor S W^H = U^H Z is one
// product with a copy of Z.  The others (a wide theta left-canonical, a tall one
// right-canonical) work on the other side, X = Z^H, and accumulate V.  So does a
// right-canonical theta at least twice as wide as tall: the few rows of V cost
// less than finishing long columns (a 14-qubit from_wavefunction, whose blocks
// are such, takes 14.5 ms so and 16.4 otherwise).
__host__ __device__ __forceinline__ bool job_tracks_v(int m, int n, int keep_left_canonical) {
    return keep_left_canonical != 0 ? m < n : (m > n || n >= 2 * m);
}

// Whether X holds theta itself (its columns); else theta's conjugate transpose
// (jobs that track V) or transpose (the others).
__host__ __device__ __forceinline__ bool job_tall(int m, int n, int keep_left_canonical) {
    return keep_left_canonical != 0 ? m >= n : m > n;
}

// The jobs of a mixed call that take the tensor-core sweeps: left-canonical,
// tall, 64+ columns (their left factor comes from the final columns).
__host__ __device__ __forceinline__ bool tc_job(int m, int n, int keep_left_canonical) {
    return keep_left_canonical != 0 && m >= n && n >= 64;
}

// ... and whose merge runs on the tensor cores as well (theta not given;
// qudits of up to 4 levels: the gate step keeps a d^2 block in registers).
__host__ __device__ __forceinline__ bool merge_on_tensor_cores(const mps_2q_job& job, int d) {
    return d <= 4 && tc_job(job.chi_l * d, job.chi_r * d, job.keep_left_canonical) &&
           (job.flags & MPS_JOB_THETA_GIVEN) == 0;
}

// Column length of a job's slot: the sweep kernels' row steps.
__host__ __device__ __forceinline__ int slot_rows(int L) {
    return L <= 64 ? 64 : L <= 128 ? 128 : L <= 256 ? 256 : L <= 512 ? 512 : L <= 576 ? 576
           : L <= 1024 ? 1024 : L <= 1792 ? 1792 : (L + 31) / 32 * 32;
}

// The default threshold on a pair's squared cosine for columns of that length.
// The computed x_p^H x_q carries a rounding error of a few 2^-24
// sum_r |x_r||q_r|, growing slowly with the length L; tol = 2^-24 max(8,
// sqrt(L)) stays above that noise (no sweep keeps rotating noise) while the
// kept subspace -- whose error is about tol s_k / gap at the truncation cut --
// stays close to what a backward-stable complex64 SVD gives.
__host__ __device__ __forceinline__ float default_tol2(int rows) {
    const float tol = 5.9604645e-8f * fmaxf(8.f, sqrtf((float)rows));
    return tol * tol;
}

// Singular values at or below this (relative to max(s_0, 1); theta's norm is in
// [1, 2)) are treated as zeros: the isometric factor gets an orthonormal completion
// there.  A little above the norm of columns that the sweeps leave as they are
// (kZeroNorm2 in rot.cuh); divided by their norms those need not be orthogonal: of
// 128 equal columns 113 ended between 1e-21 and 1e-20, all parallel.
constexpr float kZeroSigma = 2e-15f;

// Replaces X by its L factor (X = L Q) for the jobs whose left factor comes
// from the final columns (lq.cu); the sweeps then need fewer passes.
int lq_precondition(const mps_2q_job* jobs, int njobs, int max_m, int max_n, const TwoQGeom& g,
                    cudaStream_t s);

// One sweep of the SIMT jobs by Gram visits (gramsweep.cu): slots of up to
// kGramRows rows, blocks of kGramBlock columns; arguments as for jacobi.cu's
// sweep kernel, but tol2 = 0 asks for each job's own default (by its own
// length, so that it does not depend on the jobs it shares the call with).
constexpr int kGramRows = 1024;
constexpr int kGramBlock = 8;
// gram_begin_launch, before each sweep, lists the jobs left in g.gact and clears
// counter[0] (and [4], [5] of a mixed call) and the item counter; as asked it
// first ends the sweep before (jobs without a pair over the tolerance are
// done), clears the error word, and writes (jobs left, NaN count, error word,
// seq) to a record in pinned host memory.  With sort_cols (the slots' columns) it
// also sorts the columns of the jobs left (presort_job, at time tpre).
struct GramBegin {
    bool end_sweep, clear_error;
    float tol2;
    int* record;
    int seq;
    int sort_cols, tpre;
};
int gram_begin_launch(const mps_2q_job* jobs, int njobs, const TwoQGeom& g, const SweepSync& sync,
                      const GramBegin& b, cudaStream_t s);
int gram_sweep_launch(int njobs, int rounds, int pairs, const TwoQGeom& g,
                      float tol2, const SweepSync& sync, int tbase, cudaStream_t s);

// Tensor-core block sweeps (tcjacobi.cu): one persistent launch runs every
// round of one sweep of the tc_job() jobs, 32-column blocks, with the sweep
// kernel's round flags (sync, with its own item counter) and visit stamps
// (tbase).  counter[3] (and sync.error) is set when a bounded MMA wait
// expired.
int tc_sweep_launch(const mps_2q_job* jobs, int njobs, int rounds, int pairs, const TwoQGeom& g,
                    float tol2, const SweepSync& sync, int tbase, cudaStream_t s);
// X -> its bf16 piece planes (before the first tensor-core sweep), and the
// planes summed back into X (after the last one), for the tc_job() jobs.
int tc_split_launch(const mps_2q_job* jobs, int njobs, const TwoQGeom& g, cudaStream_t s);
int tc_merge_launch(const mps_2q_job* jobs, int njobs, const TwoQGeom& g, cudaStream_t s);

// The mixed form's merge of the merge_on_tensor_cores() jobs (tcgemm.cu): M =
// A B on tcgen05 (split bf16, FP32-grade) into X, then the gate mixed in
// place and copied to T.  The SIMT merge skips those jobs in such a call.
int merge_tc_launch(const mps_2q_job* jobs, int njobs, int max_m, int max_n, const TwoQGeom& g,
                    cudaStream_t s);
int merge_gate_launch(const mps_2q_job* jobs, int njobs, int max_chil, int max_chir,
                      const TwoQGeom& g, cudaStream_t s);

}  // namespace mps
