// One-qudit gate, left-to-right contraction sweeps (overlap/norm,
// wavefunction, sampled amplitudes, single-site marginals), a strided batched
// complex GEMM and elementwise scale/conjugate.
//
// mpsim performs these with TensorNetwork contractions on the host:
//   apply_one_qudit_gate   mpsim/core.py:820-826
//   wavefunction           mpsim/core.py:483-500
//   inner_product / norm   mpsim/core.py:543-565
//   renormalize / dagger   mpsim/core.py:567-594, 502-505
//   marginals for sample   mpsim/core.py:655-667 (reduced_density_matrix(i)
//                          diagonal, core.py:596-653)
#include <atomic>
#include <string>
#include <vector>

#include "common.cuh"
#include "gemm.cuh"

namespace mps {

thread_local std::string t_error;
static std::atomic<unsigned long long> g_launches{0};

void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

void set_error(const std::string& msg) { t_error = msg; }

int fail(int code, const std::string& msg) {
    t_error = msg;
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    t_error = std::string(what) + ": " + cudaGetErrorString(e);
    return MPS_ERR_CUDA;
}

namespace {

// ---------------------------------------------------------------------------
// One-qudit gate: one thread per (l, r); consecutive threads take consecutive
// r, so every load/store of a (l, a, :) row is coalesced.  HBM-bound:
// 2 * chi_l * d * chi_r * 8 bytes per call.
template <int DMAX>
__global__ void apply_1q_kernel(cf* __restrict__ site, int chil, int d, int chir,
                                const cf* __restrict__ gate) {
    __shared__ cf U[DMAX * DMAX];
    for (int e = threadIdx.x; e < d * d; e += blockDim.x) U[e] = gate[e];
    __syncthreads();
    const size_t total = (size_t)chil * chir;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t l = t / chir, r = t % chir;
        cf* base = site + l * d * chir + r;
        cf v[DMAX];
#pragma unroll
        for (int a = 0; a < DMAX; ++a)
            if (a < d) v[a] = base[(size_t)a * chir];
#pragma unroll
        for (int ap = 0; ap < DMAX; ++ap) {
            if (ap < d) {
                cf acc = cmake(0.f, 0.f);
#pragma unroll
                for (int a = 0; a < DMAX; ++a)
                    if (a < d) cfma(acc, U[ap * d + a], v[a]);
                base[(size_t)ap * chir] = acc;
            }
        }
    }
}

// Batched one-qudit gates: blockIdx.y selects the (site, gate) job.  A job
// whose chi_r is even and whose site is 16-byte aligned (every torch
// allocation is) runs the vectorised form: each thread owns two adjacent r
// and moves them as one 16-byte load and store per a; the 128 threads of a
// CTA form rows of rpw = next power of two of (chi_r / 2), capped at 128,
// lanes, so (l, r) comes from shifts and masks, never from an integer divide.
// Other jobs take the scalar form (one thread per (l, r)).
constexpr int ONEQ_T = 128;

template <int DMAX>
__global__ void __launch_bounds__(ONEQ_T) apply_1q_batch_kernel(const mps_1q_job* __restrict__ jobs,
                                                                int d) {
    __shared__ cf U[DMAX * DMAX];
    const mps_1q_job job = jobs[blockIdx.y];
    const cf* gate = reinterpret_cast<const cf*>(job.gate);
    for (int e = threadIdx.x; e < d * d; e += blockDim.x) U[e] = gate[e];
    __syncthreads();
    const int chil = job.chi_l, chir = job.chi_r;
    cf* site = reinterpret_cast<cf*>(job.site);
    if ((chir & 1) == 0 && (reinterpret_cast<uintptr_t>(site) & 15) == 0) {
        const int rp = chir >> 1;                       // r pairs per row
        int sh = 0;
        while ((1 << sh) < rp && sh < 7) ++sh;          // rpw = 2^sh lanes per row
        const int rows = ONEQ_T >> sh;                  // rows per pass of the CTA
        const int ly = threadIdx.x >> sh, qx = threadIdx.x & ((1 << sh) - 1);
        const size_t rs = (size_t)d * chir;             // complex per l row
        const int step = gridDim.x * rows;
        // two rows per iteration, every load issued before any arithmetic:
        // 2 d 16-byte loads in flight per thread (the kernel is bound by
        // load latency, not by instructions)
        for (int l = blockIdx.x * rows + ly; l < chil; l += 2 * step) {
            const int l2 = l + step;
            const bool two = l2 < chil;
            float4* row = reinterpret_cast<float4*>(site + (size_t)l * rs);
            float4* row2 = reinterpret_cast<float4*>(site + (size_t)(two ? l2 : l) * rs);
            for (int q = qx; q < rp; q += 1 << sh) {
                float4 v[DMAX], w[DMAX];
#pragma unroll
                for (int a = 0; a < DMAX; ++a) {
                    if (a < d) {
                        v[a] = __ldcs(row + (size_t)a * rp + q);
                        if (two) w[a] = __ldcs(row2 + (size_t)a * rp + q);
                    }
                }
#pragma unroll
                for (int ap = 0; ap < DMAX; ++ap) {
                    if (ap < d) {
                        cf a0 = cmake(0.f, 0.f), a1 = cmake(0.f, 0.f);
                        cf b0 = cmake(0.f, 0.f), b1 = cmake(0.f, 0.f);
#pragma unroll
                        for (int a = 0; a < DMAX; ++a) {
                            if (a < d) {
                                const cf u = U[ap * d + a];
                                cfma(a0, u, cmake(v[a].x, v[a].y));
                                cfma(a1, u, cmake(v[a].z, v[a].w));
                                if (two) {
                                    cfma(b0, u, cmake(w[a].x, w[a].y));
                                    cfma(b1, u, cmake(w[a].z, w[a].w));
                                }
                            }
                        }
                        __stcs(row + (size_t)ap * rp + q, make_float4(a0.x, a0.y, a1.x, a1.y));
                        if (two) __stcs(row2 + (size_t)ap * rp + q, make_float4(b0.x, b0.y, b1.x, b1.y));
                    }
                }
            }
        }
        return;
    }
    const size_t total = (size_t)chil * chir;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t l = t / chir, r = t % chir;
        cf* base = site + l * d * chir + r;
        cf v[DMAX];
#pragma unroll
        for (int a = 0; a < DMAX; ++a)
            if (a < d) v[a] = base[(size_t)a * chir];
#pragma unroll
        for (int ap = 0; ap < DMAX; ++ap) {
            if (ap < d) {
                cf acc = cmake(0.f, 0.f);
#pragma unroll
                for (int a = 0; a < DMAX; ++a)
                    if (a < d) cfma(acc, U[ap * d + a], v[a]);
                base[(size_t)ap * chir] = acc;
            }
        }
    }
}

__global__ void scale_kernel(cf* __restrict__ x, size_t count, cf alpha, int conj) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < count;
         t += (size_t)gridDim.x * blockDim.x) {
        cf v = x[t];
        if (conj) v = cconj(v);
        x[t] = cmul(alpha, v);
    }
}

// ---------------------------------------------------------------------------
// Generic complex GEMM C = op(A) op(B) with arbitrary element strides and
// optional conjugation, batched over blockIdx.z with element strides bsa,
// bsb, bsc between batches (zero: the same matrix for every batch), or two
// different products in one launch (the two directions of a sweep).
//
// What bounds it: the FP32 pipes for large products (gemm.cuh), and the few tiles of the sweeps'
// 256 x 512 x 256 steps otherwise -- there 32 x 32 tiles, and both directions
// of a sweep in one launch, put work on every SM.  Measured (GB300) against one
// direction at a time, 64 x 64 tiles and loads that were waited for chunk by
// chunk: norm and overlap of a 64-site chi=256 state 14.3 -> 2.65 ms (FMA pipe
// 53% busy, 74% of issue slots), marginals of 48 sites of chi=128 8.1 -> 0.96 ms
// (the third product a site is gone too), 4096 amplitudes at chi=256 7.6 -> 3.1 ms
// (half of the products were of digits not asked for).
// GATHER (sampled amplitudes): row i of A and C is row rows[i] of the arrays
// (negative: none), and B is shifted by digit * bdig, one digit per TM rows
// (negative: no row; >= ndig: the product is zero).
struct GemmGather {
    const int* rows;
    const int* digit;
    long long bdig;
    int ndig;
};

struct GemmLaunch {
    GemmArgs p[2];
    int two;                    // blockIdx.z selects p[0] or p[1], else the batch
    GemmGather ga;
};

template <int TM, int TN, int KS, bool CONJ, bool GATHER>
__global__ void __launch_bounds__(256, 2) cgemm_kernel(const __grid_constant__ GemmLaunch gl) {
    using Tile = GemmTile<TM, TN, KS>;
    __shared__ __align__(16) cf sm[Tile::ST * Tile::BUF];
    if (GATHER) {
        // (see launch_gather) the site before has to have ended before anything is
        // read or written; from here on the next one's CTAs may come
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;");
    }
    GemmArgs g = gl.p[gl.two && blockIdx.z ? 1 : 0];
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    if (m0 >= g.M || n0 >= g.N) return;
    if (!gl.two) {
        g.A += blockIdx.z * g.bsa;
        g.B += blockIdx.z * g.bsb;
        g.C += blockIdx.z * g.bsc;
    }
    if (GATHER) {
        const int x = gl.ga.digit[blockIdx.y];
        if (x < 0) return;
        if (x >= gl.ga.ndig) g.K = 0;
        else g.B += x * gl.ga.bdig;
    }
    Tile::template run<CONJ, GATHER>(g, m0, n0, gl.ga.rows, sm, [&](int row, int col, cf v) {
        g.C[row * g.scm + col * g.scn] = v;
    });
}

// 64 x 64 tiles once they give every SM a CTA, else 32 x 32 (four times the tiles,
// the K loop split over four groups of threads).  Measured with each: 64 steps
// of two 256 x 512 x 256 products (64 large tiles), 2.64 ms small against 5.00
// large; 64 products of 4096 x 256 x 256 (256 large tiles), 3.13 against 3.05.
bool small_tiles(long long m, long long n, long long count) {
    return ((m + 63) / 64) * ((n + 63) / 64) * count < kSms;
}

// The amplitudes' product of a site is queued so that its CTAs take their places
// while the site before still runs and wait inside, instead of being launched
// after it: early, for 64 x 64 tiles (several a SM: 4096 amplitudes, 64 sites
// chi=256, 3.05 -> 2.94 ms) and for so few 32 x 32 ones that those of two sites hardly
// share SMs (68 of them, 60 sites chi=33, 0.54 -> 0.435 ms; 84, 64 qutrits chi=192,
// 0.795 -> 0.685; but 104, 40 qutrits chi=100, 0.473 -> 0.491, the SMs shared unevenly).
// (The next site is let in after the wait, so that one site at most is ahead; before
// it, the 84 took 0.97 ms and the overlap sweeps lost a tenth.)
template <typename Kernel>
int launch_gather(Kernel kernel, int tile, dim3 grid, cudaStream_t s, const GemmLaunch& gl) {
    const bool early = tile == 64 || (long long)grid.x * grid.y * 8 <= 5 * kSms;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    MPS_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, gl));
    MPS_LAUNCH_CHECK("cgemm_kernel");
    return MPS_OK;
}

int cgemm_launch(const GemmLaunch& gl, int m, int n, int z, cudaStream_t s) {
    const bool small = small_tiles(m, n, z);
    const int t = small ? 32 : 64;
    const dim3 grid((n + t - 1) / t, (m + t - 1) / t, z);
    if (grid.y > 65535) return fail(MPS_ERR_ARG, "cgemm: too many rows");
    if (grid.z > 65535) return fail(MPS_ERR_ARG, "cgemm: batch above 65535");
    const bool conj = gl.p[0].conjA != gl.p[0].conjB;
    if (small) {
        if (conj) cgemm_kernel<32, 32, 4, true, false><<<grid, 256, 0, s>>>(gl);
        else cgemm_kernel<32, 32, 4, false, false><<<grid, 256, 0, s>>>(gl);
    } else {
        if (conj) cgemm_kernel<64, 64, 1, true, false><<<grid, 256, 0, s>>>(gl);
        else cgemm_kernel<64, 64, 1, false, false><<<grid, 256, 0, s>>>(gl);
    }
    MPS_LAUNCH_CHECK("cgemm_kernel");
    return MPS_OK;
}

int cgemm(const GemmArgs& a, cudaStream_t s) {
    if (a.M <= 0 || a.N <= 0 || a.batch < 0) return MPS_OK;
    GemmLaunch gl{};
    gl.p[0] = a;
    return cgemm_launch(gl, a.M, a.N, a.batch > 1 ? a.batch : 1, s);
}

// Two independent products in one launch (either may be empty).
int cgemm2(const GemmArgs& a, const GemmArgs& b, cudaStream_t s) {
    const bool ea = a.M <= 0 || a.N <= 0, eb = b.M <= 0 || b.N <= 0;
    if (ea) return cgemm(b, s);
    if (eb) return cgemm(a, s);
    if ((a.conjA != a.conjB) != (b.conjA != b.conjB)) {
        if (int rc = cgemm(a, s)) return rc;
        return cgemm(b, s);
    }
    GemmLaunch gl{};
    gl.p[0] = a;
    gl.p[1] = b;
    gl.two = 1;
    return cgemm_launch(gl, max(a.M, b.M), max(a.N, b.N), 2, s);
}

// ---------------------------------------------------------------------------
// Sampled amplitudes: a site's digit picks which of its d matrices multiplies
// a bitstring's environment, so the bitstrings are grouped by digit, each
// group padded to whole row tiles, and only the matrix picked is multiplied.
// A block per site and chunk of bitstrings lists them: rows[site][...] (order kept
// within a digit), one digit per tile (digits outside 0..d-1, whose amplitude is
// zero, come last as digit d; -1: no tile).  Where there are several chunks, a launch
// before counts the digits of each (count_digits_kernel), from which every block
// knows where its rows begin.  One block per site for any number of bitstrings was
// slower than the products it saved: 10^6 of them, 12 sites of bond 1, 7.8 ms so
// against 3.6 now (4.5 with every digit's product); 64 sites of bond 16, 32.1 against
// 24.7 (29.5).
constexpr int kGroupT = 256;
constexpr int kGroupChunk = 4096;
constexpr int kDigits = 128;                  // digits that an int8 can name
int group_chunks(int nbits) { return (nbits + kGroupChunk - 1) / kGroupChunk; }

// The digit's group: itself, or d where it is none of the site's (d <= kDigits).
__device__ __forceinline__ int digit_group(int v, int d) { return v < 0 || v >= d ? d : v; }

// counts[site][chunk][x]: bitstrings of the chunk whose digit at the site is x (d: none).
__global__ void __launch_bounds__(kGroupT) count_digits_kernel(const int8_t* __restrict__ bits,
                                                               int nbits, int n, int d,
                                                               int* __restrict__ counts) {
    __shared__ int s_count[kDigits + 1];
    const int site = blockIdx.x, chunk = blockIdx.y;
    for (int x = threadIdx.x; x <= d; x += kGroupT) s_count[x] = 0;
    __syncthreads();
    const int end = min(nbits, (chunk + 1) * kGroupChunk);
    for (int q = chunk * kGroupChunk + threadIdx.x; q < end; q += kGroupT)
        atomicAdd(&s_count[digit_group(bits[(size_t)q * n + site], d)], 1);
    __syncthreads();
    int* out = counts + ((size_t)site * gridDim.y + chunk) * (d + 1);
    for (int x = threadIdx.x; x <= d; x += kGroupT) out[x] = s_count[x];
}

__global__ void __launch_bounds__(kGroupT) group_bits_kernel(const int8_t* __restrict__ bits,
                                                             int nbits, int n, int d, int tile,
                                                             int tiles, const int* __restrict__ counts,
                                                             int* __restrict__ rows,
                                                             int* __restrict__ digit) {
    __shared__ int s_warp[kGroupT / 32];
    __shared__ int s_before[kDigits + 1], s_total[kDigits + 1];      // several chunks only
    const int site = blockIdx.x, chunk = blockIdx.y, chunks = gridDim.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int* r = rows + (size_t)site * tiles * tile;
    int* g = digit + (size_t)site * tiles;
    if (chunks > 1) {
        const int* c = counts + (size_t)site * chunks * (d + 1);
        for (int x = warp; x <= d; x += kGroupT / 32) {
            int before = 0, total = 0;
            for (int b = lane; b < chunks; b += 32) {
                const int v = c[(size_t)b * (d + 1) + x];
                total += v;
                if (b < chunk) before += v;
            }
            for (int o = 16; o > 0; o >>= 1) {
                before += __shfl_xor_sync(0xffffffffu, before, o);
                total += __shfl_xor_sync(0xffffffffu, total, o);
            }
            if (lane == 0) {
                s_before[x] = before;
                s_total[x] = total;
            }
        }
        __syncthreads();
    }
    const int first = chunk * kGroupChunk, last = min(nbits, first + kGroupChunk);
    int at = 0;                               // the digit's first position, a multiple of tile
    for (int x = 0; x <= d; ++x) {
        int count = chunks > 1 ? s_before[x] : 0;
        for (int s0 = first; s0 < last; s0 += kGroupT) {
            const int sidx = s0 + tid;
            const bool mine = sidx < last && digit_group(bits[(size_t)sidx * n + site], d) == x;
            const unsigned mask = __ballot_sync(0xffffffffu, mine);
            if (lane == 0) s_warp[warp] = __popc(mask);
            __syncthreads();
            int before = 0, all = 0;
            for (int w = 0; w < kGroupT / 32; ++w) {
                if (w < warp) before += s_warp[w];
                all += s_warp[w];
            }
            if (mine) r[at + count + before + __popc(mask & ((1u << lane) - 1u))] = sidx;
            count += all;
            __syncthreads();
        }
        const int total = chunks > 1 ? s_total[x] : count;
        const int end = at + (total + tile - 1) / tile * tile;
        if (chunk == 0) {
            for (int q = at + total + tid; q < end; q += kGroupT) r[q] = -1;
            for (int q = at / tile + tid; q < end / tile; q += kGroupT) g[q] = x;
        }
        at = end;
    }
    if (chunk == 0)
        for (int q = at / tile + tid; q < tiles; q += kGroupT) g[q] = -1;
}

// env'[s, r] = full[s, x_s * chir + r]
__global__ void select_kernel(const cf* __restrict__ full, cf* __restrict__ env, int nbits,
                              int chir, int d, const int8_t* __restrict__ bits, int n, int site) {
    const size_t total = (size_t)nbits * chir;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t sidx = t / chir, r = t % chir;
        const int x = bits[sidx * n + site];
        env[t] = (x >= 0 && x < d) ? full[sidx * (size_t)d * chir + (size_t)x * chir + r]
                                   : cmake(0.f, 0.f);
    }
}

// What the two directions of a marginal sweep leave for one site.
struct MarginalSite {
    const cf* T;                // T[l, x, r'] = sum_l' L[l, l'] conj(A[l', x, r'])
    const cf* V;                // V[l, x, r'] = sum_r  conj(A[l, x, r]) R[r', r]
    int chil, chir;
};
constexpr int kMarginalBatch = 64;
struct MarginalArgs {
    MarginalSite s[kMarginalBatch];
};

// probs[site * d + x] = Re sum_{l, r'} T[l, x, r'] conj(V[l, x, r']): block (x, site),
// FP64 sum.
__global__ void __launch_bounds__(256) marginal_kernel(const __grid_constant__ MarginalArgs a, int d,
                                                       float* __restrict__ probs) {
    __shared__ double part[256];
    const int x = blockIdx.x;
    const MarginalSite& s = a.s[blockIdx.y];
    const int chir = s.chir, rows = s.chil;
    double acc = 0.0;
    // 8 warps take rows l in turn, lanes consecutive r'
    for (int l = threadIdx.x >> 5; l < rows; l += 8) {
        const size_t o = ((size_t)l * d + x) * chir;
        for (int r = threadIdx.x & 31; r < chir; r += 32) {
            const cf t = s.T[o + r], v = s.V[o + r];
            acc += (double)t.x * v.x + (double)t.y * v.y;
        }
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) probs[(size_t)blockIdx.y * d + x] = (float)part[0];
}

// sum_i a[i] b[i] in FP64 (one block) into out (re, im).
__global__ void __launch_bounds__(1024) dot_kernel(const cf* __restrict__ a, const cf* __restrict__ b,
                                                   size_t count, double* __restrict__ out) {
    __shared__ double pr[1024], pi[1024];
    double re = 0.0, im = 0.0;
    for (size_t t = threadIdx.x; t < count; t += 1024) {
        const cf x = a[t], y = b[t];
        re += (double)x.x * y.x - (double)x.y * y.y;
        im += (double)x.x * y.y + (double)x.y * y.x;
    }
    pr[threadIdx.x] = re;
    pi[threadIdx.x] = im;
    __syncthreads();
    for (int o = 512; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            pr[threadIdx.x] += pr[threadIdx.x + o];
            pi[threadIdx.x] += pi[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = pr[0];
        out[1] = pi[0];
    }
}

__global__ void fill_one_kernel(cf* x, size_t count) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < count;
         t += (size_t)gridDim.x * blockDim.x)
        x[t] = cmake(1.f, 0.f);
}

int grid_for(size_t total) {
    size_t b = (total + 255) / 256;
    if (b < 1) b = 1;
    if (b > 8192) b = 8192;
    return (int)b;
}

}  // namespace
}  // namespace mps

using namespace mps;

extern "C" int mps_version(void) { return 100; }

extern "C" const char* mps_last_error(void) { return t_error.c_str(); }

extern "C" unsigned long long mps_kernel_launches(void) { return g_launches.load(); }

extern "C" int mps_apply_1q(void* stream, mps_c64* site, int chi_l, int d, int chi_r,
                            const mps_c64* gate) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (chi_l < 0 || chi_r < 0 || d < 1 || d > 64) return fail(MPS_ERR_ARG, "mps_apply_1q: bad shape");
    const size_t total = (size_t)chi_l * chi_r;
    if (total == 0) return MPS_OK;
    if (!site || !gate) return fail(MPS_ERR_ARG, "mps_apply_1q: null pointer");
    cf* x = reinterpret_cast<cf*>(site);
    const cf* u = reinterpret_cast<const cf*>(gate);
    const int blocks = grid_for(total);
    if (d <= 2) apply_1q_kernel<2><<<blocks, 256, 0, s>>>(x, chi_l, d, chi_r, u);
    else if (d <= 4) apply_1q_kernel<4><<<blocks, 256, 0, s>>>(x, chi_l, d, chi_r, u);
    else if (d <= 8) apply_1q_kernel<8><<<blocks, 256, 0, s>>>(x, chi_l, d, chi_r, u);
    else if (d <= 16) apply_1q_kernel<16><<<blocks, 256, 0, s>>>(x, chi_l, d, chi_r, u);
    else apply_1q_kernel<64><<<blocks, 256, 0, s>>>(x, chi_l, d, chi_r, u);
    MPS_LAUNCH_CHECK("apply_1q_kernel");
    return MPS_OK;
}

extern "C" int mps_apply_1q_batch(void* stream, const mps_1q_job* jobs, int njobs, int d) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (njobs == 0) return MPS_OK;
    if (njobs < 0 || njobs > 65535 || !jobs) return fail(MPS_ERR_ARG, "mps_apply_1q_batch: bad job list");
    if (d < 1 || d > 64) return fail(MPS_ERR_ARG, "mps_apply_1q_batch: bad qudit dimension");
    // 16 CTAs per job, two rows per thread per iteration: a 64-site chi=256
    // layer is 1024 CTAs of 128 threads, ~27 warps and ~55 KB of loads in
    // flight per SM
    dim3 grid(16, njobs);
    if (d <= 2) apply_1q_batch_kernel<2><<<grid, ONEQ_T, 0, s>>>(jobs, d);
    else if (d <= 4) apply_1q_batch_kernel<4><<<grid, ONEQ_T, 0, s>>>(jobs, d);
    else if (d <= 8) apply_1q_batch_kernel<8><<<grid, ONEQ_T, 0, s>>>(jobs, d);
    else if (d <= 16) apply_1q_batch_kernel<16><<<grid, ONEQ_T, 0, s>>>(jobs, d);
    else apply_1q_batch_kernel<64><<<grid, ONEQ_T, 0, s>>>(jobs, d);
    MPS_LAUNCH_CHECK("apply_1q_batch_kernel");
    return MPS_OK;
}

extern "C" int mps_scale(void* stream, mps_c64* site, size_t count, float alpha_re,
                         float alpha_im, int conj) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (count == 0) return MPS_OK;
    if (!site) return fail(MPS_ERR_ARG, "mps_scale: null pointer");
    scale_kernel<<<grid_for(count), 256, 0, s>>>(reinterpret_cast<cf*>(site), count,
                                                 cmake(alpha_re, alpha_im), conj);
    MPS_LAUNCH_CHECK("scale_kernel");
    return MPS_OK;
}

extern "C" size_t mps_sweep_workspace_bytes(int max_chi, int d) {
    if (max_chi < 1) max_chi = 1;
    const size_t c = (size_t)max_chi;        // two environments and a product, for each direction
    return align_up(2 * (2 * c * c + (size_t)d * c * c) * sizeof(cf) + 1024, 256);
}

extern "C" int mps_inner_product(void* stream, const mps_c64* const* a_sites, const int* chis_a,
                                 const mps_c64* const* b_sites, const int* chis_b, int n, int d,
                                 void* workspace, size_t workspace_bytes, double* result_host) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n < 1 || d < 1 || !a_sites || !b_sites || !chis_a || !chis_b || !result_host)
        return fail(MPS_ERR_ARG, "mps_inner_product: bad arguments");
    if (chis_a[0] != 1 || chis_b[0] != 1 || chis_a[n] != 1 || chis_b[n] != 1)
        return fail(MPS_ERR_ARG, "mps_inner_product: end bonds must be 1");
    int maxchi = 1;
    for (int i = 0; i <= n; ++i) maxchi = max(maxchi, max(chis_a[i], chis_b[i]));
    if (workspace_bytes < mps_sweep_workspace_bytes(maxchi, d) || !workspace)
        return fail(MPS_ERR_WORKSPACE, "mps_inner_product: workspace too small");
    // The left half of the chain is contracted from the left and the right half
    // from the right, side by side: half the dependent steps, twice the work
    // in each.  The two environments meet at the middle bond.
    const size_t cc = (size_t)maxchi * maxchi;
    double* dot = static_cast<double*>(workspace);
    cf* E[2] = {reinterpret_cast<cf*>(dot + 2), nullptr};
    E[1] = E[0] + cc;
    cf* R[2] = {E[1] + cc, E[1] + 2 * cc};
    cf* T = R[1] + cc;
    cf* V = T + (size_t)d * cc;
    fill_one_kernel<<<1, 32, 0, s>>>(E[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    fill_one_kernel<<<1, 32, 0, s>>>(R[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    const int mid = n / 2;
    const GemmArgs none{};
    int ce = 0, cr = 0;
    for (int t = 0; t < n - mid; ++t) {
        GemmArgs l1 = none, l2 = none, r1 = none, r2 = none;
        if (t < mid) {
            const int al = chis_a[t], ar = chis_a[t + 1], bl = chis_b[t], br = chis_b[t + 1];
            const cf* A = reinterpret_cast<const cf*>(a_sites[t]);
            const cf* B = reinterpret_cast<const cf*>(b_sites[t]);
            // T[l, (x, r')] = sum_l' E[l, l'] conj(B[l', x, r'])
            l1 = GemmArgs{al, d * br, bl, E[ce], bl, 1, 0, B, (long long)d * br, 1, 1,
                          T, (long long)d * br, 1};
            // E'[r, r'] = sum_(l,x) A[(l,x), r] T[(l,x), r']
            l2 = GemmArgs{ar, br, al * d, A, 1, ar, 0, T, br, 1, 0, E[ce ^ 1], br, 1};
            ce ^= 1;
        }
        {
            const int i = n - 1 - t;
            const int al = chis_a[i], ar = chis_a[i + 1], bl = chis_b[i], br = chis_b[i + 1];
            const cf* A = reinterpret_cast<const cf*>(a_sites[i]);
            const cf* B = reinterpret_cast<const cf*>(b_sites[i]);
            // V[(l', x), r] = sum_r' conj(B[(l', x), r']) R[r, r']
            r1 = GemmArgs{bl * d, ar, br, B, br, 1, 1, R[cr], 1, br, 0, V, ar, 1};
            // R'[l, l'] = sum_(x,r) A[l, (x, r)] V[l', (x, r)]
            r2 = GemmArgs{al, bl, d * ar, A, (long long)d * ar, 1, 0, V, 1, (long long)d * ar, 0,
                          R[cr ^ 1], bl, 1};
            cr ^= 1;
        }
        int rc = cgemm2(l1, r1, s);
        if (rc) return rc;
        rc = cgemm2(l2, r2, s);
        if (rc) return rc;
    }
    dot_kernel<<<1, 1024, 0, s>>>(E[ce], R[cr], (size_t)chis_a[mid] * chis_b[mid], dot);
    MPS_LAUNCH_CHECK("dot_kernel");
    double res[2];
    MPS_CUDA_CHECK(cudaMemcpyAsync(res, dot, sizeof(res), cudaMemcpyDeviceToHost, s));
    MPS_CUDA_CHECK(cudaStreamSynchronize(s));
    result_host[0] = res[0];
    result_host[1] = res[1];
    return MPS_OK;
}

extern "C" int mps_wavefunction(void* stream, const mps_c64* const* sites, const int* chis,
                                int n, int d, mps_c64* out_dev, void* workspace,
                                size_t workspace_bytes) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n < 1 || d < 1 || !sites || !chis || !out_dev)
        return fail(MPS_ERR_ARG, "mps_wavefunction: bad arguments");
    size_t need = 1, p = 1;
    for (int i = 0; i < n; ++i) {
        p *= (size_t)d;
        need = max(need, p * (size_t)max(chis[i + 1], 1));
    }
    if (!workspace || workspace_bytes < 2 * need * sizeof(cf))
        return fail(MPS_ERR_WORKSPACE, "mps_wavefunction: workspace too small");
    cf* buf[2] = {static_cast<cf*>(workspace), static_cast<cf*>(workspace) + need};
    fill_one_kernel<<<1, 32, 0, s>>>(buf[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    size_t P = 1;
    int cur = 0;
    for (int i = 0; i < n; ++i) {
        const int cl = chis[i], cr = chis[i + 1];
        cf* dst = (i == n - 1) ? reinterpret_cast<cf*>(out_dev) : buf[cur ^ 1];
        const size_t rows = P;
        if (rows > 0x7fffffff) return fail(MPS_ERR_ARG, "mps_wavefunction: state too large");
        if (cl == 0) {
            MPS_CUDA_CHECK(cudaMemsetAsync(dst, 0, rows * d * cr * sizeof(cf), s));
        } else {
            GemmArgs g{(int)rows, d * cr, cl, buf[cur], cl, 1, 0,
                       reinterpret_cast<const cf*>(sites[i]), (long long)d * cr, 1, 0,
                       dst, (long long)d * cr, 1};
            // cgemm tiles rows in grid.y (<= 65535 * 64 rows); split larger ones
            const long long chunk = 65535LL * 64;
            for (long long r0 = 0; r0 < (long long)rows; r0 += chunk) {
                GemmArgs gc = g;
                gc.M = (int)(((long long)rows - r0) < chunk ? ((long long)rows - r0) : chunk);
                gc.A = buf[cur] + r0 * cl;
                gc.C = dst + r0 * (long long)d * cr;
                int rc = cgemm(gc, s);
                if (rc) return rc;
            }
        }
        P = rows * d;
        cur ^= 1;
    }
    return MPS_OK;
}

namespace {

// Row tile of the grouped amplitude products: 64 where such tiles fill the GPU.
int amplitude_tile(int nbits, int maxchi, int d) {
    (void)d;
    return small_tiles(nbits, maxchi, 1) ? 32 : 64;
}
int amplitude_tiles(int nbits, int d, int tile) {
    return (nbits + tile - 1) / tile + min(d, kDigits) + 1;
}
// Counts of a call's digits at every site (none where there is one chunk).
size_t amplitude_counts(int nbits, int n, int d) {
    const int chunks = group_chunks(nbits);
    return chunks > 1 ? (size_t)n * chunks * (min(d, kDigits) + 1) : 0;
}
// Lists of n sites.
size_t amplitude_lists(int nbits, int maxchi, int n, int d) {
    const int tile = amplitude_tile(nbits, maxchi, d);
    const size_t tiles = (size_t)amplitude_tiles(nbits, d, tile);
    return ((size_t)n * tiles * (tile + 1) + amplitude_counts(nbits, n, d)) * sizeof(int);
}
// Sites whose lists are made together: all of them, if the lists stay within 256 MiB or
// within what a product of every digit would take (4 10^6 bitstrings of 1000 sites
// would be 16 GB); else as many as do, and the lists are made again for the next ones.
int amplitude_group_sites(int nbits, int maxchi, int n, int d) {
    const size_t room = max((size_t)256 << 20, (size_t)nbits * d * maxchi * sizeof(cf));
    const size_t sites = room / amplitude_lists(nbits, maxchi, 1, d);
    return sites < 1 ? 1 : (int)min(sites, (size_t)n);
}
size_t amplitude_bytes(int nbits, int maxchi, int n, int d) {
    return 2 * (size_t)nbits * maxchi * sizeof(cf) +
           amplitude_lists(nbits, maxchi, amplitude_group_sites(nbits, maxchi, n, d), d);
}

}  // namespace

extern "C" size_t mps_amplitudes_workspace_bytes(int nbits, int max_chi, int n, int d) {
    if (nbits < 1 || max_chi < 1 || n < 1 || d < 1) return 0;
    const size_t ungrouped = ((size_t)nbits * d * max_chi + 2 * (size_t)nbits * max_chi) * sizeof(cf);
    return max(ungrouped, amplitude_bytes(nbits, max_chi, n, d));
}

extern "C" int mps_amplitudes(void* stream, const mps_c64* const* sites, const int* chis, int n,
                              int d, const int8_t* bits_dev, int nbits, mps_c64* out_dev,
                              void* workspace, size_t workspace_bytes) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n < 1 || d < 1 || nbits < 0 || !sites || !chis || (nbits > 0 && (!bits_dev || !out_dev)))
        return fail(MPS_ERR_ARG, "mps_amplitudes: bad arguments");
    if (nbits == 0) return MPS_OK;
    int maxchi = 1;
    for (int i = 0; i <= n; ++i) maxchi = max(maxchi, chis[i]);
    const size_t full_sz = (size_t)nbits * d * maxchi, env_sz = (size_t)nbits * maxchi;
    if (!workspace || workspace_bytes < (full_sz + 2 * env_sz) * sizeof(cf))
        return fail(MPS_ERR_WORKSPACE, "mps_amplitudes: workspace too small");
    const int tile = amplitude_tile(nbits, maxchi, d);
    if (workspace_bytes >= amplitude_bytes(nbits, maxchi, n, d) &&
        amplitude_tiles(nbits, d, tile) <= 65535) {
        cf* ge[2] = {static_cast<cf*>(workspace), static_cast<cf*>(workspace) + env_sz};
        const int tiles = amplitude_tiles(nbits, d, tile);
        const int group = amplitude_group_sites(nbits, maxchi, n, d), nd = min(d, kDigits);
        int* rows = reinterpret_cast<int*>(ge[1] + env_sz);
        int* digit = rows + (size_t)group * tiles * tile;
        int* counts = digit + (size_t)group * tiles;
        fill_one_kernel<<<grid_for(nbits), 256, 0, s>>>(ge[0], nbits);
        MPS_LAUNCH_CHECK("fill_one_kernel");
        for (int i = 0, at = 0; i < n; ++i, at ^= 1) {
            if (i % group == 0) {
                const dim3 grid(min(group, n - i), group_chunks(nbits));
                if (grid.y > 1) {
                    count_digits_kernel<<<grid, kGroupT, 0, s>>>(bits_dev + i, nbits, n, nd, counts);
                    MPS_LAUNCH_CHECK("count_digits_kernel");
                }
                group_bits_kernel<<<grid, kGroupT, 0, s>>>(bits_dev + i, nbits, n, nd, tile, tiles,
                                                           counts, rows, digit);
                MPS_LAUNCH_CHECK("group_bits_kernel");
            }
            const int cl = chis[i], cr = chis[i + 1];
            if (cr == 0) continue;
            cf* dst = (i == n - 1) ? reinterpret_cast<cf*>(out_dev) : ge[at ^ 1];
            GemmLaunch gl{};
            gl.p[0] = GemmArgs{tiles * tile, cr, cl, ge[at], cl, 1, 0,
                               reinterpret_cast<const cf*>(sites[i]), (long long)d * cr, 1, 0,
                               dst, cr, 1};
            gl.ga = GemmGather{rows + (size_t)(i % group) * tiles * tile,
                               digit + (size_t)(i % group) * tiles, cr, nd};
            const dim3 grid((cr + tile - 1) / tile, tiles);
            const int rc = tile == 32
                               ? launch_gather(cgemm_kernel<32, 32, 4, false, true>, 32, grid, s, gl)
                               : launch_gather(cgemm_kernel<64, 64, 1, false, true>, 64, grid, s, gl);
            if (rc) return rc;
        }
        return MPS_OK;
    }
    // a workspace without room for the groups: every digit's product, then the
    // one picked
    cf* full = static_cast<cf*>(workspace);
    cf* env[2] = {full + full_sz, full + full_sz + env_sz};
    fill_one_kernel<<<grid_for(nbits), 256, 0, s>>>(env[0], nbits);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    int cur = 0;
    for (int i = 0; i < n; ++i) {
        const int cl = chis[i], cr = chis[i + 1];
        cf* dst = (i == n - 1) ? reinterpret_cast<cf*>(out_dev) : env[cur ^ 1];
        if (cl == 0) {
            MPS_CUDA_CHECK(cudaMemsetAsync(full, 0, (size_t)nbits * d * cr * sizeof(cf), s));
        } else {
            GemmArgs g{nbits, d * cr, cl, env[cur], cl, 1, 0, reinterpret_cast<const cf*>(sites[i]),
                       (long long)d * cr, 1, 0, full, (long long)d * cr, 1};
            int rc = cgemm(g, s);
            if (rc) return rc;
        }
        select_kernel<<<grid_for((size_t)nbits * cr), 256, 0, s>>>(full, dst, nbits, cr, d,
                                                                    bits_dev, n, i);
        MPS_LAUNCH_CHECK("select_kernel");
        cur ^= 1;
    }
    return MPS_OK;
}

extern "C" int mps_cgemm(void* stream, int m, int n, int k, const mps_c64* a, long long sam,
                         long long sak, int conj_a, const mps_c64* b, long long sbk,
                         long long sbn, int conj_b, mps_c64* c, long long scm, long long scn,
                         int batch, long long bsa, long long bsb, long long bsc) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (m < 0 || n < 0 || k < 0 || batch < 0 || (m > 0 && n > 0 && (!c || (k > 0 && (!a || !b)))))
        return fail(MPS_ERR_ARG, "mps_cgemm: bad arguments");
    GemmArgs g{m, n, k, reinterpret_cast<const cf*>(a), sam, sak, conj_a ? 1 : 0,
               reinterpret_cast<const cf*>(b), sbk, sbn, conj_b ? 1 : 0,
               reinterpret_cast<cf*>(c), scm, scn, batch, bsa, bsb, bsc};
    return cgemm(g, s);
}

namespace {

// Elements of the products T_i and V_i of every site (each 16-byte aligned).
size_t marginal_cells(const int* chis, int n, int d) {
    size_t cells = 0;
    for (int i = 0; i < n; ++i) cells += align_up((size_t)chis[i] * d * chis[i + 1], 2);
    return cells;
}

size_t marginal_bytes(size_t cells, int n, int d) {
    return align_up(cells * sizeof(cf) + (size_t)n * d * sizeof(float) + 1024, 256);
}

int max_bond(const int* chis, int n) {
    int mx = 1;
    for (int i = 0; i <= n; ++i) mx = max(mx, chis[i]);
    return mx;
}

// Scratch of the two routes of mps_site_marginals: both products of every site (twice
// the state), or the left environments (1 / d of it) and the products of one site.
size_t marginal_bytes_kept(const int* chis, int n, int d) {
    const size_t mx = max_bond(chis, n);
    return marginal_bytes(2 * marginal_cells(chis, n, d) + 4 * mx * mx, n, d);
}
size_t marginal_bytes_lean(const int* chis, int n, int d) {
    const size_t mx = max_bond(chis, n);
    size_t envs = 0;
    for (int i = 0; i < n; ++i) envs += (size_t)chis[i] * chis[i];
    return marginal_bytes(envs + 2 * mx * mx + 2 * mx * d * mx, n, d);
}

// Keeping every site's products saves forming one of the two again and lets the two
// sweeps run side by side (48 sites chi=128, 0.90 ms against 3.16; 120 sites chi=700,
// 57 against 175), but takes twice the state, and the caller's pool holds on to
// it: only up to this much scratch, 6% of the memory.  A state beyond (more than 8
// GiB) could otherwise no longer be sampled where it takes up much of the device.
constexpr size_t kMarginalKept = (size_t)16 << 30;
bool marginals_kept(const int* chis, int n, int d) {
    return marginal_bytes_kept(chis, n, d) <= max(kMarginalKept, marginal_bytes_lean(chis, n, d));
}

// The sums of sites i0 .. i0 + count - 1 (at most kMarginalBatch) into probs_dev.
int launch_marginals(const MarginalArgs& a, int count, int d, float* probs_dev, cudaStream_t s) {
    marginal_kernel<<<dim3(d, count), 256, 0, s>>>(a, d, probs_dev);
    MPS_LAUNCH_CHECK("marginal_kernel");
    return MPS_OK;
}

// One site's products (see mps_site_marginals): from the left environment L, T and
// the next one; from the right environment R, V and the next one.
struct MarginalLeft {
    GemmArgs t, next;
    MarginalLeft(const cf* A, int cl, int d, int cr, const cf* L, cf* T, cf* Ln)
        // T[l, (x, r')] = sum_l' L[l, l'] conj(A[l', x, r']);  L'[r, r'] = A^T T
        : t{cl, d * cr, cl, L, cl, 1, 0, A, (long long)d * cr, 1, 1, T, (long long)d * cr, 1},
          next{cr, cr, cl * d, A, 1, cr, 0, T, cr, 1, 0, Ln, cr, 1} {}
};
struct MarginalRight {
    GemmArgs v, next;
    MarginalRight(const cf* A, int cl, int d, int cr, const cf* R, cf* V, cf* Rn)
        // V[(l, x), r'] = sum_r conj(A[(l, x), r]) R[r', r];  R'[l, l'] = A V^T
        : v{cl * d, cr, cr, A, cr, 1, 1, R, 1, cr, 0, V, cr, 1},
          next{cl, cl, d * cr, A, (long long)d * cr, 1, 0, V, 1, (long long)d * cr, 0, Rn, cl, 1} {}
};

// The sweep from the left forms T at every site on its way and the one from the
// right V, side by side, a product of each in a launch.
int marginals_both_ends(const mps_c64* const* sites, const int* chis, int n, int d, cf* ws,
                        float** probs_dev, cudaStream_t s) {
    const size_t mx = max_bond(chis, n), cc = mx * mx, cells = marginal_cells(chis, n, d);
    cf* L[2] = {ws, ws + cc};
    cf* R[2] = {L[1] + cc, L[1] + 2 * cc};
    cf* T = R[1] + cc;
    cf* V = T + cells;
    *probs_dev = reinterpret_cast<float*>(V + cells);
    fill_one_kernel<<<1, 32, 0, s>>>(L[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    fill_one_kernel<<<1, 32, 0, s>>>(R[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    std::vector<size_t> off(n + 1, 0);
    for (int i = 0; i < n; ++i) off[i + 1] = off[i] + align_up((size_t)chis[i] * d * chis[i + 1], 2);
    for (int t = 0; t < n; ++t) {
        const int j = n - 1 - t, cur = t & 1;
        const MarginalLeft l(reinterpret_cast<const cf*>(sites[t]), chis[t], d, chis[t + 1], L[cur],
                             T + off[t], L[cur ^ 1]);
        const MarginalRight r(reinterpret_cast<const cf*>(sites[j]), chis[j], d, chis[j + 1], R[cur],
                              V + off[j], R[cur ^ 1]);
        if (int rc = cgemm2(l.t, r.v, s)) return rc;
        if (t + 1 < n)
            if (int rc = cgemm2(l.next, r.next, s)) return rc;
    }
    for (int i0 = 0; i0 < n; i0 += kMarginalBatch) {
        MarginalArgs a{};
        const int count = min(kMarginalBatch, n - i0);
        for (int q = 0; q < count; ++q)
            a.s[q] = MarginalSite{T + off[i0 + q], V + off[i0 + q], chis[i0 + q], chis[i0 + q + 1]};
        if (int rc = launch_marginals(a, count, d, *probs_dev + (size_t)i0 * d, s)) return rc;
    }
    return MPS_OK;
}

// The left environments first, then back from the right with each site's T again.
int marginals_lean(const mps_c64* const* sites, const int* chis, int n, int d, cf* ws,
                   float** probs_dev, cudaStream_t s) {
    const size_t mx = max_bond(chis, n), cc = mx * mx;
    std::vector<size_t> off(n + 1, 0);        // of the left environments
    for (int i = 0; i < n; ++i) off[i + 1] = off[i] + (size_t)chis[i] * chis[i];
    cf* R[2] = {ws + off[n], ws + off[n] + cc};
    cf* T = R[1] + cc;
    cf* V = T + mx * d * mx;
    *probs_dev = reinterpret_cast<float*>(V + mx * d * mx);
    fill_one_kernel<<<1, 32, 0, s>>>(ws, 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    fill_one_kernel<<<1, 32, 0, s>>>(R[0], 1);
    MPS_LAUNCH_CHECK("fill_one_kernel");
    for (int i = 0; i + 1 < n; ++i) {
        const MarginalLeft l(reinterpret_cast<const cf*>(sites[i]), chis[i], d, chis[i + 1], ws + off[i],
                             T, ws + off[i + 1]);
        if (int rc = cgemm(l.t, s)) return rc;
        if (int rc = cgemm(l.next, s)) return rc;
    }
    for (int i = n - 1, cur = 0; i >= 0; --i, cur ^= 1) {
        const cf* A = reinterpret_cast<const cf*>(sites[i]);
        const MarginalLeft l(A, chis[i], d, chis[i + 1], ws + off[i], T, nullptr);
        const MarginalRight r(A, chis[i], d, chis[i + 1], R[cur], V, R[cur ^ 1]);
        if (int rc = cgemm2(l.t, r.v, s)) return rc;
        MarginalArgs a{};
        a.s[0] = MarginalSite{T, V, chis[i], chis[i + 1]};
        if (int rc = launch_marginals(a, 1, d, *probs_dev + (size_t)i * d, s)) return rc;
        if (i > 0)
            if (int rc = cgemm(r.next, s)) return rc;
    }
    return MPS_OK;
}

}  // namespace

extern "C" size_t mps_marginals_workspace_bytes(const int* chis, int n, int d) {
    if (!chis || n < 1 || d < 1) return 0;
    return marginals_kept(chis, n, d) ? marginal_bytes_kept(chis, n, d) : marginal_bytes_lean(chis, n, d);
}

extern "C" int mps_site_marginals(void* stream, const mps_c64* const* sites, const int* chis,
                                  int n, int d, void* workspace, size_t workspace_bytes,
                                  float* probs_host) {
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (n < 1 || d < 1 || !sites || !chis || !probs_host)
        return fail(MPS_ERR_ARG, "mps_site_marginals: bad arguments");
    if (chis[0] != 1 || chis[n] != 1) return fail(MPS_ERR_ARG, "mps_site_marginals: end bonds must be 1");
    // p_i(x) = sum L_i[l,l'] A[l,x,r] conj(A[l',x,r']) R_i[r,r']: with T = L A* and
    // V the conjugate of A R (R is Hermitian), their elementwise product is all that
    // is left to sum.
    const bool kept = marginals_kept(chis, n, d) && workspace_bytes >= marginal_bytes_kept(chis, n, d);
    if (!workspace || (!kept && workspace_bytes < marginal_bytes_lean(chis, n, d)))
        return fail(MPS_ERR_WORKSPACE, "mps_site_marginals: workspace too small");
    float* probs_dev = nullptr;
    const int rc = kept ? marginals_both_ends(sites, chis, n, d, static_cast<cf*>(workspace), &probs_dev, s)
                        : marginals_lean(sites, chis, n, d, static_cast<cf*>(workspace), &probs_dev, s);
    if (rc) return rc;
    MPS_CUDA_CHECK(cudaMemcpyAsync(probs_host, probs_dev, (size_t)n * d * sizeof(float),
                                   cudaMemcpyDeviceToHost, s));
    MPS_CUDA_CHECK(cudaStreamSynchronize(s));
    return MPS_OK;
}
