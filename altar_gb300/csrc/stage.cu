// Per-stage CATMIP kernels: prior, Metropolis proposal/accept, COV β schedule,
// weighted covariance, Cholesky, multinomial resampling, scaling adaptation.
//
// Every kernel is a fixed launch shape on the caller's stream with all
// data-dependent control flow kept on the device (a "done" flag in the
// schedule state instead of host round trips), so one annealing stage can be
// captured into one CUDA graph.  All reductions run in a fixed order, so
// repeated runs are bitwise identical.
#include <cooperative_groups.h>
#include <math.h>
#include <stdint.h>

#include <mutex>

#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace ag {

constexpr int kMaxP = 32;          // parameter counts up to this use the proposal by blocks of chains
constexpr int kMaxPLarge = 512;    // largest parameter count of the stage kernels
constexpr int kGridPoints = 11;    // COV.cc:276 Nbeta = 10 -> 11 points per level
constexpr int kBrentMaxIter = 128;   // Brent iterations run on the device per stage
constexpr int kGridLevels = 11;    // COV.cc:313 Nloop <= Nbeta
constexpr int kEvalChunk = 1024;   // chains per CTA in a COV evaluation
constexpr int kSigmaChunk = 256;   // chains per CTA in the covariance

// ---------------------------------------------------------------------------
// prior
__global__ void prior_sample_kernel(int n, int p, const double* __restrict__ lo,
                                    const double* __restrict__ hi, uint64_t seed, uint32_t attempt,
                                    const uint32_t* __restrict__ redraw, double* __restrict__ theta) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (redraw && !redraw[i]) return;
    for (int j = 0; j < p; ++j) {
        u32x4 r = draw(seed, (uint32_t)i, (uint32_t)j, STREAM_PRIOR, 0u, attempt);
        double u = u01_closed_open(r.x, r.y);
        // gsl_ran_flat: a (1 - u) + b u
        theta[(size_t)i * p + j] = lo[j] * (1.0 - u) + hi[j] * u;
    }
}

// log density of the Uniform prior, the same for every chain inside the support: one warp takes
// the logarithms, a lane each, and subtracts them in parameter order (every chain's thread taking
// all p logarithms was most of the proposal's time: ~60 FP64 instructions each)
__device__ inline double uniform_log_prior(int p, const double* lo, const double* hi) {
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    for (int j0 = 0; j0 < p; j0 += 32) {
        const double l = j0 + lane < p ? log(hi[j0 + lane] - lo[j0 + lane]) : 0.0;
        const int cnt = p - j0 < 32 ? p - j0 : 32;
        for (int j = 0; j < cnt; ++j) s -= __shfl_sync(0xffffffffu, l, j);
    }
    return s;
}

__global__ void prior_llk_kernel(const double* __restrict__ theta, int n, int p,
                                 const double* __restrict__ lo, const double* __restrict__ hi,
                                 uint32_t* __restrict__ mask, double* __restrict__ prior) {
    __shared__ double s_prior;
    if (threadIdx.x < 32 && prior) {
        const double lp = uniform_log_prior(p, lo, hi);
        if (threadIdx.x == 0) s_prior = lp;
    }
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (mask) {
        bool out = false;
        for (int j = 0; j < p; ++j) {
            double v = theta[(size_t)i * p + j];
            out |= !(lo[j] <= v && v <= hi[j]);
        }
        if (out) mask[i] |= CHAIN_OUT_OF_SUPPORT;
    }
    if (prior) prior[i] = s_prior;
}

// log u > d for u in (0, 1]: decided in FP32 unless the two are closer than that logarithm's error
// (u rounds to FP32 within 2^-24 of itself and logf is good to 2 ulp: below 1e-6 (1 + |log u|)).
// The FP64 logarithm was a quarter of accept_kernel: 4,096 chains 7.7 -> 5.7 µs.
__device__ inline bool log_exceeds(double u, double d) {
    const float l = logf((float)u);
    const double gap = (double)l - d;
    if (fabs(gap) > 1e-5 * (1.0 + fabs((double)l))) return gap > 0.0;
    return log(u) > d;
}

// the acceptance floor of a chain inside the support from its post + log u (accept_floor_kernel)
__device__ inline double floor_of(double post_logu, double cprior, double b) {
    double f = (post_logu - cprior) / b;
    f -= (fabs(f) + 1.0) * 1e-9;
    return f == f ? f : -INFINITY;
}

// ---------------------------------------------------------------------------
// Metropolis proposal, verify and prior (Metropolis.py:160-183, 236-259).  A block takes
// kProposeChains chains: a thread per pair of normals (a logarithm, a square root and a sine and
// cosine, ~150 dependent FP64 instructions: one thread per chain took its pairs one after
// another), then a thread per entry of L z, summed over k in order as a thread per chain does,
// then the rows, replaced by θ where an entry left the support.  Measured:
// 4,096 chains, 6 parameters 7.3 µs (23.5 µs with a thread per chain); 1,024 chains, 4 parameters
// 7.0 µs (16.4 µs).
//
// ACCEPT: first accepts or rejects the previous step's candidates, as accept_kernel does, in a warp
// of its own beside the normals, and forms the new candidates' floors, as accept_floor_kernel does.
// Each is a launch of 5 to 6 µs, nearly all latency; the kernel takes 7.5 µs with and 7.4 without them, and
// a Reverso run of 4,096 chains and 20 steps per stage 4.3 ms instead of 4.6.
constexpr int kProposeChains = 32;
struct AcceptArgs {
    const double *beta, *cdata;
    double *prior, *data, *post;
    unsigned long long* counters;
    double* floor;                             // null: none wanted
};
template <bool ACCEPT> constexpr int kProposeThreads = ACCEPT ? 224 : 192;

template <bool ACCEPT>
__global__ void __launch_bounds__(kProposeThreads<ACCEPT>)
propose_kernel(double* theta, int n, int p, const double* __restrict__ chol,
               const double* __restrict__ lo, const double* __restrict__ hi, uint64_t seed, uint32_t step,
               const uint32_t* __restrict__ epoch, double* cand, uint32_t* mask, double* cprior, int chain0,
               AcceptArgs acc) {
    constexpr int kThreads = kProposeThreads<ACCEPT>;
    __shared__ double sz[kProposeChains * kMaxP], sv[kProposeChains * kMaxP], sL[kMaxP * kMaxP];
    __shared__ double s_prior, s_floor[kProposeChains];
    __shared__ int s_out[kProposeChains], s_take[kProposeChains];
    const int tid = threadIdx.x, i0 = blockIdx.x * kProposeChains;
    const int chains = n - i0 < kProposeChains ? n - i0 : kProposeChains;
    const uint32_t ep = *epoch;
    const int pairs = (p + 1) >> 1;
    for (int k = tid; k < p * p; k += kThreads) sL[k] = chol[k];
    if (tid < kProposeChains) s_out[tid] = 0;
    if (tid >= kThreads - 32) {                // the last warp has the fewest pairs
        const double lp = uniform_log_prior(p, lo, hi);
        if (tid == kThreads - 1) s_prior = lp;
    } else if (ACCEPT && tid >= kThreads - 64) {
        const int c = tid & 31, i = i0 + c;
        int kind = 3;                          // accepted, rejected, unlikely
        if (c < chains) {
            double now = acc.post[i];
            kind = 1;
            if (!mask[i]) {
                const double b = *acc.beta;
                const double cp = cprior[i] + b * acc.cdata[i];
                const u32x4 r = draw(seed, (uint32_t)(chain0 + i), 0u, STREAM_ACCEPT, step - 1, ep);
                kind = log_exceeds(u01_open_closed(r.x, r.y), cp - now) ? 2 : 0;
                if (kind == 0) {
                    acc.prior[i] = cprior[i];
                    acc.data[i] = acc.cdata[i];
                    acc.post[i] = now = cp;
                }
            }
            s_take[c] = kind == 0;
            if (acc.floor) {
                const u32x4 r = draw(seed, (uint32_t)(chain0 + i), 0u, STREAM_ACCEPT, step, ep);
                s_floor[c] = now + log(u01_open_closed(r.x, r.y));
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, kind == k);
            if (c == k && m) atomicAdd(&acc.counters[k], (unsigned long long)__popc(m));
        }
    }
    for (int t = tid; t < chains * pairs; t += kThreads) {
        const int c = t / pairs, j = 2 * (t - c * pairs);
        double z0, z1;
        normal_pair(draw(seed, (uint32_t)(chain0 + i0 + c), (uint32_t)(j >> 1), STREAM_PROPOSAL, step, ep), z0, z1);
        sz[c * p + j] = z0;
        if (j + 1 < p) sz[c * p + j + 1] = z1;
    }
    __syncthreads();
    double* th = theta + (size_t)i0 * p;
    double* cd = cand + (size_t)i0 * p;
    for (int t = tid; t < chains * p; t += kThreads) {
        const int c = t / p, j = t - c * p;
        double d = 0.0;
        for (int k = 0; k <= j; ++k) d = fma(sL[j * p + k], sz[c * p + k], d);
        if (ACCEPT && s_take[c]) th[t] = cd[t];
        const double v = th[t] + d;
        sv[t] = v;
        if (!(lo[j] <= v && v <= hi[j])) s_out[c] = 1;
    }
    __syncthreads();
    for (int t = tid; t < chains * p; t += kThreads) cd[t] = s_out[t / p] ? th[t] : sv[t];
    if (tid < chains) {
        mask[i0 + tid] = s_out[tid] ? CHAIN_OUT_OF_SUPPORT : 0u;
        cprior[i0 + tid] = s_prior;
        if (ACCEPT && acc.floor) {
            const double b = *acc.beta;
            acc.floor[i0 + tid] = !s_out[tid] && b > 0.0 ? floor_of(s_floor[tid], s_prior, b) : -INFINITY;
        }
    }
}

// The same proposal for many parameters: one warp per chain, the chain's normals in
// shared memory, lane j computing the rows j, j + 32, ... of L z with the same
// sequential k order as propose_kernel (identical results).
constexpr int kProposeWarps = 8;
__global__ void __launch_bounds__(kProposeWarps * 32)
propose_warp_kernel(const double* __restrict__ theta, int n, int p, const double* __restrict__ chol,
                    const double* __restrict__ lo, const double* __restrict__ hi, uint64_t seed,
                    uint32_t step, const uint32_t* __restrict__ epoch, double* __restrict__ cand,
                    uint32_t* __restrict__ mask, double* __restrict__ cprior, int chain0) {
    extern __shared__ double sz[];                 // [kProposeWarps][p] normals
    __shared__ double s_prior;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * kProposeWarps + warp;
    if (warp == 0) {
        const double lp = uniform_log_prior(p, lo, hi);
        if (lane == 0) s_prior = lp;
    }
    __syncthreads();
    if (i >= n) return;
    double* z = sz + (size_t)warp * p;
    const uint32_t ep = *epoch;
    for (int q = lane; 2 * q < p; q += 32) {
        double z0, z1;
        normal_pair(draw(seed, (uint32_t)(chain0 + i), (uint32_t)q, STREAM_PROPOSAL, step, ep), z0, z1);
        z[2 * q] = z0;
        if (2 * q + 1 < p) z[2 * q + 1] = z1;
    }
    __syncwarp();
    const double* th = theta + (size_t)i * p;
    double* c = cand + (size_t)i * p;
    bool out = false;
    for (int j = lane; j < p; j += 32) {
        const double* row = chol + (size_t)j * p;
        double d = 0.0;
        for (int k = 0; k <= j; ++k) d = fma(row[k], z[k], d);
        const double v = th[j] + d;
        c[j] = v;
        out |= !(lo[j] <= v && v <= hi[j]);
    }
    out = __any_sync(0xffffffffu, out);
    if (out)
        for (int j = lane; j < p; j += 32) c[j] = th[j];
    if (lane == 0) {
        mask[i] = out ? CHAIN_OUT_OF_SUPPORT : 0u;
        cprior[i] = s_prior;
    }
}

// ---------------------------------------------------------------------------
// Metropolis accept/reject (Metropolis.py:185-223)
__global__ void accept_kernel(int n, int p, const double* __restrict__ beta, uint64_t seed,
                              uint32_t step, const uint32_t* __restrict__ epoch,
                              const uint32_t* __restrict__ mask, const double* __restrict__ cand,
                              const double* __restrict__ cprior, const double* __restrict__ cdata,
                              double* __restrict__ theta, double* __restrict__ prior,
                              double* __restrict__ data, double* __restrict__ post,
                              unsigned long long* __restrict__ counters, int chain0) {
    __shared__ unsigned int s_cnt[3];
    if (threadIdx.x < 3) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        if (mask[i]) {
            atomicAdd(&s_cnt[1], 1u);
        } else {
            const double b = *beta;
            const double cp = cprior[i] + b * cdata[i];
            u32x4 r = draw(seed, (uint32_t)(chain0 + i), 0u, STREAM_ACCEPT, step, *epoch);
            if (log_exceeds(u01_open_closed(r.x, r.y), cp - post[i])) {
                atomicAdd(&s_cnt[2], 1u);
            } else {
                atomicAdd(&s_cnt[0], 1u);
                for (int j = 0; j < p; ++j) theta[(size_t)i * p + j] = cand[(size_t)i * p + j];
                prior[i] = cprior[i];
                data[i] = cdata[i];
                post[i] = cp;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_cnt[threadIdx.x])
        atomicAdd(&counters[threadIdx.x], (unsigned long long)s_cnt[threadIdx.x]);
}

// The data log-likelihood below which each proposal is certainly rejected (early rejection,
// Solonen et al. 2012, Bayesian Analysis 7(3)).  accept_kernel rejects when
// log u > cprior + β cdata − post; with the same uniform u, every cdata below
// (post + log u − cprior)/β is rejected.  The floor is lowered by a relative 1e-9 so that a
// likelihood evaluation stopped below it is rejected whatever the rounding of the test;
// chains outside the support, and β = 0, get -inf (never stopped).
__global__ void accept_floor_kernel(int n, const double* __restrict__ beta, uint64_t seed, uint32_t step,
                                    const uint32_t* __restrict__ epoch, const uint32_t* __restrict__ mask,
                                    const double* __restrict__ cprior, const double* __restrict__ post,
                                    double* __restrict__ floor, int chain0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double b = *beta;
    double f = -INFINITY;
    if (!mask[i] && b > 0.0) {
        u32x4 r = draw(seed, (uint32_t)(chain0 + i), 0u, STREAM_ACCEPT, step, *epoch);
        f = floor_of(post[i] + log(u01_open_closed(r.x, r.y)), cprior[i], b);
    }
    floor[i] = f;
}

__global__ void posterior_kernel(int n, const double* __restrict__ beta,
                                 const double* __restrict__ prior, const double* __restrict__ data,
                                 double* __restrict__ post) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) post[i] = prior[i] + (*beta) * data[i];
}

// ---------------------------------------------------------------------------
// COV β schedule (COV.cc:222-368).
struct CovState {
    double median;
    double llk_max;
    double beta0;          // β at the start of the stage
    double low, high, step;
    double pts[2];         // points of the next round (round 0, Brent)
    double cov_high;       // COV at the full remaining δβ
    double dbeta;          // chosen δβ
    double cov;            // COV at dbeta
    double s1;             // shifted weight sum at dbeta
    int npts;              // points to evaluate in the next round
    int level;             // levels done (Nloop)
    int done;
    int skip;              // jumped straight to β = 1
    // Brent's method (minimisation of (COV - target)² on [low, high])
    double a, b, x, w, v, fx, fw, fv, d, e, u;
    int iter;
    int phase;             // 0: evaluating the initial point, 1: iterating
};

// blocks of the schedule kernel for n chains, and the partial sums one round of it writes
constexpr int kCovBlocks = 152;
// up to this many blocks form one cluster, whose barrier is hardware's; few chains are spread over it
constexpr int kCovCluster = 8;
__host__ __device__ constexpr int cov_blocks(int n) {
    return n <= 256 * kCovCluster ? (n <= 128 * kCovCluster ? (n + 127) / 128 : kCovCluster)
           : (n + 255) / 256 < kCovBlocks ? (n + 255) / 256 : kCovBlocks;
}
// a block's share of the chains, whole warps of them
__device__ __forceinline__ long cov_share(int n) { return ((n + gridDim.x - 1) / gridDim.x + 31) / 32 * 32; }
__host__ __device__ constexpr size_t cov_round_partials(int n) {
    // a grid level's moments per block, or Brent's two points per chunk
    const size_t level = (size_t)2 * kGridPoints * cov_blocks(n), brent = 4 * (size_t)((n + kEvalChunk - 1) / kEvalChunk);
    return level > brent ? level : brent;
}
__host__ __device__ constexpr size_t cov_part_doubles(int n) {
    return 2 * cov_round_partials(n) + 2 * (size_t)((n + kEvalChunk - 1) / kEvalChunk);
}

// order-preserving map of a double onto uint64
__device__ inline uint64_t dkey(double x) {
    uint64_t b = (uint64_t)__double_as_longlong(x);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ inline double dkey_inv(uint64_t k) {
    uint64_t b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
    return __longlong_as_double((long long)b);
}

// Median and maximum of llk, one CTA.  The range of the keys that can hold the wanted rank is
// cut into 2^11 buckets of equal width (in key space), counted in shared memory, and narrowed to
// one bucket; once a bucket holds at most kMedianList keys they are collected and ranked against
// each other.  Starting from the keys' own range, the log-likelihoods of a stage take one or two
// counting passes (a radix select over the fixed bytes of the key took 16): 32,768 values in
// 23 µs (129 µs), 1,024 in 11 µs (50 µs).  The passes are bound by the latency of reading llk from L2 on one SM.
constexpr int kMedianThreads = 1024;
constexpr int kMedianBits = 11;
constexpr int kMedianList = 128;        // 8 threads rank each key

template <class F>
__device__ __forceinline__ void median_each(const double* __restrict__ llk, int n, F f) {
    for (long i0 = threadIdx.x; i0 < n; i0 += 8 * kMedianThreads) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const long i = i0 + (long)q * kMedianThreads;
            v[q] = i < n ? __ldg(llk + i) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (i0 + (long)q * kMedianThreads < n) f(dkey(v[q]));
    }
}

__device__ inline uint64_t u64_min(uint64_t a, uint64_t b) { return a < b ? a : b; }
__device__ inline uint64_t u64_max(uint64_t a, uint64_t b) { return a > b ? a : b; }

__global__ void __launch_bounds__(kMedianThreads) cov_median_kernel(const double* __restrict__ llk, int n,
                                                                    const double* __restrict__ beta,
                                                                    CovState* __restrict__ S) {
    after_previous();
    __shared__ int s_hist[1 << kMedianBits];
    __shared__ uint64_t s_list[kMedianList];
    __shared__ uint64_t s_a[32], s_b[32];
    __shared__ double s_max[32];
    __shared__ int s_warp[32];
    __shared__ uint64_t s_key[2];
    __shared__ int s_bucket, s_before, s_count, s_fill;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // smallest and largest key; the maximum as fmax has it (NaN left out)
    uint64_t mn = ~0ull, mx = 0ull;
    uint64_t big = dkey(-INFINITY);
    median_each(llk, n, [&](uint64_t k) {
        mn = u64_min(mn, k);
        mx = u64_max(mx, k);
        if (k <= dkey(INFINITY)) big = u64_max(big, k);
    });
    double top = dkey_inv(big);
    for (int o = 16; o > 0; o >>= 1) {
        mn = u64_min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = u64_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if (lane == 0) {
        s_a[warp] = mn;
        s_b[warp] = mx;
        s_max[warp] = top;
    }
    __syncthreads();
    uint64_t lo = s_a[lane], hi = s_b[lane];
    for (int o = 16; o > 0; o >>= 1) {
        lo = u64_min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = u64_max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    // rank k among the `count` keys in [lo, lo + range]
    uint64_t range = hi - lo;
    int k = (n - 1) / 2, count = n;
    while (range > 0 && count > kMedianList) {
        const int width = 64 - __clzll((long long)range);
        const int shift = width > kMedianBits ? width - kMedianBits : 0;
        for (int b = tid; b < 1 << kMedianBits; b += kMedianThreads) s_hist[b] = 0;
        __syncthreads();
        median_each(llk, n, [&](uint64_t key) {
            if (key - lo <= range) atomicAdd(&s_hist[(key - lo) >> shift], 1);
        });
        __syncthreads();
        // the bucket of rank k: two buckets per thread
        const int h0 = s_hist[2 * tid], h1 = s_hist[2 * tid + 1];
        int s = h0 + h1;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane == 31) s_warp[warp] = s;
        __syncthreads();
        int w = lane < warp ? s_warp[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        const int before = w + s - h0 - h1;
        if (k >= before && k < before + h0 + h1) {
            const bool second = k >= before + h0;
            s_bucket = 2 * tid + second;
            s_before = before + (second ? h0 : 0);
            s_count = second ? h1 : h0;
        }
        __syncthreads();
        lo += (uint64_t)s_bucket << shift;
        range = (1ull << shift) - 1;           // may reach past hi: no keys lie there
        k -= s_before;
        count = s_count;
        __syncthreads();
    }
    // klo, the key of rank (n-1)/2; khi, the next one of rank n/2 (gsl_stats_median_from_sorted_data)
    if (tid == 0) {
        s_fill = 0;
        s_key[0] = s_key[1] = lo;
    }
    __syncthreads();
    if (range > 0) {
        median_each(llk, n, [&](uint64_t key) {
            if (key - lo <= range) s_list[atomicAdd(&s_fill, 1)] = key;
        });
        __syncthreads();
        const int c = tid >> 3;
        const uint64_t key = s_list[c < count ? c : 0];
        int rank = 0;
        for (int j = tid & 7; j < count; j += 8) {
            const uint64_t other = s_list[j];
            rank += other < key || (other == key && j < c);
        }
        for (int o = 4; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
        if (c < count) {
            if (rank == k) s_key[0] = key;
            if (rank == k + 1) s_key[1] = key;
        }
        __syncthreads();
    }
    if (n % 2 == 0 && k + 1 >= count) {
        // the next key lies beyond the bucket
        uint64_t next = ~0ull;
        const uint64_t last = lo + range < lo ? ~0ull : lo + range;
        median_each(llk, n, [&](uint64_t key) {
            if (key > last) next = u64_min(next, key);
        });
        for (int o = 16; o > 0; o >>= 1) next = u64_min(next, __shfl_xor_sync(0xffffffffu, next, o));
        if (lane == 0) s_a[warp] = next;
        __syncthreads();
        if (tid == 0) {
            for (int j = 1; j < 32; ++j) next = u64_min(next, s_a[j]);
            s_key[1] = next;
        }
    }
    if (tid == 0) {
        double m = s_max[0];
        for (int w = 1; w < 32; ++w) m = fmax(m, s_max[w]);
        const double vlo = dkey_inv(s_key[0]), vhi = dkey_inv(s_key[1]);
        S->median = (n % 2) ? vlo : (vlo + vhi) / 2.0;
        S->llk_max = m;
        S->beta0 = *beta;
        S->low = 0.0;
        S->high = 1.0 - *beta;
        S->step = 0.0;
        S->pts[0] = S->high;     // round 0 evaluates the full remaining step
        S->npts = 1;
        S->level = 0;
        S->done = 0;
        S->skip = 0;
    }
}

// Σe and Σe² over one chunk of kEvalChunk chains (in thread 0's out): 256 threads each sum their
// chains in index order, then the warps' sums are added in warp order
template <class F>
__device__ void chunk_sums(int n, int chunk, F value, double (&out)[2]) {
    __shared__ double r1[8], r2[8];
    double s1 = 0.0, s2 = 0.0;
    const int begin = chunk * kEvalChunk;
    const int end = min(n, begin + kEvalChunk);
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const double e = value(i);
        s1 += e;
        s2 = fma(e, e, s2);
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if ((threadIdx.x & 31) == 0) {
        r1[threadIdx.x >> 5] = s1;
        r2[threadIdx.x >> 5] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            a += r1[w];
            b += r2[w];
        }
        out[0] = a;
        out[1] = b;
    }
    __syncthreads();      // r1 and r2 are reused by the next chunk
}

// the shifted weight moments, e = exp(g (llk − median) − g (llk_max − median)), of one chunk
__device__ void chunk_moments(const double* __restrict__ llk, int n, double g, double med, double llk_max, int chunk,
                              double (&out)[2]) {
    const double mx = g * (llk_max - med);
    chunk_sums(n, chunk, [&](int i) { return exp(g * (llk[i] - med) - mx); }, out);
}

// COV of the normalised weights from the shifted moments, with the reference's
// convention that a non-finite COV counts as 1e100 (COV.cc:355-364)
__device__ double cov_from_moments(double s1, double s2, double mx, int n) {
    // an infinite weight in the reference (exp overflow) or an infinite weight sum (the sum is at
    // most n: neither is possible for the small exponents)
    if (!(s1 > 0.0)) return 1e100;
    if (mx > 600.0 && (isinf(exp(mx)) || isinf(exp(mx) * s1))) return 1e100;
    double v = (s2 / (s1 * s1) - 1.0 / n) / (double)(n - 1);
    if (v < 0.0) v = 0.0;
    double c = (double)n * sqrt(v);
    if (!isfinite(c)) return 1e100;
    return c;
}

// Where the COV of a point lies against the target: 0 at most target - tol, 1 within tol of the
// target, 2 above.  COV = n sqrt((Σe²/(Σe)² − 1/n)/(n − 1)) >= c is Σe² >= X(c) (Σe)² with
// X(c) = (c/n)² (n − 1) + 1/n, so a decision takes a product and a comparison where the COV itself
// takes two divisions and a square root (~4,000 cycles of dependent FP64).
__device__ double cov_threshold(double c, int n) {
    const double r = c / (double)n;
    return c < 0.0 ? -1.0 : r * r * (double)(n - 1) + 1.0 / n;
}

__device__ int cov_class(double s1, double s2, double mx, double below, double above) {
    // the reference's 1e100: no weights, an infinite weight or weight sum, a NaN
    if (!(s1 > 0.0)) return 2;
    if (mx > 600.0 && (isinf(exp(mx)) || isinf(exp(mx) * s1))) return 2;
    const double q = s1 * s1;
    return s2 <= below * q ? 0 : s2 < above * q ? 1 : 2;
}

// One level of the grid search (COV.cc:240-326): round 0 evaluated the full remaining step (cls is
// its class), later rounds the kGridPoints points of a level; hit is the first point of the level
// that is not below the target (kGridPoints if none), cls its class.
__device__ void grid_step(CovState& S, int hit, int cls) {
    const double Nbeta = 10.0;
    if (S.level == 0) {
        // skip straight to β = 1 (COV.cc:257-268)
        if (cls < 2) {
            S.done = 1;
            S.skip = 1;
            S.dbeta = S.high;
            return;
        }
    } else {
        // scan of one level (COV.cc:287-311); the points are low, low + step, ... accumulated as the
        // reference does.  A completed scan leaves the reference's accumulator one step past the
        // last point and steps it back (COV.cc:301), which can differ from that point in the last bit
        const double step = S.step;
        double guess = S.low;
        for (int k = 0; k < hit; ++k) guess += step;
        if (hit == kGridPoints) guess -= step;
        S.high = guess;
        S.low = guess - step;
        if (cls == 1 || hit == 0 || S.level >= kGridLevels) {
            S.done = 1;
            S.dbeta = guess;
            return;
        }
    }
    S.level += 1;
    S.step = (S.high - S.low) / Nbeta;
}

// Brent's minimiser for δβ (COV.cc:58-219).  The reference minimises f(δβ) = (COV − target)²
// with GSL's Brent minimiser, primed with the guess δβ = 5e-5 inside [0, 1 − β], and stops
// when the COV at the latest evaluated point is within tol of the target (or after maxiter
// iterations), returning the best point found.  GSL is not part of the reference, so the
// iteration itself is Brent's published method (R. P. Brent, "Algorithms for Minimization
// without Derivatives", 1973, ch. 5, procedure localmin: parabolic interpolation through the
// three best points, golden-section steps when the parabola is unacceptable) restated here.
// One call per evaluation round: the COVs of the points of the previous round come in as
// cov[], the next point goes out through S.pts.
__device__ inline double brent_metric(double cov, double target) {
    return (cov >= 1e100) ? 1e100 : (cov - target) * (cov - target);
}

__device__ void brent_step(CovState& S, const double* cov, double target, double tol, int maxiter) {
    const double golden = 0.3819660112501051;      // (3 − √5) / 2
    if (S.level == 0) {
        // full remaining step first: skip straight to β = 1 if it meets the target (COV.cc:103-116)
        S.cov_high = cov[0];
        if (cov[0] < target || fabs(cov[0] - target) < tol) {
            S.done = 1;
            S.skip = 1;
            S.dbeta = S.high;
            return;
        }
        // bracket [0, 1 − β], first point the reference's guess, interior point v = w at the
        // golden section of the bracket; both evaluated in the next round
        S.level = 1;
        S.a = 0.0;
        S.b = S.high;
        S.x = (5.0e-5 < S.high) ? 5.0e-5 : 0.5 * S.high;
        S.v = S.w = S.a + golden * (S.b - S.a);
        S.d = S.e = 0.0;
        S.iter = 0;
        S.phase = 0;
        S.pts[0] = S.x;
        S.pts[1] = S.v;
        S.npts = 2;
        return;
    }
    if (S.phase == 0) {
        S.fx = brent_metric(cov[0], target);
        S.fv = S.fw = brent_metric(cov[1], target);
        S.phase = 1;
    } else {
        // fold the new point u into the bracket and the three best points
        const double u = S.u, fu = brent_metric(cov[0], target);
        if (fu <= S.fx) {
            if (u < S.x) S.b = S.x; else S.a = S.x;
            S.v = S.w; S.fv = S.fw;
            S.w = S.x; S.fw = S.fx;
            S.x = u; S.fx = fu;
        } else {
            if (u < S.x) S.a = u; else S.b = u;
            if (fu <= S.fw || S.w == S.x) {
                S.v = S.w; S.fv = S.fw;
                S.w = u; S.fw = fu;
            } else if (fu <= S.fv || S.v == S.x || S.v == S.w) {
                S.v = u; S.fv = fu;
            }
        }
        S.iter += 1;
        // the reference's convergence test is on the COV of the latest point (COV.cc:182)
        if (fabs(cov[0] - target) < tol || S.iter >= maxiter) {
            S.done = 1;
            S.dbeta = S.x;
            return;
        }
    }
    // next point
    const double x = S.x, a = S.a, b = S.b;
    const double xm = 0.5 * (a + b);
    const double tol1 = 1.4901161193847656e-08 * fabs(x) + 1e-15;   // √ε·|x| plus an absolute floor
    const double tol2 = 2.0 * tol1;
    if (fabs(x - xm) <= tol2 - 0.5 * (b - a)) {                     // bracket down to the tolerance
        S.done = 1;
        S.dbeta = x;
        return;
    }
    double d = S.d, e = S.e;
    bool parabolic = false;
    if (fabs(e) > tol1) {
        double r = (x - S.w) * (S.fx - S.fv);
        double q = (x - S.v) * (S.fx - S.fw);
        double pp = (x - S.v) * q - (x - S.w) * r;
        q = 2.0 * (q - r);
        if (q > 0.0) pp = -pp; else q = -q;
        const double e_prev = e;
        e = d;
        if (fabs(pp) < fabs(0.5 * q * e_prev) && pp > q * (a - x) && pp < q * (b - x)) {
            d = pp / q;
            const double u = x + d;
            if (u - a < tol2 || b - u < tol2) d = (xm >= x) ? tol1 : -tol1;
            parabolic = true;
        }
    }
    if (!parabolic) {
        e = (x >= xm) ? a - x : b - x;
        d = golden * e;
    }
    const double u = (fabs(d) >= tol1) ? x + d : x + ((d >= 0.0) ? tol1 : -tol1);
    S.d = d;
    S.e = e;
    S.u = u;
    S.pts[0] = u;
    S.npts = 1;
}

// Grid-wide barrier of a cooperative launch (every block of the grid is resident).  The
// barrier words (arrival count, generation) are cleared by the host before the launch and
// the count returns to zero at every barrier.  A block that waits more than kBarrierLimit
// polls raises DEV_ERR_TIMEOUT and returns false; every later barrier then gives up too, so a
// lost block ends the kernel with the flag set instead of hanging it.
constexpr uint32_t kBarrierLimit = 1u << 22;
struct __align__(256) GridBarrier {
    unsigned count;
    unsigned gen;
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ bool grid_sync(GridBarrier* bar, uint32_t* flags) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = ld_acquire_gpu(&bar->gen);
        __threadfence();
        int ok = 1;
        if (atomicAdd(&bar->count, 1u) == gridDim.x - 1) {
            atomicExch(&bar->count, 0u);
            __threadfence();
            atomicAdd(&bar->gen, 1u);
        } else {
            uint32_t polls = 0;
            while (ld_acquire_gpu(&bar->gen) == gen) {
                if (++polls > kBarrierLimit) {
                    ok = 0;
                    raise_flag(flags, DEV_ERR_TIMEOUT);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Sum of each of N <= 32 per-lane values over the warp: after the call, v[0] of lane l holds the
// sum of value l (bit-reversed halving: 31 additions per lane where N butterflies take 5 N)
template <int N>
__device__ __forceinline__ void warp_sum_each(double (&v)[N], int lane) {
    static_assert(N <= 32, "one value per lane");
#pragma unroll
    for (int h = 16; h > 0; h >>= 1) {
        const bool up = lane & h;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double a = i < N ? v[i < N ? i : 0] : 0.0, b = i + h < N ? v[i + h < N ? i + h : 0] : 0.0;
            const double got = __shfl_xor_sync(0xffffffffu, up ? a : b, h);
            if (i < N) v[i < N ? i : 0] = (up ? b : a) + got;
        }
    }
}

// Moments Σe and Σe², e = exp(g (llk − llk_max)), of this block's share of the chains at the
// points of one grid level, pts[k] ≈ low + k step: e at successive points is a geometric
// sequence, so a chain takes two exponentials and ten products instead of eleven exponentials
// (FP64: 64 cycles per warp instruction and SM quarter is what bounds a round).  They only choose
// among the grid points; the COV and the weights reported for the chosen δβ come from
// exponentials of their own.
template <int POINTS>
__device__ void level_moments(const double* __restrict__ llk, int n, double low, double step, double llk_max,
                              double* __restrict__ out, int stride) {
    constexpr int N = 2 * POINTS;
    __shared__ double s_part[8][N];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double m[N];
#pragma unroll
    for (int k = 0; k < N; ++k) m[k] = 0.0;
    const long share = cov_share(n), end = min((long)n, (blockIdx.x + 1) * share);
    for (long i = blockIdx.x * share + threadIdx.x; i < end; i += blockDim.x) {
        const double y = llk[i] - llk_max;
        double e = exp(low * y);
        const double f = POINTS > 1 ? exp(step * y) : 1.0;
#pragma unroll
        for (int k = 0; k < POINTS; ++k) {
            m[2 * k] += e;
            m[2 * k + 1] = fma(e, e, m[2 * k + 1]);
            if (k + 1 < POINTS) e *= f;
        }
    }
    warp_sum_each(m, lane);
    if (lane < N) s_part[warp][lane] = m[0];
    __syncthreads();
    if (threadIdx.x < N) {
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) a += s_part[w][threadIdx.x];
        out[(size_t)threadIdx.x * stride] = a;
    }
}

// The whole δβ search of one stage and its weights in one cooperative launch (COV.cc:58-368).
// Each round, the blocks evaluate the moments of the round's points, meet at a grid barrier, and
// then every block adds the partials in a fixed order and takes the same decision on its own
// copy of the search state, so a round needs one barrier.  A grid level has one partial per
// block and moment, spread over the whole GPU; Brent's single points one per chunk of
// kEvalChunk chains.  The partials alternate between two buffers, so a block that starts the next
// round cannot overwrite partials that a slower block is still adding.  Then the exponentials at
// the chosen δβ, their moments per chunk in chunk order, and the normalised weights.
// With few chains a round is a chain of dependent FP64 instructions (67 cycles each) and the
// barrier; with many the exponentials add to that.  Measured:
// 32,768 chains 110 µs (352 µs with eleven exponentials per chain and level and the eleven COVs
// formed in a row), 1,024 chains 70 µs without a cluster (177 µs).
// CLUSTER: the blocks are one cluster (up to 2,048 chains; Brent 4,096) and meet at its barrier, which
// needs no cooperative launch and no words to clear: 1,024 chains 51 µs.  4,096 chains, 53 µs in 16
// blocks, would have two per thread in a cluster of eight.
template <bool BRENT, bool CLUSTER>
__global__ void __launch_bounds__(256) cov_schedule_kernel(const double* __restrict__ llk, int n, double target,
                                                           double tol, int maxiter, int rounds,
                                                           CovState* __restrict__ S, double* __restrict__ part,
                                                           GridBarrier* __restrict__ bar, double* __restrict__ beta,
                                                           double* __restrict__ dbeta_cov, double* __restrict__ w,
                                                           uint32_t* __restrict__ flags) {
    if (CLUSTER) after_previous();
    auto meet = [&]() {
        if constexpr (CLUSTER) {
            cg::this_cluster().sync();        // orders the global writes before it, cluster-wide
            return true;
        } else {
            return grid_sync(bar, flags);
        }
    };
    __shared__ CovState sS;
    __shared__ double s_tot[2 * kGridPoints], s_limit[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) sS = *S;                // median, maximum and the first round's point
    if (!BRENT && (tid == 32 || tid == 64)) {
        const double t = tol > 0.0 ? tol : 0.0;
        s_limit[tid >> 6] = cov_threshold(tid == 32 ? target - t : target + t, n);
    }
    __syncthreads();
    const int nblk = (n + kEvalChunk - 1) / kEvalChunk;
    const size_t pbuf = cov_round_partials(n);
    const double med = sS.median, lmax = sS.llk_max;
    for (int round = 0; round < rounds && !sS.done; ++round) {
        double* pr = part + (size_t)(round & 1) * pbuf;
        if constexpr (!BRENT) {
            const int points = round == 0 ? 1 : kGridPoints, parts = gridDim.x;
            const double low = sS.low, step = sS.step;
            if (round == 0)
                level_moments<1>(llk, n, sS.high, 0.0, lmax, pr + blockIdx.x, parts);
            else
                level_moments<kGridPoints>(llk, n, low, step, lmax, pr + blockIdx.x, parts);
            if (!meet()) return;
            // eight lanes per moment
            const int q = tid >> 3;
            double a = 0.0;
            if (q < 2 * points) {
#pragma unroll 4
                for (int k = tid & 7; k < parts; k += 8) a += __ldcg(pr + (size_t)q * parts + k);
            }
            for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (q < 2 * points && (tid & 7) == 0) s_tot[q] = a;
            __syncthreads();
            if (warp == 0) {
                int cls = 0;
                if (lane < points) {
                    const double g = round == 0 ? sS.high : low + lane * step;
                    cls = cov_class(s_tot[2 * lane], s_tot[2 * lane + 1], g * (lmax - med), s_limit[0], s_limit[1]);
                }
                const unsigned up = __ballot_sync(0xffffffffu, cls > 0);
                const int hit = up ? __ffs(up) - 1 : points;
                cls = __shfl_sync(0xffffffffu, cls, hit & 31);
                if (lane == 0) grid_step(sS, hit, hit < points ? cls : 0);
            }
        } else {
            const int npts = sS.npts;
            for (int it = blockIdx.x; it < npts * nblk; it += gridDim.x) {
                const int pt = it / nblk, c = it - pt * nblk;
                double m[2];
                chunk_moments(llk, n, sS.pts[pt], med, lmax, c, m);
                if (tid == 0) {
                    pr[(size_t)(2 * pt) * nblk + c] = m[0];
                    pr[(size_t)(2 * pt + 1) * nblk + c] = m[1];
                }
            }
            if (!meet()) return;
            if (tid < 2 * npts) {
                double a = 0.0;
                for (int k = 0; k < nblk; ++k) a += __ldcg(pr + (size_t)tid * nblk + k);
                s_tot[tid] = a;
            }
            __syncthreads();
            if (tid == 0) {
                double cov[2];
                for (int pt = 0; pt < npts; ++pt)
                    cov[pt] = cov_from_moments(s_tot[2 * pt], s_tot[2 * pt + 1], sS.pts[pt] * (lmax - med), n);
                brent_step(sS, cov, target, tol, maxiter);
            }
        }
        __syncthreads();
    }
    // the exponentials at the chosen δβ, their moments, then the state, β, and the normalised weights
    double* fp = part + 2 * pbuf;
    const double g = sS.dbeta, mx = g * (lmax - med);
    const long share = cov_share(n), begin = blockIdx.x * share + threadIdx.x, end = min((long)n, (blockIdx.x + 1) * share);
    for (long i = begin; i < end; i += blockDim.x) w[i] = exp(g * (llk[i] - med) - mx);
    if (!meet()) return;
    for (int c = blockIdx.x; c < nblk; c += gridDim.x) {
        double m[2];
        chunk_sums(n, c, [&](int i) { return __ldcg(w + i); }, m);
        if (threadIdx.x == 0) {
            fp[2 * c] = m[0];
            fp[2 * c + 1] = m[1];
        }
    }
    if (!meet()) return;
    if (threadIdx.x < 2) {
        double a = 0.0;
        for (int k = 0; k < nblk; ++k) a += __ldcg(fp + 2 * k + threadIdx.x);
        s_tot[threadIdx.x] = a;
    }
    __syncthreads();
    const double s1 = s_tot[0];
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        sS.s1 = s1;
        sS.cov = cov_from_moments(s1, s_tot[1], mx, n);
        *S = sS;
        // β bookkeeping (COV.cc:264, 323)
        *beta = sS.skip ? 1.0 : sS.beta0 + sS.dbeta;
        dbeta_cov[0] = sS.dbeta;
        dbeta_cov[1] = sS.cov;
    }
    for (long i = begin; i < end; i += blockDim.x) w[i] = w[i] / s1;
}

// ---------------------------------------------------------------------------
// weighted covariance (COV.py:106-156): per-block partial sums in fixed order.
//
// With x = (1, θ) the sums Σw, Σ w θ_a and Σ w θ_a θ_b are the lower triangle of Σ (w x)(x)ᵀ: one
// FP64 FMA per entry and chain, the products w x formed once per chain in shared memory.  FP64
// issue bounds it (64 cycles per warp instruction and SM quarter), so the chains are spread over
// all SMs (as few as kSigmaMinRows per block, so that few chains still fill them) and, where the
// entries leave threads over, groups of threads share a block's chains.  Measured, 10
// parameters: 32,768 chains 24 µs (56 µs with one thread per entry and three instructions per
// term); 4 parameters, 1,024 chains 8 µs (43 µs).
constexpr size_t kSigmaSmem = 160 * 1024;
constexpr int kSigmaBlocks = 152;  // one per SM
constexpr int kSigmaMinRows = 16;      // of a chunk (kSigmaSmem holds as many at kMaxPLarge)
static_assert(kSigmaMinRows * 2 * (kMaxPLarge + 1) * sizeof(double) <= kSigmaSmem, "the workspace counts on it");
static void sigma_grid(int n, int p, int* chunk, int* nblk, int* cpb) {
    int most = (int)(kSigmaSmem / (2 * (p + 1) * sizeof(double)));
    if (most > kSigmaChunk) most = kSigmaChunk;
    const int rows = (n - 1) / kSigmaBlocks + 1;
    *chunk = rows < kSigmaMinRows ? kSigmaMinRows : rows < most ? rows : most;
    if (*chunk > most) *chunk = most;
    const int nchunks = (n - 1) / *chunk + 1;
    *cpb = (nchunks - 1) / kSigmaBlocks + 1;
    *nblk = (nchunks - 1) / *cpb + 1;
}

// entry e of a lower triangle stored by rows: row a starts at a (a + 1) / 2
__device__ __forceinline__ void triangle_entry(int e, int& a, int& b) {
    a = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while ((a + 1) * (a + 2) / 2 <= e) ++a;
    while (a * (a + 1) / 2 > e) --a;
    b = e - a * (a + 1) / 2;
}

// Block b sums the chunks [b·cpb, (b+1)·cpb) in order into part[b][e]; the last block to
// finish adds the blocks' partials in block order and assembles Σ.
__global__ void __launch_bounds__(256) sigma_kernel(const double* __restrict__ theta,
                                                    const double* __restrict__ w, int n, int p, int chunk,
                                                    int cpb, double* __restrict__ part, double* __restrict__ tot,
                                                    unsigned* __restrict__ done, double* __restrict__ sigma) {
    after_previous();
    extern __shared__ double sm[];      // x [chunk][p + 1], w x [chunk][p + 1]
    __shared__ double s_red[256];
    const int tid = threadIdx.x, q = p + 1, nent = q * (q + 1) / 2;
    double* sx = sm;
    double* sy = sm + (size_t)chunk * q;
    const int groups = nent < 256 ? 256 / nent : 1;
    const int grp = groups > 1 ? tid / nent : 0;
    const int c0 = blockIdx.x * cpb;
    // the sum over this group's share of count terms, two chains of dependent FMAs
    auto group_sum = [&](double acc, int count, auto term) {
        double odd = 0.0;
        int i = grp;
        for (; i + groups < count; i += 2 * groups) {
            acc = term(i, acc);
            odd = term(i + groups, odd);
        }
        if (i < count) acc = term(i, acc);
        return acc + odd;
    };
    for (int c = c0; c < c0 + cpb; ++c) {
        const long begin = (long)c * chunk;
        if (begin >= n) break;
        const int cnt = (int)(n - begin < chunk ? n - begin : chunk);
        __syncthreads();
        for (int k = tid; k < cnt * p; k += blockDim.x) {
            const int i = k / p, j = i * q + 1 + (k - i * p);
            const double x = theta[(size_t)begin * p + k];
            sx[j] = x;
            sy[j] = w[begin + i] * x;
        }
        for (int i = tid; i < cnt; i += blockDim.x) {
            sx[(size_t)i * q] = 1.0;
            sy[(size_t)i * q] = w[begin + i];
        }
        __syncthreads();
        for (int e = groups > 1 ? tid - grp * nent : tid; e < nent; e += 256) {
            double acc = (c == c0 || grp > 0) ? 0.0 : part[(size_t)blockIdx.x * nent + e];
            if (grp < groups) {
                int a, b;
                triangle_entry(e, a, b);
                acc = group_sum(acc, cnt, [&](int i, double t) { return fma(sy[i * q + a], sx[i * q + b], t); });
            }
            if (groups == 1) {
                part[(size_t)blockIdx.x * nent + e] = acc;
            } else {
                s_red[tid] = acc;
                break;                  // one entry per thread
            }
        }
        if (groups > 1) {
            __syncthreads();
            if (tid < nent) {
                double acc = s_red[tid];
                for (int g = 1; g < min(groups, cnt); ++g) acc += s_red[g * nent + tid];
                part[(size_t)blockIdx.x * nent + tid] = acc;
            }
        }
    }
    // the last block to finish (threadfence reduction: the count is cleared before the launch)
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(done, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // totals over the blocks, each group its share of them in block order
    const int parts = (int)gridDim.x;
    if (groups > 1) {
        const int e = tid - grp * nent;
        s_red[tid] = grp >= groups ? 0.0 : group_sum(0.0, parts, [&](int k, double t) {
            return t + __ldcg(part + (size_t)k * nent + e);
        });
        __syncthreads();
        if (tid < nent) {
            double acc = s_red[tid];
            for (int g = 1; g < min(groups, parts); ++g) acc += s_red[g * nent + tid];
            tot[tid] = acc;
        }
    } else {
        // the same two chains, with the loads of 16 partials in flight: one SM reads them all, and two loads at
        // a time were most of the kernel (2,400 chains, 200 parameters 2,222 -> 1,167 µs; 1,000, 512 6,956 -> 4,139)
        constexpr int kAhead = 16;
        for (int e = tid; e < nent; e += 256) {
            const double* p0 = part + e;
            double acc = 0.0, odd = 0.0;
            int k = 0;
            for (; k + kAhead <= parts; k += kAhead, p0 += (size_t)kAhead * nent) {
                double v[kAhead];
#pragma unroll
                for (int q = 0; q < kAhead; ++q) v[q] = __ldcg(p0 + (size_t)q * nent);
#pragma unroll
                for (int q = 0; q < kAhead; q += 2) {
                    acc += v[q];
                    odd += v[q + 1];
                }
            }
            for (; k < parts; k += 2, p0 += 2 * (size_t)nent) {
                acc += __ldcg(p0);
                if (k + 1 < parts) odd += __ldcg(p0 + nent);
            }
            tot[e] = acc + odd;
        }
    }
    __syncthreads();
    // Σ_ab = Σ w θ_a θ_b - θ̄_a θ̄_b with θ̄ = Σ w θ / Σ w (gsl_stats_wmean)
    for (int e = tid; e < nent; e += 256) {
        int a, b;
        triangle_entry(e, a, b);
        if (b == 0) continue;
        const double ma = tot[a * (a + 1) / 2] / tot[0], mb = tot[b * (b + 1) / 2] / tot[0];
        const double v = tot[e] - ma * mb;
        sigma[(a - 1) * p + b - 1] = v;
        sigma[(b - 1) * p + a - 1] = v;
    }
}

// chol(scaling² Σ), lower triangle row-major (Metropolis.py:103-107).  One CTA,
// left-looking by columns in L itself: thread 0 forms the diagonal, then every
// thread forms one entry below it; each entry sums over k in increasing order, as
// the sequential Cholesky–Crout loop does.
__global__ void cholesky_kernel(int p, const double* __restrict__ sigma,
                                const double* __restrict__ scaling, double* __restrict__ L,
                                uint32_t* __restrict__ flags) {
    __shared__ double s_ljj;
    __shared__ int s_ok;
    const double s2 = (*scaling) * (*scaling);
    for (int k = threadIdx.x; k < p * p; k += blockDim.x) L[k] = s2 * sigma[k];
    if (threadIdx.x == 0) s_ok = 1;
    __syncthreads();
    for (int j = 0; j < p; ++j) {
        if (threadIdx.x == 0) {
            double d = L[j * p + j];
            for (int k = 0; k < j; ++k) d -= L[j * p + k] * L[j * p + k];
            if (!(d > 0.0)) {
                s_ok = 0;
            } else {
                s_ljj = sqrt(d);
                L[j * p + j] = s_ljj;
            }
        }
        __syncthreads();
        if (!s_ok) break;
        const double ljj = s_ljj;
        for (int i = j + 1 + threadIdx.x; i < p; i += blockDim.x) {
            double v = L[i * p + j];
            for (int k = 0; k < j; ++k) v -= L[i * p + k] * L[j * p + k];
            L[i * p + j] = v / ljj;
        }
        __syncthreads();
    }
    if (!s_ok) {
        // keep the walk defined: fall back to the scaled diagonal and report
        if (threadIdx.x == 0) raise_flag(flags, DEV_ERR_NOT_SPD);
        for (int k = threadIdx.x; k < p * p; k += blockDim.x) {
            const int i = k / p, c = k % p;
            L[k] = (i == c) ? sqrt(fmax(s2 * sigma[k], 0.0)) : 0.0;
        }
        return;
    }
    for (int k = threadIdx.x; k < p * p; k += blockDim.x)
        if (k % p > k / p) L[k] = 0.0;              // clear the upper triangle
}

// ---------------------------------------------------------------------------
// multinomial resampling (COV.py:160-251)
struct ResampleHdr {
    int total;        // number of copied rows (Σ counts)
    int first_src;    // source row of output row 0
    int pad[2];
};

// Sequential FP64 partial sums, as itertools.accumulate (COV.py:242-251): edges[i + 1] =
// fl(edges[i] + w[i]), bit for bit, without the chain of dependent additions (67 cycles each:
// 1,326 µs for 32,768 weights, measured).
//
// While the running sum stays in one binade, [2^e, 2^(e+1)) with unit u = 2^(e-52) in the last
// place, it is an integer multiple S u of u, 2^52 <= S < 2^53, and adding w rounds to S + q with
// q = w/u rounded to the nearest integer: the same q whatever S, except when w/u lies exactly
// between two integers, where the even sum is taken and q depends on the parity of S alone.
// So an addition is a map S -> S + (S even ? a0 : a1), such maps compose into maps of the same
// form, and a tile of additions is one parallel scan in 64-bit integers.  The first addition
// that leaves the binade (or meets a negative or non-finite weight) is done in FP64 and the scan
// starts again behind it; the binade then grows by at least one, so a sum of n positive
// weights restarts about log2(n) times after the first kCdfHead weights, which one thread adds.
// Below 2^-1021 (zeros and subnormals included) the unit is 2^-1074 and the same holds.
// A tie needs the dropped bits of w to be exactly a half, once in 2^s weights for a shift of s
// bits, so most warps see none and scan plain sums; the pair of increments is carried only by
// the warps that do and between the warps.  What bounds the kernel is the integer work of the
// restarts on one SM: short tiles by one warp up to kCdfWarpEnd weights, where most restarts
// fall, then tiles of kCdfTile by the whole block.  Measured: 32,768
// weights 71 µs (1,326 µs with the additions in a row), 1,024 weights 17 µs (43 µs).
constexpr int kCdfThreads = 512;
constexpr int kCdfPer = 8;
constexpr int kCdfTile = kCdfThreads * kCdfPer;
constexpr int kCdfHead = 16;
constexpr int kCdfWarpPer = 4;
constexpr int kCdfWarpEnd = 1024;
// Weights that rise by a binade every few additions would restart the scan at each of them.  After more
// than kCdfPatience tiles running that place fewer than kCdfFew (kCdfWarpFew for the warp; about what a
// tile costs in additions) come that many additions one after another, twice as many behind each further
// such tile; ordinary weights have two or three of them running at most, while the sum doubles within few.
// Resampling with weights rising over 260 decades: 1,000 chains 73 µs and 4,096 235 (762 and 2,615 with a tile per
// restart, 134 and 295 with all additions in a row).
constexpr int kCdfPatience = 4;
constexpr int kCdfWarpFew = 24;
constexpr int kCdfFew = 96;
constexpr uint64_t kCdfBig = 1ull << 58;       // saturation: anything >= 2^53 leaves the binade

struct CdfAdd { uint64_t a0, a1; };            // increment of an even and of an odd sum

__device__ __forceinline__ CdfAdd cdf_then(CdfAdd f, CdfAdd g) {
    const uint64_t r0 = f.a0 + ((f.a0 & 1) ? g.a1 : g.a0);
    const uint64_t r1 = f.a1 + ((f.a1 & 1) ? g.a0 : g.a1);
    return {r0 < kCdfBig ? r0 : kCdfBig, r1 < kCdfBig ? r1 : kCdfBig};
}

// the addition of weight w to a sum of binade e (e = -1022 also covers the subnormals)
__device__ __forceinline__ CdfAdd cdf_add(double w, int e) {
    const uint64_t bits = (uint64_t)__double_as_longlong(w);
    if ((bits << 1) == 0) return {0, 0};
    const int x = (int)(bits >> 52);           // sign and exponent
    if (x >= 0x7ff) return {kCdfBig, kCdfBig};
    const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (x ? 1ull << 52 : 0ull);
    const int s = e - (x ? x - 1023 : -1022);
    if (s < 0) return {kCdfBig, kCdfBig};
    if (s == 0) return {m, m};
    if (s > 53) return {0, 0};                 // below half a unit
    const uint64_t q = m >> s, rem = m & ((1ull << s) - 1), half = 1ull << (s - 1);
    if (rem == half) return {q + (q & 1), q + ((q + 1) & 1)};
    return {q + (rem > half), q + (rem > half)};
}

// S u as a double (S < 2^53; S >= 2^52 unless e = -1022)
__device__ __forceinline__ double cdf_value(uint64_t S, int e) {
    return __longlong_as_double((long long)(S >> 52 ? ((uint64_t)(e + 1023) << 52) | (S & 0xFFFFFFFFFFFFFull) : S));
}

// the sum acc as S and e; false if it is negative or not finite
__device__ __forceinline__ bool cdf_split(double acc, uint64_t& S, int& e) {
    const uint64_t bits = (uint64_t)__double_as_longlong(acc);
    const int x = (int)(bits >> 52);
    if (x >= 0x7ff && bits != 1ull << 63) return false;
    e = (x & 0x7ff) ? x - 1023 : -1022;
    S = (bits & 0xFFFFFFFFFFFFFull) | ((x & 0x7ff) ? 1ull << 52 : 0ull);
    return true;
}

// additions in a row behind a tile that placed `placed` weights, `before` of them behind the last tile; up to
// kCdfPatience it counts the tiles of few and nothing is added in a row
__device__ __forceinline__ int cdf_row(int before, int placed, int few) {
    if (placed >= few) return 0;
    return before < kCdfPatience ? before + 1 : before == kCdfPatience ? few
           : 2 * before < kCdfWarpEnd ? 2 * before : kCdfWarpEnd;
}

// this lane's PER additions (f), the map of the lanes before it (pre) and of the whole warp (all)
template <int PER>
__device__ __forceinline__ void cdf_warp_scan(const double (&v)[PER], int e, int lane, CdfAdd (&f)[PER], CdfAdd& pre,
                                              CdfAdd& all) {
    CdfAdd tot{0, 0};
    bool tie = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        f[k] = cdf_add(v[k], e);
        tie |= f[k].a0 != f[k].a1;
    }
    if (!__any_sync(0xffffffffu, tie)) {
        // 32 PER increments below 2^53 stay below 2^61; a saturated one (2^58) may be among them
        uint64_t t = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) t += f[k].a0;
        t = t < kCdfBig ? t : kCdfBig;
        uint64_t s = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t p = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += p;
        }
        pre.a0 = pre.a1 = s - t < kCdfBig ? s - t : kCdfBig;
        s = __shfl_sync(0xffffffffu, s, 31);
        all.a0 = all.a1 = s < kCdfBig ? s : kCdfBig;
        return;
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) tot = cdf_then(tot, f[k]);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const CdfAdd p{__shfl_up_sync(0xffffffffu, tot.a0, o), __shfl_up_sync(0xffffffffu, tot.a1, o)};
        if (lane >= o) tot = cdf_then(p, tot);
    }
    pre = CdfAdd{__shfl_up_sync(0xffffffffu, tot.a0, 1), __shfl_up_sync(0xffffffffu, tot.a1, 1)};
    if (lane == 0) pre = CdfAdd{0, 0};
    all = CdfAdd{__shfl_sync(0xffffffffu, tot.a0, 31), __shfl_sync(0xffffffffu, tot.a1, 31)};
}

// this thread's edges from the sum S before its first weight (index i0): those inside the binade
// (the sums only grow, so the others come after them).  True where this thread holds the tile's
// new position and sum: behind the first addition that leaves the binade, or at the tile's end.
template <int PER>
__device__ __forceinline__ bool cdf_apply(const double (&v)[PER], const CdfAdd (&f)[PER], uint64_t S, int e, int i0,
                                          int end, double* __restrict__ edges, int& pos, double& acc) {
    int last = -1;                             // the first of my sums outside the binade
    uint64_t at = 0;
    double left = 0.0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        if (i0 + k >= end) break;
        const uint64_t next = S + ((S & 1) ? f[k].a1 : f[k].a0);
        if ((next >> 53) == 0) {
            edges[i0 + k + 1] = cdf_value(next, e);
        } else if ((S >> 53) == 0) {
            last = k;
            at = S;
            left = v[k];
        }
        S = next;
    }
    if (last >= 0) {
        pos = i0 + last + 1;
        acc = cdf_value(at, e) + left;
        edges[pos] = acc;
        return true;
    }
    if ((S >> 53) || i0 >= end || i0 + PER < end) return false;
    pos = end;
    acc = cdf_value(S, e);
    return true;
}

// one CTA; also clears the counts that the next kernel adds to
__global__ void __launch_bounds__(kCdfThreads) cdf_kernel(const double* __restrict__ w, int n,
                                                          double* __restrict__ edges, int* __restrict__ counts) {
    after_previous();
    __shared__ CdfAdd s_warp[kCdfThreads / 32];
    __shared__ double s_w[kCdfWarpEnd];
    __shared__ double s_acc;
    __shared__ int s_pos;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int stop = n < kCdfWarpEnd ? n : kCdfWarpEnd;
    for (int i = tid; i < stop; i += kCdfThreads) s_w[i] = w[i];
    __syncthreads();
    if (warp == 0) {
        int pos = 0, row = 0;
        double acc = 0.0;
        auto add = [&](int count) {            // count weights one after another
            const int end = stop - pos < count ? stop : pos + count;
            if (lane == 0) {
                for (int i = pos; i < end; ++i) {
                    acc += s_w[i];
                    edges[i + 1] = acc;
                }
            }
            acc = __shfl_sync(0xffffffffu, acc, 0);
            pos = end;
        };
        if (lane == 0) edges[0] = 0.0;
        add(kCdfHead);
        uint64_t S;
        int e;
        while (pos < stop && cdf_split(acc, S, e)) {
            const int from0 = pos, end = stop - pos < 32 * kCdfWarpPer ? stop : pos + 32 * kCdfWarpPer;
            const int i0 = pos + lane * kCdfWarpPer;
            double v[kCdfWarpPer];
            CdfAdd f[kCdfWarpPer], pre, all;
#pragma unroll
            for (int k = 0; k < kCdfWarpPer; ++k) v[k] = i0 + k < end ? s_w[i0 + k] : 0.0;
            cdf_warp_scan(v, e, lane, f, pre, all);
            const bool mine = cdf_apply(v, f, S + ((S & 1) ? pre.a1 : pre.a0), e, i0, end, edges, pos, acc);
            const int from = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
            pos = __shfl_sync(0xffffffffu, pos, from);
            acc = __shfl_sync(0xffffffffu, acc, from);
            row = cdf_row(row, pos - from0, kCdfWarpFew);
            if (row > kCdfPatience) add(row);
        }
        if (lane == 0) {
            s_acc = acc;
            s_pos = pos;
        }
    } else {
        for (int i = tid - 32; i < n; i += kCdfThreads - 32) counts[i] = 0;
    }
    __syncthreads();
    int row = 0, next = 0;                     // of the last tile; additions in a row now
    for (;;) {
        const int pos0 = s_pos;
        int pos = pos0;
        double acc = s_acc;
        if (pos >= n) return;
        uint64_t S;
        int e;
        const bool split = cdf_split(acc, S, e);
        if (next > kCdfPatience || !split) {              // (a negative or non-finite sum: plain additions to the end)
            const int most = split ? next : kCdfWarpEnd, len = n - pos < most ? n - pos : most;
            for (int i = tid; i < len; i += kCdfThreads) s_w[i] = w[pos + i];
            __syncthreads();
            if (tid == 0) {
                for (int i = 0; i < len; ++i) {
                    acc += s_w[i];
                    edges[pos + i + 1] = acc;
                }
                s_acc = acc;
                s_pos = pos + len;
            }
            next = 0;
            __syncthreads();
            continue;
        }
        const int end = n - pos < kCdfTile ? n : pos + kCdfTile;
        const int i0 = pos + tid * kCdfPer;
        double v[kCdfPer];
        CdfAdd f[kCdfPer], pre, all;
#pragma unroll
        for (int k = 0; k < kCdfPer; ++k) v[k] = i0 + k < end ? __ldg(w + i0 + k) : 0.0;
        cdf_warp_scan(v, e, lane, f, pre, all);
        if (lane == 0) s_warp[warp] = all;
        __syncthreads();
        if (warp > 0) {
            // the warps before this one, in order: lane l takes warp l's map
            CdfAdd t = lane < warp ? s_warp[lane] : CdfAdd{0, 0};
#pragma unroll
            for (int o = 1; o < kCdfThreads / 32; o <<= 1) {
                const CdfAdd p{__shfl_up_sync(0xffffffffu, t.a0, o), __shfl_up_sync(0xffffffffu, t.a1, o)};
                if (lane >= o) t = cdf_then(p, t);
            }
            t = CdfAdd{__shfl_sync(0xffffffffu, t.a0, kCdfThreads / 32 - 1),
                       __shfl_sync(0xffffffffu, t.a1, kCdfThreads / 32 - 1)};
            pre = cdf_then(t, pre);
        }
        if (cdf_apply(v, f, S + ((S & 1) ? pre.a1 : pre.a0), e, i0, end, edges, pos, acc)) {
            s_acc = acc;
            s_pos = pos;
        }
        __syncthreads();
        next = row = cdf_row(row, s_pos - pos0, kCdfFew);
    }
}

// counts[i] = #{j : edges[i] <= r_j < edges[i+1]}; r_j >= edges[n] dropped (gsl_histogram).
// One thread per uniform.
__global__ void __launch_bounds__(256) counts_kernel(int n, uint64_t seed, const uint32_t* __restrict__ epoch,
                                                     const double* __restrict__ edges, int* __restrict__ counts) {
    after_previous();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    u32x4 r = draw(seed, (uint32_t)j, 0u, STREAM_RESAMPLE, 0u, *epoch);
    const double x = u01_closed_open(r.x, r.y);
    if (!(x >= edges[0] && x < edges[n])) return;
    // largest i with edges[i] <= x
    int lo = 0, hi = n;          // edges[lo] <= x < edges[hi]
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (x >= edges[mid]) lo = mid; else hi = mid;
    }
    atomicAdd(&counts[lo], 1);
}

// start[i] = first output row of chain i's copies: rows in order of decreasing count, ties by
// increasing index.  One CTA; each thread owns kRankPer consecutive chains of a chunk and one
// column of counters per small count (s_col[c][thread], column 0 for the counts of kRankSmall
// and more), so a thread's chains come in order, a scan over the threads of each column gives the
// stable ranks, and no two threads share a counter.  The few chains with large counts (at most
// n/kRankSmall, since the counts add up to at most n) are ranked against each other.  Counts
// and results pass through shared memory so that global accesses are coalesced, and only as many
// columns as the chains need are cleared and scanned.  Measured:
// 32,768 chains 22 µs (375 µs with one warp walking the chains in order), 1,024 chains 9 µs.
constexpr int kRankThreads = 1024;
constexpr int kRankPer = 32;
constexpr int kRankSmall = 32;
constexpr int kRankChunk = kRankThreads * kRankPer;
constexpr size_t kRankSmem = (size_t)kRankChunk * sizeof(int) + (size_t)kRankSmall * kRankThreads * sizeof(uint16_t);

__global__ void __launch_bounds__(kRankThreads) rank_kernel(int n, const int* __restrict__ counts,
                                                            int* __restrict__ big_row, int* __restrict__ big_cnt,
                                                            int* __restrict__ start, ResampleHdr* __restrict__ hdr) {
    after_previous();
    extern __shared__ int s_chunk[];               // [kRankThreads][kRankPer]
    uint16_t* s_col = reinterpret_cast<uint16_t*>(s_chunk + kRankChunk);     // [kRankSmall][kRankThreads]
    __shared__ int s_tot[kRankSmall], s_base[kRankSmall], s_seen[kRankSmall];
    __shared__ int s_bigsum;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int threads = n < kRankChunk ? ((n + kRankPer - 1) / kRankPer + 31) / 32 * 32 : kRankThreads;
    const bool owner = tid < threads;
    uint16_t* col = s_col + tid;
    // chain k of thread t lies at word t kRankPer + (k ^ (t mod 32)): no bank conflicts by row or column
    auto word = [](int i) { return (i & ~31) | ((i ^ (i >> 5)) & 31); };
    auto clear = [&]() {
        for (int v = warp; v < kRankSmall; v += 32)
            for (int k = lane * 2; k < threads; k += 64) *reinterpret_cast<uint32_t*>(s_col + v * kRankThreads + k) = 0u;
    };
    int c[kRankPer];
    auto load = [&](long c0) {
        const int len = n - c0 < kRankChunk ? (int)(n - c0) : kRankChunk;
        for (int i = tid; i < threads * kRankPer; i += kRankThreads) s_chunk[word(i)] = i < len ? counts[c0 + i] : 0;
        __syncthreads();
        if (owner) {
#pragma unroll
            for (int k = 0; k < kRankPer; ++k) c[k] = s_chunk[word(tid * kRankPer + k)];
        }
    };
    auto tally = [&]() {
        int big = 0;
        if (owner) {
#pragma unroll
            for (int k = 0; k < kRankPer; ++k) {
                if (c[k] <= 0) continue;
                const int v = c[k] < kRankSmall ? c[k] : 0;
                col[v * kRankThreads] += 1;
                if (v == 0) big += c[k];
            }
        }
        return big;
    };
    int total = 0;                                 // warp v: chains with count v so far
    auto add_columns = [&]() {
        int t = 0;
        for (int k = lane; k < threads; k += 32) t += s_col[warp * kRankThreads + k];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        total += t;
    };
    clear();
    if (tid == 0) {
        s_bigsum = 0;
        hdr->first_src = -1;
    }
    // totals per count over all chunks, each thread in its own column
    for (long c0 = 0; c0 < n; c0 += kRankChunk) {
        if (c0 > 0) {
            __syncthreads();
            clear();
        }
        load(c0);
        const int big = tally();
        if (big) atomicAdd(&s_bigsum, big);
        __syncthreads();
        add_columns();
    }
    if (lane == 0) s_tot[warp] = total;
    __syncthreads();
    if (warp == 0) {
        // base[v] = Σ_{v' > v} v' chains(v') (lane v), behind the large counts
        int x = lane * s_tot[lane], s = x;
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_down_sync(0xffffffffu, s, o);
            if (lane + o < 32) s += t;
        }
        s_base[lane] = s_bigsum + s - x;
        s_seen[lane] = 0;
        if (lane == 0) hdr->total = s_bigsum + s;
    }
    for (long c0 = 0; c0 < n; c0 += kRankChunk) {
        if (n > kRankChunk) {
            // the columns hold the last chunk's counts: this chunk's alone again
            __syncthreads();
            clear();
            load(c0);
            tally();
        }
        __syncthreads();
        // exclusive scan of column `warp` over the threads, behind the earlier chunks' chains
        int carry = 0;
        for (int k = 0; k < threads; k += 32) {
            uint16_t* at = s_col + warp * kRankThreads + k + lane;
            const int v = *at;
            int s = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += t;
            }
            *at = (uint16_t)(carry + s - v);
            carry += __shfl_sync(0xffffffffu, s, 31);
        }
        __syncthreads();
        if (owner) {
            const long i0 = c0 + tid * kRankPer;
#pragma unroll
            for (int k = 0; k < kRankPer; ++k) {
                int st = -1;
                if (c[k] > 0) {
                    const int v = c[k] < kRankSmall ? c[k] : 0;
                    const int rank = s_seen[v] + col[v * kRankThreads]++;
                    if (v == 0) {
                        big_row[rank] = (int)(i0 + k);
                        big_cnt[rank] = c[k];
                    } else {
                        st = s_base[v] + v * rank;
                        if (st == 0) hdr->first_src = (int)(i0 + k);
                    }
                }
                s_chunk[word(tid * kRankPer + k)] = st;
            }
        }
        __syncthreads();
        const int len = n - c0 < kRankChunk ? (int)(n - c0) : kRankChunk;
        for (int i = tid; i < len; i += kRankThreads) start[c0 + i] = s_chunk[word(i)];
        if (lane == 0) s_seen[warp] += carry;
    }
    __syncthreads();
    const int nbig = s_tot[0];
    for (int a = tid; a < nbig; a += kRankThreads) {
        const int ca = big_cnt[a];
        int st = 0;
        for (int b = 0; b < nbig; ++b) {
            const int cb = big_cnt[b];
            st += (cb > ca || (cb == ca && b < a)) ? cb : 0;
        }
        start[big_row[a]] = st;
        if (st == 0) hdr->first_src = big_row[a];
    }
}

// one thread per element of θ, so that consecutive threads copy consecutive parameters
__global__ void gather_kernel(int n, int p, const double* __restrict__ beta,
                              const int* __restrict__ counts, const int* __restrict__ start,
                              const ResampleHdr* __restrict__ hdr,
                              const double* __restrict__ th_in, const double* __restrict__ pr_in,
                              const double* __restrict__ da_in, double* __restrict__ th_out,
                              double* __restrict__ pr_out, double* __restrict__ da_out,
                              double* __restrict__ po_out) {
    after_previous();
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(t / p), j = (int)(t - (long)i * p);
    if (i >= n) return;
    const double b = *beta;
    auto copy = [&](int src, int d0, int c) {
        const double v = th_in[(size_t)src * p + j];
        for (int k = 0; k < c; ++k) th_out[(size_t)(d0 + k) * p + j] = v;
        if (j != 0) return;
        const double pr = pr_in[src], da = da_in[src];
        const double po = pr + b * da;
        for (int k = 0; k < c; ++k) {
            pr_out[d0 + k] = pr;
            da_out[d0 + k] = da;
            po_out[d0 + k] = po;
        }
    };
    const int c = counts[i];
    if (c > 0) copy(i, start[i], c);
    // rows left over when uniforms fell beyond the last edge repeat the first group's row
    if (i >= hdr->total && hdr->first_src >= 0) copy(hdr->first_src, i, 1);
}

// ---------------------------------------------------------------------------
// scaling adaptation (Metropolis.py:262-281); then a new epoch
__global__ void adapt_kernel(double aw, double rw, unsigned long long* __restrict__ counters,
                             double* __restrict__ scaling, uint32_t* __restrict__ epoch) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double acc = (double)counters[0];
    const double tot = (double)(counters[0] + counters[1] + counters[2]);
    const double acceptance = tot > 0.0 ? acc / tot : 0.0;
    double kc = (aw * acceptance + rw) / (aw + rw);
    if (kc < 0.1) kc = 0.1;
    if (kc > 1.0) kc = 1.0;
    *scaling = kc;
    counters[0] = counters[1] = counters[2] = 0ull;
    *epoch += 1u;
}

}  // namespace ag

// ---------------------------------------------------------------------------
// C ABI
using namespace ag;

static inline int blocks(int n, int t) { return (n + t - 1) / t; }

static int check_state(const ag_stage_state* st) {
    AG_REQUIRE(st && st->beta && st->dbeta_cov && st->scaling && st->sigma && st->chol && st->w &&
                   st->counters && st->epoch && st->dev_flags,
               "stage state has a NULL member");
    AG_REQUIRE(st->chain0 >= 0, "stage state chain0 must be >= 0 (got %d)", st->chain0);
    return AG_OK;
}

extern "C" int ag_prior_sample(int32_t n, int32_t p, const double* lo, const double* hi,
                               uint64_t seed, uint32_t attempt, const uint32_t* redraw,
                               double* theta, void* stream) {
    AG_REQUIRE(n > 0 && p > 0 && lo && hi && theta, "invalid arguments");
    prior_sample_kernel<<<blocks(n, 256), 256, 0, as_stream(stream)>>>(n, p, lo, hi, seed, attempt,
                                                                        redraw, theta);
    return launch_status("prior_sample_kernel");
}

extern "C" int ag_prior_llk(const double* theta, int32_t n, int32_t p, const double* lo,
                            const double* hi, uint32_t* mask, double* prior, void* stream) {
    AG_REQUIRE(n > 0 && p > 0 && theta && lo && hi, "invalid arguments");
    prior_llk_kernel<<<blocks(n, 256), 256, 0, as_stream(stream)>>>(theta, n, p, lo, hi, mask, prior);
    return launch_status("prior_llk_kernel");
}

extern "C" int ag_propose(const ag_stage_state* st, const double* theta, int32_t n, int32_t p,
                          const double* lo, const double* hi, uint64_t seed, uint32_t step,
                          double* cand, uint32_t* mask, double* cprior, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && p > 0 && p <= kMaxPLarge && theta && lo && hi && cand && mask && cprior,
               "invalid arguments (p must be in 1..%d)", kMaxPLarge);
    cudaStream_t s = as_stream(stream);
    if (p <= kMaxP) {
        propose_kernel<false><<<blocks(n, kProposeChains), kProposeThreads<false>, 0, s>>>(
            const_cast<double*>(theta), n, p, st->chol, lo, hi, seed, step, st->epoch, cand, mask, cprior, st->chain0,
            AcceptArgs{});
        return launch_status("propose_kernel");
    }
    const size_t smem = (size_t)kProposeWarps * p * sizeof(double);
    if (smem > 48 * 1024) {
        rc = cuda_status(cudaFuncSetAttribute(propose_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem),
                         "cudaFuncSetAttribute(propose_warp_kernel)");
        if (rc) return rc;
    }
    propose_warp_kernel<<<blocks(n, kProposeWarps), kProposeWarps * 32, smem, s>>>(
        theta, n, p, st->chol, lo, hi, seed, step, st->epoch, cand, mask, cprior, st->chain0);
    return launch_status("propose_warp_kernel");
}

extern "C" int ag_accept(const ag_stage_state* st, int32_t n, int32_t p, uint64_t seed,
                         uint32_t step, const uint32_t* mask, const double* cand,
                         const double* cprior, const double* cdata, double* theta, double* prior,
                         double* data, double* post, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && p > 0 && mask && cand && cprior && cdata && theta && prior && data && post,
               "invalid arguments");
    accept_kernel<<<blocks(n, 256), 256, 0, as_stream(stream)>>>(
        n, p, st->beta, seed, step, st->epoch, mask, cand, cprior, cdata, theta, prior, data, post,
        st->counters, st->chain0);
    return launch_status("accept_kernel");
}

extern "C" int ag_accept_floor(const ag_stage_state* st, int32_t n, uint64_t seed, uint32_t step,
                               const uint32_t* mask, const double* cprior, const double* post, double* llk_floor,
                               void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && mask && cprior && post && llk_floor, "invalid arguments");
    accept_floor_kernel<<<blocks(n, 256), 256, 0, as_stream(stream)>>>(n, st->beta, seed, step, st->epoch, mask,
                                                                        cprior, post, llk_floor, st->chain0);
    return launch_status("accept_floor_kernel");
}

extern "C" int ag_accept_propose(const ag_stage_state* st, int32_t n, int32_t p, const double* lo, const double* hi,
                                 uint64_t seed, uint32_t step, uint32_t* mask, double* cand, double* cprior,
                                 const double* cdata, double* theta, double* prior, double* data, double* post,
                                 double* llk_floor, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && p > 0 && p <= kMaxPLarge && lo && hi && mask && cand && cprior && cdata && theta && prior &&
                   data && post,
               "invalid arguments (p must be in 1..%d)", kMaxPLarge);
    if (p > kMaxP) {
        rc = ag_accept(st, n, p, seed, step, mask, cand, cprior, cdata, theta, prior, data, post, stream);
        if (!rc) rc = ag_propose(st, theta, n, p, lo, hi, seed, step + 1, cand, mask, cprior, stream);
        return rc || !llk_floor ? rc : ag_accept_floor(st, n, seed, step + 1, mask, cprior, post, llk_floor, stream);
    }
    propose_kernel<true><<<blocks(n, kProposeChains), kProposeThreads<true>, 0, as_stream(stream)>>>(
        theta, n, p, st->chol, lo, hi, seed, step + 1, st->epoch, cand, mask, cprior, st->chain0,
        AcceptArgs{st->beta, cdata, prior, data, post, st->counters, llk_floor});
    return launch_status("propose_kernel (accept)");
}

extern "C" int ag_posterior(const ag_stage_state* st, int32_t n, const double* prior,
                            const double* data, double* post, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && prior && data && post, "invalid arguments");
    posterior_kernel<<<blocks(n, 256), 256, 0, as_stream(stream)>>>(n, st->beta, prior, data, post);
    return launch_status("posterior_kernel");
}

// COV workspace: schedule state | grid barrier | partial moments (two round buffers, then the
// final chunks x 2)
static size_t cov_part_offset() { return (sizeof(CovState) + 255) / 256 * 256; }

extern "C" size_t ag_cov_workspace_bytes(int32_t n) {
    if (n <= 0) return 0;
    return cov_part_offset() + sizeof(GridBarrier) + cov_part_doubles(n) * sizeof(double);
}

// blocks of cov_schedule_kernel<BRENT> that fit on the current device at once (the cooperative
// launch's limit), looked up once per device
constexpr int kCoopMaxDevices = 64;
template <bool BRENT>
static int cov_coresident_blocks(int* out) {
    static std::mutex mu;
    static int cache[kCoopMaxDevices] = {};
    int dev = 0;
    int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= kCoopMaxDevices)
        return set_error(AG_ERR_SIZE, "device %d is beyond the %d devices the COV schedule tracks", dev,
                         kCoopMaxDevices);
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[dev]) {
        int occ = 0, sms = 0;
        rc = cuda_status(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, cov_schedule_kernel<BRENT, false>, 256, 0),
                         "cudaOccupancyMaxActiveBlocksPerMultiprocessor(cov_schedule_kernel)");
        if (rc) return rc;
        rc = cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
                         "cudaDeviceGetAttribute(multiprocessor count)");
        if (rc) return rc;
        if (occ < 1) return set_error(AG_ERR_CUDA, "cov_schedule_kernel does not fit on an SM");
        cache[dev] = occ * sms;
    }
    *out = cache[dev];
    return AG_OK;
}

// median (one CTA), then the whole search and the weights in one cooperative launch; the
// caller's scratch holds the state, the barrier words and the partials
template <bool BRENT>
static int cov_schedule_launch(const ag_stage_state* st, const double* data_llk, int n, double target,
                               double tol, int maxiter, int rounds, void* scratch, cudaStream_t s) {
    char* base = static_cast<char*>(scratch);
    CovState* S = reinterpret_cast<CovState*>(base);
    GridBarrier* bar = reinterpret_cast<GridBarrier*>(base + cov_part_offset());
    double* part = reinterpret_cast<double*>(base + cov_part_offset() + sizeof(GridBarrier));
    // a grid level splits the chains over the GPU; Brent's one or two points have a chunk per block
    const int want = BRENT ? 2 * blocks(n, kEvalChunk) : cov_blocks(n);
    const bool cluster = want <= kCovCluster;
    int grid = want, rc = AG_OK;
    if (!cluster) {
        rc = cov_coresident_blocks<BRENT>(&grid);
        if (rc) return rc;
        if (grid > want) grid = want;
        rc = cuda_status(cudaMemsetAsync(bar, 0, sizeof(GridBarrier), s), "cudaMemsetAsync(COV barrier)");
        if (rc) return rc;
    }
    launch_after(cov_median_kernel, 1, 1024, 0, s, data_llk, n, st->beta, S);
    rc = launch_status("cov_median_kernel");
    if (rc) return rc;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = attr;
    if (cluster) {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = grid;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
        return cuda_status(cudaLaunchKernelEx(&cfg, cov_schedule_kernel<BRENT, true>, data_llk, n, target, tol, maxiter,
                                              rounds, S, part, bar, st->beta, st->dbeta_cov, st->w, st->dev_flags),
                           "cov_schedule_kernel (cluster launch)");
    }
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, cov_schedule_kernel<BRENT, false>, data_llk, n, target, tol, maxiter,
                                          rounds, S, part, bar, st->beta, st->dbeta_cov, st->w, st->dev_flags),
                       "cov_schedule_kernel (cooperative launch)");
}

extern "C" int ag_cov_schedule(const ag_stage_state* st, const double* data_llk, int32_t n,
                               double target, double tol, void* workspace, size_t workspace_bytes,
                               void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 1 && data_llk, "invalid arguments (need at least two chains)");
    const size_t need = ag_cov_workspace_bytes(n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "ag_cov_schedule needs %zu bytes of 256-byte aligned workspace", need);
    // round 0 evaluates the full remaining step, rounds 1..kGridLevels one level each
    return cov_schedule_launch<false>(st, data_llk, n, target, tol, 0, kGridLevels + 1, workspace,
                                      as_stream(stream));
}

extern "C" int ag_cov_schedule_brent(const ag_stage_state* st, const double* data_llk, int32_t n,
                                     double target, double tol, int32_t maxiter, void* workspace,
                                     size_t workspace_bytes, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 1 && data_llk && maxiter > 0, "invalid arguments");
    const size_t need = ag_cov_workspace_bytes(n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "ag_cov_schedule_brent needs %zu bytes of 256-byte aligned workspace", need);
    const int iters = maxiter < kBrentMaxIter ? maxiter : kBrentMaxIter;
    // round 0: the full step; round 1: the guess and the interior point; then one point per iteration
    return cov_schedule_launch<true>(st, data_llk, n, target, tol, iters, iters + 2, workspace,
                                     as_stream(stream));
}

extern "C" size_t ag_sigma_workspace_bytes(int32_t n, int32_t p) {
    if (n <= 0 || p <= 0 || p > kMaxPLarge) return 0;
    // the most blocks that any smaller number of chains takes, so that more chains never need less
    const size_t rows = ((size_t)n - 1) / kSigmaMinRows + 1, nblk = rows < kSigmaBlocks ? rows : kSigmaBlocks;
    const size_t nent = 1 + p + (size_t)p * (p + 1) / 2;
    return (nblk + 1) * nent * sizeof(double) + 256;    // partials, totals, the block count
}

extern "C" int ag_weighted_cov(const ag_stage_state* st, const double* theta, int32_t n, int32_t p,
                               void* workspace, size_t workspace_bytes, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && p > 0 && p <= kMaxPLarge && theta, "invalid arguments (p <= %d)", kMaxPLarge);
    const size_t need = ag_sigma_workspace_bytes(n, p);
    AG_REQUIRE(workspace && workspace_bytes >= need, "ag_weighted_cov needs %zu bytes", need);
    cudaStream_t s = as_stream(stream);
    int chunk, nblk, cpb;
    sigma_grid(n, p, &chunk, &nblk, &cpb);
    const int nent = 1 + p + p * (p + 1) / 2;
    const size_t smem = (size_t)chunk * 2 * (p + 1) * sizeof(double);
    if (smem > 48 * 1024) {
        rc = cuda_status(cudaFuncSetAttribute(sigma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                         "cudaFuncSetAttribute(sigma_kernel)");
        if (rc) return rc;
    }
    double* part = reinterpret_cast<double*>(workspace);
    double* tot = part + (size_t)nblk * nent;
    unsigned* done = reinterpret_cast<unsigned*>(tot + nent);
    rc = cuda_status(cudaMemsetAsync(done, 0, sizeof(unsigned), s), "cudaMemsetAsync(Σ block count)");
    if (rc) return rc;
    launch_after(sigma_kernel, nblk, 256, smem, s, theta, st->w, n, p, chunk, cpb, part, tot, done, st->sigma);
    return launch_status("sigma_kernel");
}

extern "C" int ag_cholesky_scaled(const ag_stage_state* st, int32_t p, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(p > 0 && p <= kMaxPLarge, "p must be in 1..%d", kMaxPLarge);
    cholesky_kernel<<<1, 256, 0, as_stream(stream)>>>(p, st->sigma, st->scaling, st->chol, st->dev_flags);
    return launch_status("cholesky_kernel");
}

// workspace layout: hdr | edges[n+1] | counts[n] (if not given) | rows and counts of the
// chains with large counts | start[n]
static size_t align256(size_t b) { return (b + 255) / 256 * 256; }
extern "C" size_t ag_resample_workspace_bytes(int32_t n) {
    if (n <= 0) return 0;
    size_t b = align256(sizeof(ResampleHdr));
    b += align256((size_t)(n + 1) * sizeof(double));
    b += 4 * align256((size_t)(n + 1) * sizeof(int));
    return b;
}

extern "C" int ag_resample(const ag_stage_state* st, int32_t n, int32_t p, uint64_t seed,
                           const double* theta_in, const double* prior_in, const double* data_in,
                           double* theta_out, double* prior_out, double* data_out, double* post_out,
                           int32_t* counts, void* workspace, size_t workspace_bytes, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(n > 0 && p > 0 && theta_in && prior_in && data_in && theta_out && prior_out &&
                   data_out && post_out,
               "invalid arguments");
    AG_REQUIRE(theta_in != theta_out, "resampling is out of place: theta_in == theta_out");
    const size_t need = ag_resample_workspace_bytes(n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "ag_resample needs %zu bytes of 256-byte aligned workspace", need);
    cudaStream_t s = as_stream(stream);
    char* ws = static_cast<char*>(workspace);
    ResampleHdr* hdr = reinterpret_cast<ResampleHdr*>(ws);
    ws += align256(sizeof(ResampleHdr));
    double* edges = reinterpret_cast<double*>(ws);
    ws += align256((size_t)(n + 1) * sizeof(double));
    const size_t ib = align256((size_t)(n + 1) * sizeof(int));
    int* cnt_ws = reinterpret_cast<int*>(ws); ws += ib;
    int* big_row = reinterpret_cast<int*>(ws); ws += ib;
    int* big_cnt = reinterpret_cast<int*>(ws); ws += ib;
    int* start = reinterpret_cast<int*>(ws); ws += ib;
    int* cnt = counts ? counts : cnt_ws;
    rc = cuda_status(cudaFuncSetAttribute(rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRankSmem),
                     "cudaFuncSetAttribute(rank_kernel)");
    if (rc) return rc;
    launch_after(cdf_kernel, 1, kCdfThreads, 0, s, st->w, n, edges, cnt);
    launch_after(counts_kernel, blocks(n, 256), 256, 0, s, n, seed, st->epoch, edges, cnt);
    launch_after(rank_kernel, 1, kRankThreads, kRankSmem, s, n, cnt, big_row, big_cnt, start, hdr);
    launch_after(gather_kernel, (unsigned)(((long)n * p + 255) / 256), 256, 0, s, n, p,
                 st->beta, cnt, start, hdr, theta_in, prior_in, data_in, theta_out, prior_out, data_out, post_out);
    return launch_status("resample kernels");
}

extern "C" int ag_adapt_scaling(const ag_stage_state* st, double aw, double rw, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    adapt_kernel<<<1, 32, 0, as_stream(stream)>>>(aw, rw, st->counters, st->scaling, st->epoch);
    return launch_status("adapt_kernel");
}

// ---------------------------------------------------------------------------
// Allocation-free COV β schedule.
//
// Some callers cannot call cudaMalloc when they run a stage: hosts whose
// device memory is entirely reserved up front by another allocator or by a
// fixed memory budget, embedders that must not change their device footprint
// after start-up, and loops that must not enter the allocator at all because
// cudaMalloc and cudaFree may synchronise the device.  This entry point
// needs no caller workspace: its scratch (the schedule state, the grid
// barrier words and the partial moments) lives in a file-scope device array of fixed
// size, reserved when this file's module is loaded on a device and held by
// every device that loads it until the process exits.  Under CUDA's default
// lazy module loading the module is loaded by the first use of any kernel or
// symbol of this file (the first call of this entry point, ag_cov_schedule,
// ag_resample, ...), which may then enter the driver's allocator once:
// callers make such a call during start-up.
//
// * Limit: n <= kNoAllocMaxChains chains; larger n is rejected.
// * All calls share the one array, and it keeps the last call's contents:
//   calls whose work overlaps on the GPU (different streams, or a call made
//   before the previous one finished on another stream) race on it; issue
//   them in order on one stream.
// * The first call on each device looks up the array's device address
//   (cudaGetSymbolAddress) with that device current; make that first call
//   before any stream capture.
namespace {

constexpr int32_t kNoAllocMaxChains = 1 << 18;
constexpr size_t kNoAllocState = (sizeof(CovState) + 255) / 256 * 256;
constexpr size_t kNoAllocBytes =
    kNoAllocState + sizeof(GridBarrier) +
    cov_part_doubles(kNoAllocMaxChains) * sizeof(double);
static_assert(kNoAllocState == (sizeof(CovState) + 255) / 256 * 256, "no-alloc layout follows the workspace layout");
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned char g_cov_scratch[kNoAllocBytes];

std::mutex g_scratch_mutex;
void* g_scratch_addr[kNoAllocMaxDevices] = {};

int scratch_address(void** out) {
    int dev = 0;
    int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        return set_error(AG_ERR_SIZE, "device %d is beyond the %d devices this entry point tracks", dev,
                         kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        rc = cuda_status(cudaGetSymbolAddress(&p, g_cov_scratch), "cudaGetSymbolAddress(g_cov_scratch)");
        if (rc) return rc;
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return AG_OK;
}

}  // namespace

extern "C" int32_t ag_cov_schedule_noalloc_max_chains(void) { return kNoAllocMaxChains; }

extern "C" int ag_cov_schedule_noalloc(const ag_stage_state* st, const double* data_llk, int32_t n,
                                       double target, double tol, void* stream) {
    int rc = check_state(st);
    if (rc) return rc;
    AG_REQUIRE(data_llk != nullptr, "data_llk is NULL");
    if (n < 2 || n > kNoAllocMaxChains)
        return set_error(AG_ERR_SIZE,
                         "ag_cov_schedule_noalloc supports 2 to %d chains (got %d); use ag_cov_schedule "
                         "with a caller workspace for more",
                         kNoAllocMaxChains, n);
    void* scratch = nullptr;
    rc = scratch_address(&scratch);
    if (rc) return rc;
    cudaStream_t s = as_stream(stream);
    // the state block starts from zero on every call; the partials are written before they are read
    rc = cuda_status(cudaMemsetAsync(scratch, 0, kNoAllocState, s), "cudaMemsetAsync(scratch state)");
    if (rc) return rc;
    return cov_schedule_launch<false>(st, data_llk, n, target, tol, 0, kGridLevels + 1, scratch, s);
}
