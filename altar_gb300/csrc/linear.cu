// Linear Gaussian model on the 5th-generation tensor cores (tcgen05).
//
// The reference's linear model (models/linear/linear/Linear.py:152-185) forms
// r = G θ - d with a dgemm and whitens each chain's residual.  Here the data
// covariance is folded once into A = L⁻¹ G and b = L⁻¹ d (Cd = L Lᵀ), so that
// rᵀ Cd⁻¹ r = |A θ - b|², and each chain's misfit is
//     ρ = A (θ - θ₀) + ρ₀,   ρ₀ = A θ₀ - b  (FP64, the residual-correction pass),
// with θ₀ a centre of the population (the mean of up to 256 evenly spaced
// chains): the tensor-core product only carries the centred part.  A and
// δ = θ - θ₀ are split into BF16 pairs (x ≈ hi + lo) and
// the product A δ is one GEMM over the concatenated K axis
//     [δ_hi | δ_lo | δ_hi] · [A_hi | A_hi | A_lo]ᵀ
// (three BF16 products, FP32 accumulation; the dropped lo·lo term is
// ~2^-18 relative; δ is stored as [δ_hi | δ_lo], its first half read twice).  The GEMM is a persistent tcgen05 kernel: TMA loads
// 128B-swizzled K-major tiles into a 4-stage shared-memory ring guarded by
// mbarriers, one thread issues tcgen05.mma (M = 128 chains, N = 256
// observations, K = 16) into one of two TMEM accumulators, and four epilogue
// warps read the other accumulator with tcgen05.ld and reduce Σ (acc + ρ₀)²
// per chain straight from registers while the next tile's MMAs run.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "internal.h"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace ag {

// Persistent CTAs, one per SM, each taking tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...
// of 128 chains x 256 observations; partial[tile_n * n + chain] = Σ_obs (acc + ρ₀)².
// Warp roles: warp 0 lane 0 drives TMA through the TC_STAGES shared-memory ring, warp 1
// lane 0 issues tcgen05.mma into one of two TMEM accumulators (2 x 256 columns), warps
// 2-5 read the other accumulator with tcgen05.ld and reduce the previous tile, so the
// epilogue and the next tile's MMAs overlap.  Tiles are visited in groups of
// chain tiles (tile_group) so that CTAs running at the same time share both operands' k
// slices in L2.  Every wait is bounded; a timeout stops all roles, drains the copies
// and MMAs in flight and frees TMEM.
//
// LOWER: the second operand is lower triangular (W = L⁻¹), so a tile of observations n0 .. n0 + 255
// needs k < n0 + 256 only; the products left out are zeros (half the multiplications of a dense
// whitening were).  The kernel takes 296 µs for 3,000 observations and 16,384 chains (504 µs with the
// zeros).  The tiles of a group are taken longest first and every other round runs through the CTAs
// backwards, so that their loads even out; a group is as many chain tiles as keep their split rows in
// L2, since the fewer the groups, the less their ends cost.  Whole evaluations, against groups of
// eight chain tiles and one direction: 5,000 chains x 3,000 161 -> 130 µs, 5,000 x 1,300 66 -> 50,
// 8,192 x 1,200 70 -> 60, 16,384 x 3,000 388 -> 384 (groups of 48 MB 153, 51, 60, 377).  (Tiles from a
// common counter instead of a fixed stride, and the sum over observation tiles by the last CTA of a
// chain tile instead of a launch of its own, were slower: the fence before the count alone took 12 of
// 85 µs of the linear model.)
constexpr int TC_THREADS = 192;
constexpr uint32_t TC_SMEM = TC_STAGES * TC_STAGE_BYTES + 1024 /*align*/ + 256 /*bars*/;

// chain tiles per group
constexpr int TC_GROUP_M = 8;
constexpr size_t TC_GROUP_BYTES = 96u << 20;              // LOWER: split rows of a group, of 129 MB of L2
static inline int tile_group(bool lower, int mtiles, int kp) {
    if (!lower) return TC_GROUP_M;
    const size_t fit = TC_GROUP_BYTES / ((size_t)TC_BM * 2 * kp * sizeof(__nv_bfloat16));
    return fit < 1 ? 1 : fit < (size_t)mtiles ? (int)fit : mtiles;
}

// the i-th tile of this CTA, or `total` and more when there are none left
AG_DEVICE_INLINE int tile_of(int i, bool lower) {
    const int c = blockIdx.x, ctas = gridDim.x;
    return i * ctas + (lower && (i & 1) ? ctas - 1 - c : c);
}

AG_DEVICE_INLINE void tile_coords(int t, int mtiles, int ntiles, int group, bool lower, int& mt, int& nt) {
    const int span = group * ntiles;
    const int g = t / span, r = t % span;
    const int gm = (mtiles - g * group) < group ? (mtiles - g * group) : group;
    mt = g * group + r % gm;
    nt = lower ? ntiles - 1 - r / gm : r / gm;
}

template <bool LOWER>
__global__ void __launch_bounds__(TC_THREADS, 1)
linear_misfit_tc_kernel(const __grid_constant__ CUtensorMap map_a,   // chains x 2 kp (BF16)  [hi | lo]
                        const __grid_constant__ CUtensorMap map_b,   // obs    x 3 kp (BF16)  [hi | hi | lo]
                        int n, int m_obs, int kpb, int mtiles, int ntiles, int group,
                        const float* __restrict__ rho0, double* __restrict__ partial,
                        uint32_t* __restrict__ flags) {
    after_previous();
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + TC_STAGES * TC_STAGE_BYTES);
    uint64_t* full = bars;                       // [TC_STAGES]  TMA -> MMA
    uint64_t* empty = bars + TC_STAGES;          // [TC_STAGES]  MMA -> TMA
    uint64_t* tfull = bars + 2 * TC_STAGES;      // [2]          MMA -> epilogue
    uint64_t* tempty = bars + 2 * TC_STAGES + 2; // [2]          epilogue -> MMA
    uint64_t* drain = bars + 2 * TC_STAGES + 4;  // [1]          all MMAs done (teardown)
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ __align__(16) float s_rho[4][TC_BN];   // ρ₀ of the tile, a copy per epilogue warp

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = mtiles * ntiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 4);
        }
        mbar_init(drain, 1);
        fence_mbar_init();
        s_abort = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&s_tmem)), "r"(2 * TC_BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    auto aborted = [&]() { return *(volatile int*)&s_abort != 0; };
    // k blocks of each of the three products for observation tile nt
    auto blocks_of = [&](int nt) {
        const int need = (nt + 1) * (TC_BN / TC_BK);
        return LOWER && need < kpb ? need : kpb;
    };

    int issued = 0;                              // TMA stages issued (producer thread)
    if (warp == 0 && lane == 0) {
        // TMA producer: the stage ring runs on across tiles
        for (int i = 0, t; (t = tile_of(i, LOWER)) < total && !aborted(); ++i) {
            int mt, nt;
            tile_coords(t, mtiles, ntiles, group, LOWER, mt, nt);
            const int len = blocks_of(nt);
            // δ_hi A_hi, δ_lo A_hi, δ_hi A_lo: the first half's blocks serve twice on each side
            int g = 0, k = 0;
            for (int kb = 0; kb < 3 * len; ++kb, ++issued) {
                const int xa = (g == 1 ? kpb + k : k) * TC_BK, xb = (g == 2 ? 2 * kpb + k : k) * TC_BK;
                if (++k == len) {
                    k = 0;
                    ++g;
                }
                const int s = issued % TC_STAGES;
                if (issued >= TC_STAGES &&
                    !mbar_wait_bounded(&empty[s], (uint32_t)((issued / TC_STAGES) - 1) & 1u, TC_WAIT)) {
                    atomicExch(&s_abort, 1);
                    break;
                }
                if (aborted()) break;
                const uint32_t sa = base + s * TC_STAGE_BYTES;
                mbar_arrive_expect_tx(&full[s], TC_STAGE_BYTES);
                tma_load_2d(sa, &map_a, xa, mt * TC_BM, smem_addr(&full[s]));
                tma_load_2d(sa + TC_A_BYTES, &map_b, xb, nt * TC_BN, smem_addr(&full[s]));
            }
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer: tile j of this CTA accumulates into TMEM columns (j & 1) * 256
        const uint32_t idesc = idesc_bf16(TC_BM, TC_BN);
        int it = 0, local = 0;
        for (int t; (t = tile_of(local, LOWER)) < total && !aborted(); ++local) {
            const int b = local & 1;
            int mt, nt;
            tile_coords(t, mtiles, ntiles, group, LOWER, mt, nt);
            const int kblocks = 3 * blocks_of(nt);
            if (local >= 2 && !mbar_wait_bounded(&tempty[b], (uint32_t)((local >> 1) - 1) & 1u, TC_WAIT)) {
                atomicExch(&s_abort, 1);
                break;
            }
            tc_fence_after();
            const uint32_t acc_addr = tmem + (uint32_t)(b * TC_BN);
            bool ok = true;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int s = it % TC_STAGES;
                if (!mbar_wait_bounded(&full[s], (uint32_t)(it / TC_STAGES) & 1u, TC_WAIT)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = base + s * TC_STAGE_BYTES;
                const uint64_t adesc = sw128_desc(sa), bdesc = sw128_desc(sa + TC_A_BYTES);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)   // K = 16 per instruction: +32 bytes
                    mma_bf16(acc_addr, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                mma_commit(smem_addr(&empty[s]));
            }
            if (!ok) {
                atomicExch(&s_abort, 1);
                break;
            }
            mma_commit(smem_addr(&tfull[b]));    // fires when this tile's MMAs have completed
        }
        mma_commit(smem_addr(drain));            // fires when every issued MMA has completed
    } else if (warp >= 2) {
        // epilogue: thread = chain row (TMEM lane quarter of this warp), sums over observations
        const int quarter = warp & 3;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        float* rho = s_rho[quarter];
        int local = 0;
        for (int t; (t = tile_of(local, LOWER)) < total; ++local) {
            const int b = local & 1;
            int mt, nt;
            tile_coords(t, mtiles, ntiles, group, LOWER, mt, nt);
            const int n0 = nt * TC_BN;
            // observations past the end have zero rows in the operand: with ρ₀ = 0 they add nothing
#pragma unroll
            for (int c = lane; c < TC_BN; c += 32) rho[c] = n0 + c < m_obs ? __ldg(rho0 + n0 + c) : 0.f;
            const bool ok = __all_sync(0xffffffffu,
                                       mbar_wait_bounded(&tfull[b], (uint32_t)(local >> 1) & 1u, TC_WAIT));
            if (!ok || aborted()) {
                if (lane == 0) atomicExch(&s_abort, 1);
                break;
            }
            __syncwarp();
            tc_fence_after();
            const int chain = mt * TC_BM + quarter * 32 + lane;
            double acc = 0.0;
#pragma unroll 1
            for (int c0 = 0; c0 < TC_BN; c0 += 64) {
                // two 32-column loads in flight per wait
                uint32_t r0[32], r1[32];
                tmem_ld32_nowait(tmem + lane_base + (uint32_t)(b * TC_BN + c0), r0);
                tmem_ld32_nowait(tmem + lane_base + (uint32_t)(b * TC_BN + c0 + 32), r1);
                tmem_wait_ld();
                auto add = [&](const uint32_t (&r)[32], const float4* p) {
                    float sq = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i += 4) {
                        const float4 q = p[i >> 2];
                        float d = __uint_as_float(r[i]) + q.x;
                        sq = fmaf(d, d, sq);
                        d = __uint_as_float(r[i + 1]) + q.y;
                        sq = fmaf(d, d, sq);
                        d = __uint_as_float(r[i + 2]) + q.z;
                        sq = fmaf(d, d, sq);
                        d = __uint_as_float(r[i + 3]) + q.w;
                        sq = fmaf(d, d, sq);
                    }
                    acc += (double)sq;
                };
                add(r0, reinterpret_cast<const float4*>(rho + c0));
                add(r1, reinterpret_cast<const float4*>(rho + c0 + 32));
            }
            if (chain < n) partial[(size_t)nt * n + chain] = acc;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && aborted()) raise_flag(flags, DEV_ERR_TIMEOUT);
    if (warp == 0 && lane == 0 && aborted()) {
        // copies still in flight land before the CTA's shared memory goes away
        for (int k = (issued > TC_STAGES ? issued - TC_STAGES : 0); k < issued; ++k)
            mbar_wait_bounded(&full[k % TC_STAGES], (uint32_t)(k / TC_STAGES) & 1u, TC_WAIT);
    }
    if (warp == 1) {
        // every MMA this CTA issued has completed before TMEM is released
        mbar_wait_bounded(drain, 0, TC_WAIT);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TC_BN) : "memory");
    }
}

// Centring point θ₀ (or r̄): the mean of up to kCentreRows rows taken at an even stride.
// Any centre gives the same result, because ρ₀ = A θ₀ - b carries it exactly in FP64;
// the centre only has to lie inside the population so that the BF16 split of θ - θ₀ keeps
// its relative precision.  32 columns per CTA (lanes), the sampled rows split over the 8 warps
// (all of a warp's loads in flight at once), then the warp partial sums added in warp order.
// Beside the FP64 centre, its two leading FP32 parts (centre32).
constexpr int kCentreRows = 256;
static inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

template <class T>
__global__ void __launch_bounds__(256) centre_kernel(const T* __restrict__ x, int ld, int col0, int n, int cols,
                                                     double* __restrict__ centre, float2* __restrict__ centre32) {
    after_previous();
    __shared__ double part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    const int rows = n < kCentreRows ? n : kCentreRows;
    const long stride = n / rows;                      // >= 1
    T v[kCentreRows / 8];
#pragma unroll
    for (int q = 0; q < kCentreRows / 8; ++q) {
        const int k = warp + 8 * q;
        v[q] = (j < cols && k < rows) ? __ldg(x + (size_t)(k * stride) * ld + col0 + j) : (T)0;
    }
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kCentreRows / 8; ++q)
        if (warp + 8 * q < rows) s += (double)v[q];
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && j < cols) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += part[w][lane];
        t /= rows;
        centre[j] = t;
        const float hi = (float)t;
        centre32[j] = make_float2(hi, (float)(t - (double)hi));
    }
}

// a double rounded to FP32 in integer arithmetic (the conversion instruction runs at the FP64
// pipe's rate); values outside FP32's normal range take the instruction
AG_DEVICE_INLINE float to_f32(double d) {
    const uint64_t b = (uint64_t)__double_as_longlong(d);
    const int e = (int)(b >> 52) & 0x7ff;
    if (e < 1023 - 126 || e > 1023 + 126) return (float)d;
    const uint64_t m = b & 0x7FFFFFFFFFFFFFFFull;
    const uint64_t r = m + 0x0FFFFFFFull + ((m >> 29) & 1);          // to nearest, ties to even
    return __uint_as_float((uint32_t)(r >> 29) - ((1023u - 127u) << 23) | ((uint32_t)(b >> 32) & 0x80000000u));
}

// x - centre rounded to FP32.  θ in FP64: one subtraction.  Residuals in FP32 against the centre's
// two FP32 parts (48 bits): the exact error of x - hi takes the rest, so that only FP32
// instructions run (FP64 ones made the splits of 81 million residuals, 16,384 chains of
// 4,950, 455 µs and ρ₀ 45 µs more; with ρ₀ in the same launch they take 126 µs).
AG_DEVICE_INLINE float minus_centre(float x, float2 c) {
    float s, e;
    two_sum(x, -c.x, s, e);
    return s + (e - c.y);
}
AG_DEVICE_INLINE float minus_centre(double x, double c) { return to_f32(x - c); }

// Second launch of an evaluation, by CTAs of two kinds.  The first `rho_ctas`: ρ₀ = A θ₀ - b in
// FP64 (b = NULL: W r̄), one warp per observation; a lower triangular A is read up to its diagonal.
// The others: δ = x - centre split as [hi | lo] (BF16, row length 2 kp, kp = columns padded to
// 64), a thread per 8 consecutive columns of kSplitRows rows whose loads are all in flight
// together, two 16-byte stores a row.  Rows of x have stride ld and start at column col0 (θ:
// ld = p, col0 = 0; a residual block: the residual rows and the block's first column).
constexpr int kSplitRows = 2;
template <class T> struct CentreOf { typedef double type; };
template <> struct CentreOf<float> { typedef float2 type; };

template <class T, bool LOWER>
__global__ void __launch_bounds__(256) split_rho0_kernel(const T* __restrict__ x, int ld, int col0,
                                                         const double* __restrict__ centre,
                                                         const typename CentreOf<T>::type* __restrict__ shift, int n,
                                                         int cols, int kp, __nv_bfloat16* __restrict__ out, int rho_ctas,
                                                         const double* __restrict__ A, const double* __restrict__ b,
                                                         int m, float* __restrict__ rho0) {
    after_previous();
    if ((int)blockIdx.x < rho_ctas) {
        const int row = (int)blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
        if (row >= m) return;
        const int len = LOWER ? row + 1 : cols;
        double s = 0.0;
#pragma unroll 8
        for (int j = lane; j < len; j += 32) s = fma(__ldg(A + (size_t)row * cols + j), __ldg(centre + j), s);
        s = warp_sum(s);
        if (lane == 0) rho0[row] = (float)(b ? s - b[row] : s);
        return;
    }
    const int groups = kp >> 3;
    const long e = (long)((int)blockIdx.x - rho_ctas) * 256 + threadIdx.x;
    const long band = e / groups;
    const int j0 = (int)(e - band * groups) * 8;
    const long i0 = band * kSplitRows;
    if (i0 >= n) return;
    // 16-byte loads where the row segments are aligned for them
    const bool wide = j0 + 8 <= cols && ((size_t)(x + col0) % 16 == 0) && ((size_t)ld * sizeof(T)) % 16 == 0;
    __align__(16) T v[kSplitRows][8];
#pragma unroll
    for (int r = 0; r < kSplitRows; ++r) {
        const long i = i0 + r < n ? i0 + r : n - 1;
        const T* src = x + (size_t)i * ld + col0 + j0;
        if (wide) {
#pragma unroll
            for (int q = 0; q < (int)(8 * sizeof(T) / 16); ++q)
                reinterpret_cast<uint4*>(v[r])[q] = __ldg(reinterpret_cast<const uint4*>(src) + q);
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[r][q] = j0 + q < cols ? __ldg(src + q) : (T)0;
        }
    }
    // (the centre arrays are as long as a row's kp columns)
    typename CentreOf<T>::type c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = __ldg(shift + j0 + q);
#pragma unroll
    for (int r = 0; r < kSplitRows; ++r) {
        if (i0 + r >= n) break;
        __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float d = j0 + q < cols ? minus_centre(v[r][q], c[q]) : 0.f;
            hi[q] = __float2bfloat16_rn(d);
            lo[q] = __float2bfloat16_rn(d - __bfloat162float(hi[q]));
        }
        __nv_bfloat16* row = out + (size_t)(i0 + r) * 2 * kp;
        *reinterpret_cast<uint4*>(row + j0) = *reinterpret_cast<const uint4*>(hi);
        *reinterpret_cast<uint4*>(row + kp + j0) = *reinterpret_cast<const uint4*>(lo);
    }
}

// A split as [hi | hi | lo]; lower: its entries above the diagonal as zeros, whatever they hold
__global__ void split_a_kernel(const double* __restrict__ A, int m, int p, int kp, bool lower,
                               __nv_bfloat16* __restrict__ out) {
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)m * kp) return;
    const int i = (int)(e / kp), j = (int)(e % kp);
    const float a = (j < p && !(lower && j > i)) ? (float)A[(size_t)i * p + j] : 0.f;
    const __nv_bfloat16 hi = __float2bfloat16_rn(a);
    const __nv_bfloat16 lo = __float2bfloat16_rn(a - __bfloat162float(hi));
    __nv_bfloat16* row = out + (size_t)i * 3 * kp;
    row[j] = hi;
    row[kp + j] = hi;
    row[2 * kp + j] = lo;
}

__global__ void linear_reduce_kernel(int n, int tiles, const double* __restrict__ partial, double norm,
                                     double* __restrict__ llk, int accumulate) {
    after_previous();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
#pragma unroll 8
    for (int t = 0; t < tiles; ++t) s += partial[(size_t)t * n + i];
    llk[i] = (accumulate ? llk[i] : norm) - 0.5 * s;
}

// Exact FP64 path, llk = norm - ½ |A θ - b|², one warp per chain and observations over the lanes: for
// more parameters than the staged kernel below holds, and for the smallest products, whose two
// or three rounds do not pay for the staging (64 chains, 50 x 4: 4.2 µs against 6.2; 50 x 30: 10.3
// against 8.2)
constexpr int kExactSmall = 400;                        // observations x parameters
__global__ void linear_fp64_warp_kernel(const double* __restrict__ A, const double* __restrict__ b,
                                        const double* __restrict__ theta, int n, int m, int p, double norm,
                                        double* __restrict__ llk) {
    after_previous();
    const int chain = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (chain >= n) return;
    const double* th = theta + (size_t)chain * p;
    double acc = 0.0;
    for (int r = lane; r < m; r += 32) {
        double s = -b[r];
        for (int j = 0; j < p; ++j) s = fma(A[(size_t)r * p + j], th[j], s);
        acc = fma(s, s, acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) llk[chain] = norm - 0.5 * acc;
}

// The same, staged.  The floor is the FP64 pipe (64 cycles per warp
// instruction and scheduler).  A lane owns one of kExactChains chains and every kExactRows-th
// observation of its CTA's share.  Rows of A come through a double buffer of shared memory, filled
// ahead by asynchronous copies: read where they are used, each row's first touch of a line was a
// round trip to L2 that few warps per scheduler could not hide.  The observations are shared out
// over a cluster of 1 to 8 CTAs; lanes, warps and CTAs are added in a fixed order.
// 2,003 chains, 997 x 61: 264 -> 232 µs (216 are FP64 operations; 6% is the fullest SM's excess);
// 1,000 chains 196 -> 121, 64 chains 196 -> 31; 4,096 chains, 500 x 30: 140 -> 127.
constexpr int kExactWarps = 4;
constexpr int kExactThreads = kExactWarps * 32;
constexpr int kExactChains = 8;
constexpr int kExactRows = kExactThreads / kExactChains;
constexpr int kExactStage = 1024;                       // doubles of A per stage, at least kExactRows rows
constexpr int kExactMostP = 600;                        // parameters whose stages fit shared memory

// rounds of kExactRows rows per stage, and a CTA's dynamic shared memory: θ, two stages of A and b
__host__ __device__ __forceinline__ int exact_rounds(int p) {
    return p * kExactRows < kExactStage ? kExactStage / (p * kExactRows) : 1;
}
__host__ __device__ __forceinline__ size_t exact_smem(int p) {
    return ((size_t)p * kExactChains + 2 * (size_t)exact_rounds(p) * kExactRows * (p + 1)) * sizeof(double);
}

__global__ void __launch_bounds__(kExactThreads)
linear_fp64_kernel(const double* __restrict__ A, const double* __restrict__ b, const double* __restrict__ theta,
                   int n, int m, int p, double norm, int split, double* __restrict__ llk) {
    after_previous();
    extern __shared__ double s_theta[];                 // [p][kExactChains]
    __shared__ double s_part[kExactWarps][kExactChains], s_sum[kExactChains];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = blockIdx.x % split, c0 = blockIdx.x / split * kExactChains;
    const int chains = min(kExactChains, n - c0), tid = threadIdx.x;
    const int c = tid % kExactChains, row = tid / kExactChains;
    const int first = (int)((long)m * rank / split), end = (int)((long)m * (rank + 1) / split);
    double acc = 0.0;
    const int R = exact_rounds(p) * kExactRows;
    double* stage = s_theta + p * kExactChains;         // [2][R][p] A, [2][R] b
    double* stage_b = stage + 2 * R * p;
    auto load = [&](int r0, int buf) {
        const int rows = min(R, end - r0);
        const double* from = A + (size_t)r0 * p;
        for (int e = tid; e < rows * p; e += kExactThreads) cp_async8(stage + buf * R * p + e, from + e);
        for (int e = tid; e < rows; e += kExactThreads) cp_async8(stage_b + buf * R + e, b + r0 + e);
        cp_async_commit();
    };
    load(first, 0);
    for (int e = tid; e < p * kExactChains; e += kExactThreads) {
        const int q = e / p, j = e - q * p;
        s_theta[j * kExactChains + q] = theta[(size_t)(c0 + min(q, chains - 1)) * p + j];
    }
    int buf = 0;
    for (int r0 = first; r0 < end; r0 += R, buf ^= 1) {
        load(r0 + R, buf ^ 1);
        cp_async_wait<1>();
        __syncthreads();
        const int rows = min(R, end - r0);
        for (int r = row; r < rows; r += kExactRows) {
            const double* a = stage + (buf * R + r) * p;
            const double* th = s_theta + c;
            double s = -stage_b[buf * R + r];
            int j = 0;
            for (; j + 8 <= p; j += 8, th += 8 * kExactChains) {
                double u[8], v[8];                      // all loads before the chain of FMAs
#pragma unroll
                for (int q = 0; q < 8; ++q) u[q] = a[j + q], v[q] = th[q * kExactChains];
#pragma unroll
                for (int q = 0; q < 8; ++q) s = fma(u[q], v[q], s);
            }
            for (; j < p; ++j, th += kExactChains) s = fma(a[j], th[0], s);
            acc = fma(s, s, acc);
        }
        __syncthreads();
    }
    cp_async_wait<0>();
#pragma unroll
    for (int o = kExactChains; o < 32; o *= 2) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((tid & 31) < kExactChains) s_part[tid >> 5][c] = acc;
    __syncthreads();
    if (tid < kExactChains) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kExactWarps; ++w) s += s_part[w][tid];
        s_sum[tid] = s;
    }
    if (split > 1)
        cluster.sync();
    else
        __syncthreads();
    if (rank == 0 && tid < chains) {
        double s = s_sum[tid];
        for (int q = 1; q < split; ++q) s += cluster.map_shared_rank(s_sum, q)[tid];
        llk[c0 + tid] = norm - 0.5 * s;
    }
    if (split > 1) cluster.sync();                      // the sums stay until they have been read
}


}  // namespace ag

using namespace ag;

static inline size_t al256(size_t b) { return (b + 255) / 256 * 256; }

extern "C" int32_t ag_linear_kpad(int32_t p) { return p > 0 ? cdiv(p, TC_BK) * TC_BK : 0; }

static int split_a(const double* A, int m, int p, bool lower, uint16_t* a_split, void* stream) {
    AG_REQUIRE(A && a_split && m > 0 && p > 0, "invalid arguments");
    const int kp = ag_linear_kpad(p);
    split_a_kernel<<<cdiv((long)m * kp, 256), 256, 0, as_stream(stream)>>>(A, m, p, kp, lower,
                                                                         reinterpret_cast<__nv_bfloat16*>(a_split));
    return launch_status("split_a_kernel");
}

extern "C" int ag_linear_prepare(const double* A, int32_t m, int32_t p, uint16_t* a_split, void* stream) {
    return split_a(A, m, p, false, a_split, stream);
}

extern "C" int ag_whiten_prepare_lower(const double* W, int32_t m, uint16_t* w_split, void* stream) {
    return split_a(W, m, m, true, w_split, stream);
}

// workspace of an evaluation: centre [kp], FP64 and as two FP32 parts | ρ₀ [m] | split rows
// [n][2 kp] | partials [tiles][n]
static size_t eval_workspace(int m, int cols, int n) {
    const size_t kp = ag_linear_kpad(cols);
    return 2 * al256(kp * sizeof(double)) + al256((size_t)m * sizeof(float)) + al256((size_t)n * 2 * kp * 2) +
           al256((size_t)cdiv(m, TC_BN) * n * sizeof(double));
}

// llk = (accumulate ? llk : norm) - 1/2 |A (x - x̄) + ρ₀|², ρ₀ = A x̄ - b: the centre; the split of
// the centred rows with ρ₀; the tensor-core product with the fused misfit; the sum over tiles
template <class T, bool LOWER>
static int eval_llk(const T* x, int ld, int col0, int n, int cols, const double* a64, const double* b,
                    const uint16_t* a_split, int m, double norm, int accumulate, double* llk, void* workspace,
                    uint32_t* flags, cudaStream_t s) {
    const int kp = ag_linear_kpad(cols), tiles = cdiv(m, TC_BN), mtiles = cdiv(n, TC_BM);
    char* ws = static_cast<char*>(workspace);
    double* centre = reinterpret_cast<double*>(ws); ws += al256(kp * sizeof(double));
    float2* centre32 = reinterpret_cast<float2*>(ws); ws += al256(kp * sizeof(double));
    float* rho0 = reinterpret_cast<float*>(ws); ws += al256((size_t)m * sizeof(float));
    __nv_bfloat16* split = reinterpret_cast<__nv_bfloat16*>(ws); ws += al256((size_t)n * 2 * kp * 2);
    double* partial = reinterpret_cast<double*>(ws);
    launch_after(centre_kernel<T>, cdiv(cols, 32), 256, 0, s, x, ld, col0, n, cols, centre, centre32);
    int rc = launch_status("centre_kernel");
    if (rc) return rc;
    const typename CentreOf<T>::type* shift;
    if constexpr (sizeof(T) == 4)
        shift = centre32;
    else
        shift = centre;
    const int split_ctas = cdiv((long)cdiv(n, kSplitRows) * (kp / 8), 256);
    launch_after(split_rho0_kernel<T, LOWER>, cdiv(m, 8) + split_ctas, 256, 0, s, x, ld, col0, centre, shift, n,
                 cols, kp, split, cdiv(m, 8), a64, b, m, rho0);
    rc = launch_status("split_rho0_kernel");
    if (rc) return rc;
    CUtensorMap ma, mb;
    rc = make_map(&ma, split, n, 2 * kp, TC_BM);
    if (rc) return rc;
    rc = make_map(&mb, a_split, m, 3 * kp, TC_BN);
    if (rc) return rc;
    // per call: the attribute belongs to the current device's context
    rc = cuda_status(cudaFuncSetAttribute(linear_misfit_tc_kernel<LOWER>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM),
                     "cudaFuncSetAttribute(linear_misfit_tc_kernel)");
    if (rc) return rc;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    const int total = mtiles * tiles;
    launch_after(linear_misfit_tc_kernel<LOWER>, total < sms ? total : sms, TC_THREADS, TC_SMEM, s, ma, mb, n, m,
                 kp / TC_BK, mtiles, tiles, tile_group(LOWER, mtiles, kp), rho0, partial, flags);
    rc = launch_status("linear_misfit_tc_kernel");
    if (rc) return rc;
    launch_after(linear_reduce_kernel, cdiv(n, 128), 128, 0, s, n, tiles, partial, norm, llk, accumulate);
    return launch_status("linear_reduce_kernel");
}

extern "C" size_t ag_linear_workspace_bytes(int32_t m, int32_t p, int32_t n) {
    return m <= 0 || p <= 0 || n <= 0 ? 0 : eval_workspace(m, p, n);
}

extern "C" int ag_linear_llk(const ag_linear_model* lm, const double* theta, int32_t n, double norm,
                             double* llk, void* workspace, size_t workspace_bytes, uint32_t* flags,
                             void* stream) {
    AG_REQUIRE(lm && lm->a64 && lm->b64 && lm->a_split && theta && llk && n > 0, "invalid arguments");
    const int m = lm->m_obs, p = lm->p;
    AG_REQUIRE(m > 0 && p > 0, "invalid linear model sizes");
    const size_t need = ag_linear_workspace_bytes(m, p, n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "ag_linear_llk needs %zu bytes of 256-byte aligned workspace", need);
    AG_REQUIRE(aligned(lm->a_split, 16), "a_split must be 16-byte aligned");
    return eval_llk<double, false>(theta, p, 0, n, p, lm->a64, lm->b64, lm->a_split, m, norm, 0, llk, workspace, flags,
                                   as_stream(stream));
}

extern "C" size_t ag_whiten_workspace_bytes(int32_t m, int32_t n) {
    return m <= 0 || n <= 0 ? 0 : eval_workspace(m, m, n);
}

static int whiten_llk(bool lower, const ag_whiten_block* blk, const float* resid, int32_t ldr, int32_t n, double* llk,
                      void* workspace, size_t workspace_bytes, uint32_t* flags, void* stream) {
    AG_REQUIRE(blk && blk->w64 && blk->w_split && resid && llk && n > 0, "invalid arguments");
    const int m = blk->m, col0 = blk->col0;
    AG_REQUIRE(m > 0 && col0 >= 0 && col0 + m <= ldr, "block columns [%d, %d) outside rows of %d", col0, col0 + m,
               ldr);
    const size_t need = ag_whiten_workspace_bytes(m, n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "whitening needs %zu bytes of 256-byte aligned workspace", need);
    AG_REQUIRE(aligned(blk->w_split, 16), "w_split must be 16-byte aligned");
    cudaStream_t s = as_stream(stream);
    return lower ? eval_llk<float, true>(resid, ldr, col0, n, m, blk->w64, nullptr, blk->w_split, m, 0.0, 1, llk,
                                         workspace, flags, s)
                 : eval_llk<float, false>(resid, ldr, col0, n, m, blk->w64, nullptr, blk->w_split, m, 0.0, 1, llk,
                                          workspace, flags, s);
}

extern "C" int ag_whiten_llk(const ag_whiten_block* blk, const float* resid, int32_t ldr, int32_t n,
                             double* llk, void* workspace, size_t workspace_bytes, uint32_t* flags,
                             void* stream) {
    return whiten_llk(false, blk, resid, ldr, n, llk, workspace, workspace_bytes, flags, stream);
}

extern "C" int ag_whiten_llk_lower(const ag_whiten_block* blk, const float* resid, int32_t ldr, int32_t n,
                                   double* llk, void* workspace, size_t workspace_bytes, uint32_t* flags,
                                   void* stream) {
    return whiten_llk(true, blk, resid, ldr, n, llk, workspace, workspace_bytes, flags, stream);
}

extern "C" int ag_linear_llk_fp64(const ag_linear_model* lm, const double* theta, int32_t n, double norm,
                                  double* llk, void* stream) {
    AG_REQUIRE(lm && lm->a64 && lm->b64 && theta && llk && n > 0, "invalid arguments");
    if (lm->p <= 0 || lm->p > kExactMostP || (long)lm->m_obs * lm->p <= kExactSmall) {
        launch_after(linear_fp64_warp_kernel, cdiv((long)n * 32, 256), 256, 0, as_stream(stream),
                     lm->a64, lm->b64, theta, n, lm->m_obs, lm->p, norm, llk);
        return launch_status("linear_fp64_warp_kernel");
    }
    // The CTAs per group of chains: those whose fullest SM has the least to do, in FMAs per lane
    // with ~32 for a CTA's start, and a third more for a warp that has its scheduler to itself.
    // 997 x 61, one CTA against the chosen number: 64 chains 191 and 31 µs (8), 1,000: 191 and 121 (8),
    // 1,216: 191 and 144 (2), 2,003: 275 and 232 (4); 20,000 chains, 300 x 20: 232 (1) and 242 (4)
    const int groups = cdiv(n, kExactChains);
    long best = 0;
    int split = 1;
    for (int q = 1; q <= 8; q *= 2) {
        const long ctas = cdiv((long)groups * q, 152);
        const long cost = ctas * ((long)cdiv(lm->m_obs, (long)kExactRows * q) * lm->p + 32) * (ctas == 1 ? 4 : 3);
        if (q == 1 || cost < best) best = cost, split = q;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * split);
    cfg.blockDim = dim3(kExactThreads);
    cfg.dynamicSmemBytes = exact_smem(lm->p);
    cfg.stream = as_stream(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = split > 1;
    if (cfg.dynamicSmemBytes > 48 * 1024) {
        const int rc = cuda_status(cudaFuncSetAttribute(linear_fp64_kernel,
                                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)exact_smem(kExactMostP)),
                                   "cudaFuncSetAttribute(linear_fp64_kernel)");
        if (rc) return rc;
    }
    return cuda_status(cudaLaunchKernelEx(&cfg, linear_fp64_kernel, lm->a64, lm->b64, theta, (int)n,
                                          (int)lm->m_obs, (int)lm->p, norm, split, llk),
                       "cudaLaunchKernelEx(linear_fp64_kernel)");
}
