// Learned surrogate of the CDM LOS field and the delayed-acceptance steps.
//
// Network: dense layers y = x Wᵀ + b with GELU (x Φ(x)) between them and a
// linear output; weights kept as an FP32 master copy for Adam plus a BF16 copy
// that the forward and backward products read (FP32 accumulation).  Layer
// products are a tiled SIMT GEMM with fused bias / GELU epilogues.
//
// Surrogate log-likelihood: the network predicts K normalised PCA coefficients
// c of the LOS field; with the basis B (M x K), mean field μ and the diagonal
// weights W = Cd⁻¹, Σ_j w_j (ũ_j - d_j)² for ũ = μ + B diag(s) c is
//     q0 - 2 hᵀ c̃ + c̃ᵀ G c̃,  c̃ = s ⊙ c,  h = Bᵀ W (d - μ),  G = Bᵀ W B,
// so each chain costs O(K²) instead of O(M).
//
// Delayed acceptance (Christen & Fox 2005): stage 1 accepts the proposal on
// the surrogate posterior; only stage-1 survivors (compacted into an index
// list) get the exact likelihood; stage 2 accepts with
//     log u2 <= (post' - post) - (post̃' - post̃),
// which leaves the exact posterior invariant.
#include <math.h>
#include <stdint.h>
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "internal.h"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace ag {

constexpr int kMaxLayers = 8;
constexpr int BM = 64, BN = 64, BK = 16;

AG_DEVICE_INLINE float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
AG_DEVICE_INLINE float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) +
           z * 0.39894228040143268f * __expf(-0.5f * z * z);
}

enum Epilogue : int { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_GELU = 2 };

// C(m, n) = Σ_k A(m, k) B(k, n) with A(m,k) = A[m*sam + k*sak], B(k,n) = B[k*sbk + n*sbn]
// (B in BF16 or FP32), then the epilogue: + bias[n], GELU (pre-activation to Z).
//
// 64 x 64 output tile per CTA, 256 threads with 4 x 4 outputs each, k-tiles of 16 staged in
// shared memory; each operand is read along whichever of its two strides is 1 (coalesced
// rows of 16 k or of 64 m / n) and the next k-tile is prefetched into registers while the
// current one is multiplied.  Split K: the gridDim.z CTAs of one tile form a thread-block
// cluster, each multiplies one K range, and the partial tiles are summed through
// distributed shared memory in rank order (deterministic), each CTA reducing and writing
// BM / gridDim.z rows.
template <bool B_BF16>
AG_DEVICE_INLINE float load_b(const void* Bv, long idx) {
    return B_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(Bv)[idx])
                  : reinterpret_cast<const float*>(Bv)[idx];
}

// shares of K of an M x N product and their length: K is split when the output tiles alone would leave
// most of the GPU idle (the weight gradients: a few tiles, K = batch rows)
__host__ __device__ __forceinline__ int product_split(int M, int N, int K) {
    const int tiles = (N + BN - 1) / BN * ((M + BM - 1) / BM);
    int split = 1;
    while (split < 8 && tiles * split < 128 && K >= 2 * BK * (split * 2)) split *= 2;
    return split;
}
__host__ __device__ __forceinline__ int product_share(int K, int split) {
    return ((K + split - 1) / split + BK - 1) / BK * BK;
}

template <bool B_BF16>
__global__ void __launch_bounds__(256) gemm_kernel(int M, int N, int K, const float* __restrict__ A,
                                                   long sam, long sak, const void* __restrict__ Bv,
                                                   long sbk, long sbn, float* __restrict__ C, long ldc,
                                                   const float* __restrict__ bias, int epi,
                                                   float* __restrict__ Z) {
    __shared__ __align__(16) float As[BK][BM + 4];
    __shared__ __align__(16) float Bs[BK][BN + 4];
    __shared__ __align__(16) float Ps[BM][BN];          // partial tile (split K)
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int split = gridDim.z, part = blockIdx.z;
    const int kchunk = product_share(K, split);
    const int kb = min(K, part * kchunk), ke = min(K, kb + kchunk);
    // element e of a 16 x 64 operand tile: (k, m) with k fastest when that stride is 1
    const bool a_k1 = (sak == 1), b_k1 = (sbk == 1);
    float ra[4], rb[4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = tid + 256 * q;
            int kk = a_k1 ? e % BK : e / BM, mm = a_k1 ? e / BK : e % BM;
            int m = m0 + mm, k = k0 + kk;
            ra[q] = (m < M && k < ke) ? A[(long)m * sam + (long)k * sak] : 0.f;
            kk = b_k1 ? e % BK : e / BN;
            const int nn = b_k1 ? e / BK : e % BN;
            const int n = n0 + nn;
            k = k0 + kk;
            rb[q] = (n < N && k < ke) ? load_b<B_BF16>(Bv, (long)k * sbk + (long)n * sbn) : 0.f;
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = tid + 256 * q;
            As[a_k1 ? e % BK : e / BM][a_k1 ? e / BK : e % BM] = ra[q];
            Bs[b_k1 ? e % BK : e / BN][b_k1 ? e / BK : e % BN] = rb[q];
        }
    };
    float acc[4][4] = {};
    if (kb < ke) fetch(kb);
    for (int k0 = kb; k0 < ke; k0 += BK) {
        stash();
        __syncthreads();
        if (k0 + BK < ke) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    auto store = [&](int m, int n, float v) {
        if (m >= M || n >= N) return;
        if (epi != EPI_NONE) v += bias[n];
        if (epi == EPI_BIAS_GELU) {
            Z[(long)m * ldc + n] = v;
            v = gelu(v);
        }
        C[(long)m * ldc + n] = v;
    };
    if (split == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) store(m0 + ty * 4 + i, n0 + tx * 4 + j, acc[i][j]);
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(&Ps[ty * 4 + i][tx * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int rows = BM / split, r0 = part * rows;
    for (int e = tid; e < rows * BN; e += 256) {
        const int mm = r0 + e / BN, nn = e % BN;
        float v = 0.f;
        for (int r = 0; r < split; ++r) v += cluster.map_shared_rank(&Ps[0][0], r)[mm * BN + nn];
        store(m0 + mm, n0 + nn, v);
    }
    cluster.sync();                                     // partial tiles stay alive until all have read them
}


// ---------------------------------------------------------------------------
// Networks of widths up to kRowWidth (multiples of 8 behind the input): forward in one launch,
// backward in one launch per layer.  A training batch of 1,024 rows is ~0.13 GFLOP per layer
// product, a few microseconds of FP32 work that the tiled products spread over 15 µs of launch,
// load latency and reduction, 33 launches per batch.  Every sum is taken in the tiled products'
// order (shares of K by product_split, each one chain, the shares in order), so the results are
// theirs bit for bit; packed FMAs take two rows or columns, never two terms of a sum.
//
// Forward: a CTA takes kNetRows rows through all layers; the activations stay in shared memory as
// columns of eight rows, and the weights stream through a ring of chunks whose loads run ahead
// across the layers.  A chunk holds 64 columns of a layer's weights, 64 / split of each share, so
// that all shares advance together.  A thread owns four outputs of 2, 4 or 8 rows in one share: a
// shared-memory load of 16 bytes per lane costs four cycles also where all lanes read one address,
// so that one output per thread (8 cycles of loads per 4 packed FMAs) was bound by them.
// Bound by issue at two warps per scheduler and the barrier of each chunk.  10-256-256-256-256-64,
// 1,024 rows: 63.8 -> 35.1 µs.
constexpr int kRowWidth = 256;
constexpr int kNetRows = 8;
// rows that go forward here: 2,048 rows take 74 µs against 91 of the tiled products (256 wide), 21 against
// 27 (128), 15 against 25 (64); 4,096 rows 146 against 125, 38 against 33, 27 against 25, since every
// CTA streams all the weights
constexpr int kNetMost = 2048;
constexpr int kNetThreads = 256;
constexpr int kNetChunk = 64;                           // inputs per chunk of weights
constexpr int kNetStride = kNetChunk + 8;               // BF16 row in shared memory: no bank conflicts
constexpr int kNetStages = 4;
constexpr size_t kNetStage = (size_t)kRowWidth * kNetStride * sizeof(__nv_bfloat16);
constexpr int kNetSums = 4 * kNetRows * kRowWidth;      // floats: [share][row][output], 4 x 256 or 8 x 128
constexpr size_t kNetSmem = kNetStages * kNetStage + (2 * (size_t)kRowWidth * kNetRows + kNetSums) * sizeof(float);

// How the threads of a CTA divide a product of `rows` x `width` outputs with K terms: four outputs a
// thread, `slots` threads per four outputs, over the shares first and then over the rows.
struct NetSplit {
    int split, share, groups, row_groups;
};
__host__ __device__ __forceinline__ NetSplit net_split(int rows, int width, int K) {
    NetSplit v;
    v.split = product_split(rows, width, K);
    v.share = product_share(K, v.split);
    v.groups = width > kRowWidth / 2 ? kRowWidth / 4 : kRowWidth / 8;
    const int left = kNetThreads / v.groups / v.split;  // 0: more shares than slots
    v.row_groups = left > 4 ? 4 : left;
    return v;
}

struct NetLayers {
    int nlayers;
    int sizes[kMaxLayers + 1];
    int64_t w[kMaxLayers], b[kMaxLayers];
};

AG_DEVICE_INLINE f32x2 fma2_full(f32x2 a, f32x2 b, f32x2 c) {      // subnormals kept
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// the eight BF16 values of a 16-byte word as FP32
AG_DEVICE_INLINE void bf16x8(const uint4 v, float (&f)[8]) {
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f[2 * q] = __uint_as_float(u[q] << 16);
        f[2 * q + 1] = __uint_as_float(u[q] & 0xFFFF0000u);
    }
}

// one chain of a thread: four outputs x RP pairs of rows, over the eight weights of `w` and inputs `v`
template <int RP>
AG_DEVICE_INLINE void net_fma(f32x2 (&acc)[4][RP], const float (&w)[4], const float* v) {
    f32x2 x2[RP];
    if constexpr (RP == 1) {
        x2[0] = *reinterpret_cast<const f32x2*>(v);
    } else {
#pragma unroll
        for (int q = 0; q < RP; q += 2) {
            const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(v + 2 * q);
            x2[q] = u.x, x2[q + 1] = u.y;
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const f32x2 ww = pack2(w[j], w[j]);
#pragma unroll
        for (int q = 0; q < RP; ++q) acc[j][q] = fma2_full(x2[q], ww, acc[j][q]);
    }
}

// the chains of one layer, to s_red[share][row][output]; `next` waits for a chunk and returns its stage
template <int RP, class Next>
AG_DEVICE_INLINE void net_layer(const NetSplit d, int fi, int fo, const float* in, float* s_red, int stride, Next next) {
    const int slot = threadIdx.x / d.groups, first = threadIdx.x % d.groups;
    const int part = slot / d.row_groups, row = slot % d.row_groups * 2 * RP;
    const int len = kNetChunk / d.split;
    f32x2 acc[4][RP] = {};
    for (int s = 0; s < d.share; s += len) {
        const __nv_bfloat16* W = next() + part * len;
        if (part >= d.split) continue;
        const int k0 = part * d.share + s;
#pragma unroll 1
        for (int g = 0; g < len; g += 8) {
            if (s + g >= d.share || k0 + g >= fi) break;
            float w[4][8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int o = first + j * d.groups;     // rows past the last output: any values
                bf16x8(*reinterpret_cast<const uint4*>(W + (o < fo ? o : 0) * kNetStride + g), w[j]);
            }
            const float* v = in + (k0 + g) * kNetRows + row;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float wq[4] = {w[0][q], w[1][q], w[2][q], w[3][q]};
                net_fma<RP>(acc, wq, v + q * kNetRows);
            }
        }
    }
    if (part >= d.split) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int o = first + j * d.groups;
        if (o >= fo) break;
#pragma unroll
        for (int q = 0; q < RP; ++q) {
            float a, b;
            unpack2(acc[j][q], a, b);
            s_red[(part * kNetRows + row + 2 * q) * stride + o] = a;
            s_red[(part * kNetRows + row + 2 * q + 1) * stride + o] = b;
        }
    }
}

__global__ void __launch_bounds__(kNetThreads, 1)
net_forward_kernel(NetLayers net, const float* __restrict__ params, const __nv_bfloat16* __restrict__ wbf,
                   const float* __restrict__ x, int n, float* __restrict__ out, float* __restrict__ acts) {
    after_previous();
    extern __shared__ __align__(16) uint8_t s_net[];
    constexpr int kCols = kRowWidth * kNetRows;
    float* xT = reinterpret_cast<float*>(s_net + kNetStages * kNetStage);   // [2][kRowWidth][kNetRows]
    float* s_red = xT + 2 * kCols;
    const int tid = threadIdx.x;
    const long r0 = (long)blockIdx.x * kNetRows;
    const int rows = n - r0 < kNetRows ? (int)(n - r0) : kNetRows;
    int ql = 0, qs = 0, loaded = 0, used = 0;           // next chunk to load: layer, offset in the shares
    auto load = [&]() {
        if (ql < net.nlayers) {
            const int fi = net.sizes[ql], fo = net.sizes[ql + 1];
            const NetSplit d = net_split(n, fo, fi);
            const int len = kNetChunk / d.split;
            const __nv_bfloat16* W = wbf + net.w[ql];
            __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(s_net + (loaded % kNetStages) * kNetStage);
            constexpr int step = kNetThreads / (kNetChunk / 8);
            const int o = tid / (kNetChunk / 8), i = tid % (kNetChunk / 8) * 8;
            const int at = qs + i % len, k = i / len * d.share + at;       // eight inputs of one share
            if (at < d.share && k < fi) {
                if (fi % 8 == 0) {
                    const __nv_bfloat16* from = W + (size_t)o * fi + k;
#pragma unroll
                    for (int q = 0; q < kRowWidth / step; ++q, from += (size_t)step * fi)
                        if (o + q * step < fo) cp_async16(to + (o + q * step) * kNetStride + i, from);
                } else {                                // zeros past the last input
                    const unsigned short* w16 = reinterpret_cast<const unsigned short*>(W);
                    unsigned short* to16 = reinterpret_cast<unsigned short*>(to);
                    for (int q = o; q < fo; q += step)
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            to16[q * kNetStride + i + e] = k + e < fi ? __ldg(w16 + (size_t)q * fi + k + e) : 0;
                }
            }
            qs += len;
            if (qs >= d.share) {
                qs = 0;
                ++ql;
            }
        }
        cp_async_commit();
        ++loaded;
    };
    auto next = [&]() {
        cp_async_wait<kNetStages - 2>();
        __syncthreads();                                // the chunk and the layer's inputs are there
        load();                                         // into the stage that the previous chunk left
        return reinterpret_cast<const __nv_bfloat16*>(s_net + (used++ % kNetStages) * kNetStage);
    };
    for (int q = 0; q < kNetStages - 1; ++q) load();
    const int fi0 = net.sizes[0], pad0 = (fi0 + 7) / 8 * 8;
    for (int e = tid; e < pad0 * kNetRows; e += kNetThreads) {
        const int r = e / pad0, i = e - r * pad0;
        xT[i * kNetRows + r] = (r < rows && i < fi0) ? x[(r0 + r) * fi0 + i] : 0.f;
    }
    float* a = acts;
    for (int l = 0; l < net.nlayers; ++l) {
        const int fi = net.sizes[l], fo = net.sizes[l + 1];
        const bool last = l == net.nlayers - 1;
        const float* in = xT + (l & 1) * kCols;
        float* to = xT + ((l + 1) & 1) * kCols;
        const int stride = fo > kRowWidth / 2 ? kRowWidth : kRowWidth / 2;
        const int o = tid % stride, step = kNetThreads / stride;       // an output's eight rows, or four
        const float bias = o < fo ? params[net.b[l] + o] : 0.f;
        const NetSplit d = net_split(n, fo, fi);
        if (d.row_groups == 4)
            net_layer<1>(d, fi, fo, in, s_red, stride, next);
        else if (d.row_groups == 2)
            net_layer<2>(d, fi, fo, in, s_red, stride, next);
        else
            net_layer<4>(d, fi, fo, in, s_red, stride, next);
        __syncthreads();
        if (o < fo) {
            constexpr int R = kNetRows / 2;
            for (int h = tid / stride; h < 2; h += step) {
                float z[R] = {};
#pragma unroll 4
                for (int q = 0; q < d.split; ++q)
#pragma unroll
                    for (int r = 0; r < R; ++r) z[r] += s_red[(q * kNetRows + h * R + r) * stride + o];
                float y[R];
                const long at = (r0 + h * R) * fo + o;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    z[r] += bias;
                    y[r] = last ? z[r] : gelu(z[r]);
                    if (h * R + r >= rows) continue;
                    if (last) {
                        out[at + r * fo] = y[r];
                    } else {
                        a[at + r * fo] = z[r];
                        a[(long)n * fo + at + r * fo] = y[r];
                    }
                }
                *reinterpret_cast<float4*>(to + o * kNetRows + h * R) = make_float4(y[0], y[1], y[2], y[3]);
            }
        }
        a += 2 * (long)n * fo;
    }
    cp_async_wait<0>();
}

// the chains of one row block's dX = dZ W, to s_red[share][row][column]
template <int RP>
AG_DEVICE_INLINE void net_back_rows(const NetSplit d, int fi, int fo, const __nv_bfloat16* __restrict__ W,
                                    const float* zT, float* s_red, int stride) {
    const int slot = threadIdx.x / d.groups, i = threadIdx.x % d.groups * 4;
    const int part = slot / d.row_groups, row = slot % d.row_groups * 2 * RP;
    if (part >= d.split || i >= fi) return;
    const uint2* w = reinterpret_cast<const uint2*>(W + i);
    const int end = min(fo, (part + 1) * d.share);
    f32x2 acc[4][RP] = {};
#pragma unroll 16
    for (int o = part * d.share; o < end; ++o) {
        const uint2 u = __ldg(w + (size_t)o * (fi / 4));
        const float f[4] = {__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u),
                            __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u)};
        net_fma<RP>(acc, f, zT + o * kNetRows + row);
    }
#pragma unroll
    for (int q = 0; q < RP; ++q) {
        float a[4], b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(acc[j][q], a[j], b[j]);
        float* to = s_red + (part * kNetRows + row + 2 * q) * stride + i;
        *reinterpret_cast<float4*>(to) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(to + stride) = make_float4(b[0], b[1], b[2], b[3]);
    }
}

// Backward through one layer: CTAs of three kinds in clusters of kBackSplit.  The first `row_ctas` take
// kNetRows rows each: dX = dZ W and, behind it, the previous layer's dZ = dX ⊙ GELU'(Z) (a thread per
// four columns and 2, 4 or 8 rows of a share; W's rows stream from L2).  The next `sum_ctas` take eight
// columns each for the bias's gradient, as colsum_kernel sums them.  Then a cluster per 64 x 64 tile
// of dW = dZᵀ h: its CTAs take a share of the rows each, through double-buffered slabs of 64, with
// 8 x 4 outputs in each of 128 threads (12 cycles of shared-memory loads per 16 packed FMAs; 4 x 4 in
// 256 take 8 per 8), and add their tiles through distributed shared memory in rank order.
// 10-256-256-256-256-64: 173 -> 65 µs at 1,024 rows, 2,472 -> 1,701 µs at 32,768.  At 1,024 rows a
// layer's 15 µs are launch, load latency, ~4 µs of sums and the two cluster barriers in sequence.
constexpr int kBackSplit = 8;
constexpr int kBackSlab = 64;
constexpr int kBackTile = 64;
constexpr size_t kBackSmem = 4 * (size_t)kBackSlab * kBackTile * sizeof(float);
static_assert(kBackSlab == kBackTile, "the tile's sums take a slab's place");
static_assert((kRowWidth * kNetRows + kNetSums) * sizeof(float) <= kBackSmem, "row CTAs");

__global__ void __launch_bounds__(kNetThreads, 2)
net_backward_kernel(int n, int fi, int fo, const float* __restrict__ dZ, const __nv_bfloat16* __restrict__ W,
                    const float* __restrict__ Zprev, float* __restrict__ dprev, int row_ctas, int sum_ctas,
                    const float* __restrict__ h, int htiles, float* __restrict__ dW, float* __restrict__ db) {
    after_previous();
    extern __shared__ __align__(16) float s_back[];
    const int tid = threadIdx.x;
    int block = blockIdx.x;
    if (block < row_ctas) {
        const long r0 = (long)block * kNetRows;
        if (r0 >= n) return;
        const int rows = n - r0 < kNetRows ? (int)(n - r0) : kNetRows;
        float* zT = s_back;                             // [fo][kNetRows]
        float* s_red = zT + kRowWidth * kNetRows;
        float z[kNetRows];
        if (tid < fo) {
#pragma unroll
            for (int r = 0; r < kNetRows; ++r) z[r] = r < rows ? __ldg(dZ + (r0 + r) * fo + tid) : 0.f;
            *reinterpret_cast<float4*>(zT + tid * kNetRows) = make_float4(z[0], z[1], z[2], z[3]);
            *reinterpret_cast<float4*>(zT + tid * kNetRows + 4) = make_float4(z[4], z[5], z[6], z[7]);
        }
        if (tid < fi) {                                 // for the end; the loads run behind the sums
#pragma unroll
            for (int r = 0; r < kNetRows; ++r) z[r] = r < rows ? __ldg(Zprev + (r0 + r) * fi + tid) : 0.f;
        }
        __syncthreads();
        const NetSplit d = net_split(n, fi, fo);
        const int stride = fi > kRowWidth / 2 ? kRowWidth : kRowWidth / 2;
        if (d.row_groups == 4)
            net_back_rows<1>(d, fi, fo, W, zT, s_red, stride);
        else if (d.row_groups == 2)
            net_back_rows<2>(d, fi, fo, W, zT, s_red, stride);
        else
            net_back_rows<4>(d, fi, fo, W, zT, s_red, stride);
        __syncthreads();
        if (tid < fi) {
            float v[kNetRows] = {};
#pragma unroll 2
            for (int q = 0; q < d.split; ++q)
#pragma unroll
                for (int r = 0; r < kNetRows; ++r) v[r] += s_red[(q * kNetRows + r) * stride + tid];
#pragma unroll
            for (int r = 0; r < kNetRows; ++r)
                if (r < rows) dprev[(r0 + r) * fi + tid] = v[r] * gelu_grad(z[r]);
        }
        return;
    }
    block -= row_ctas;
    if (block < sum_ctas) {
        // thread t: rows t, t + 256, ... of eight columns; then the tree over t, a warp per column
        const int c0 = block * 8;
        if (c0 >= fo) return;
        float v[8] = {};
        for (int i = tid; i < n; i += kNetThreads) {
            const float* z = dZ + (size_t)i * fo + c0;
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] += __ldg(z + c);
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) s_back[c * kNetThreads + tid] = v[c];
        __syncthreads();
        const int lane = tid & 31, c = tid >> 5;
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = s_back[c * kNetThreads + 32 * q + lane];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < o; ++q) v[q] += v[q + o];
        for (int o = 16; o > 0; o >>= 1) v[0] += __shfl_down_sync(0xffffffffu, v[0], o);
        if (lane == 0) db[c0 + c] = v[0];
        return;
    }
    block -= sum_ctas;
    const int tile = block / kBackSplit, rank = block % kBackSplit;
    const int m0 = tile / htiles * kBackTile, n0 = tile % htiles * kBackTile;
    float* As = s_back;                                 // [2][kBackSlab][kBackTile] dZ
    float* Bs = As + 2 * kBackSlab * kBackTile;         // [2][kBackSlab][kBackTile] h
    float* Ps = s_back;                                 // afterwards: [kBackTile][kBackTile] sums of the share
    const int share = product_share(n, product_split(fo, fi, n));
    const int kb = min(n, rank * share), ke = min(n, kb + share);
    auto slab = [&](const float* src, int ld, int c0, int k0, float* to) {
        if (c0 + kBackTile <= ld && ld % 4 == 0 && (size_t)src % 16 == 0) {
#pragma unroll
            for (int q = 0; q < kBackSlab * kBackTile / 4 / kNetThreads; ++q) {
                const int e = q * kNetThreads + tid, k = e / (kBackTile / 4), c = e % (kBackTile / 4) * 4;
                const bool take = k0 + k < ke;
                cp_async_or_zero<16>(to + k * kBackTile + c, take ? src + (size_t)(k0 + k) * ld + c0 + c : src, take);
            }
        } else {
#pragma unroll 4
            for (int q = 0; q < kBackSlab * kBackTile / kNetThreads; ++q) {
                const int e = q * kNetThreads + tid, k = e / kBackTile, c = e % kBackTile;
                const bool take = k0 + k < ke && c0 + c < ld;
                cp_async_or_zero<4>(to + e, take ? src + (size_t)(k0 + k) * ld + c0 + c : src, take);
            }
        }
    };
    auto load = [&](int k0, int buf) {
        if (k0 < ke) {
            slab(dZ, fo, m0, k0, As + buf * kBackSlab * kBackTile);
            slab(h, fi, n0, k0, Bs + buf * kBackSlab * kBackTile);
        }
        cp_async_commit();
    };
    const int tx = tid % 16, ty = tid / 16 % 8;
    const bool sums = tid < kNetThreads / 2;
    f32x2 acc[8][2] = {};                               // rows ty * 4 + {0-3, 32-35}, columns tx * 4 + {0-3}
    load(kb, 0);
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += kBackSlab, buf ^= 1) {
        load(k0 + kBackSlab, buf ^ 1);
        cp_async_wait<1>();
        __syncthreads();
        const float* A = As + buf * kBackSlab * kBackTile + ty * 4;
        const float* B = Bs + buf * kBackSlab * kBackTile + tx * 4;
        if (sums) {
#pragma unroll 8
            for (int k = 0; k < kBackSlab; ++k) {
                const float4 a0 = *reinterpret_cast<const float4*>(A + k * kBackTile);
                const float4 a1 = *reinterpret_cast<const float4*>(A + k * kBackTile + 32);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(B + k * kBackTile);
                const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f32x2 aa = pack2(av[i], av[i]);
                    acc[i][0] = fma2_full(b.x, aa, acc[i][0]);
                    acc[i][1] = fma2_full(b.y, aa, acc[i][1]);
                }
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    if (sums) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            *reinterpret_cast<ulonglong2*>(Ps + (i / 4 * 32 + ty * 4 + i % 4) * kBackTile + tx * 4) =
                make_ulonglong2(acc[i][0], acc[i][1]);
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    constexpr int band = kBackTile / kBackSplit;
    for (int e = tid; e < band * kBackTile; e += kNetThreads) {
        const int i = rank * band + e / kBackTile, j = e % kBackTile;
        float v = 0.f;
#pragma unroll
        for (int r = 0; r < kBackSplit; ++r) v += cluster.map_shared_rank(Ps, r)[i * kBackTile + j];
        if (m0 + i < fo && n0 + j < fi) dW[(size_t)(m0 + i) * fi + n0 + j] = v;
    }
    cluster.sync();                                     // the tiles stay until all have read them
}

// ---------------------------------------------------------------------------
// Network layers on the tcgen05 tensor cores (inference).  A layer is
//     C (n x fo) = X Wᵀ,  then + b and GELU (all but the last layer),
// with X held as split BF16 rows [x_hi | x_lo] (x ≈ x_hi + x_lo, K' = 2 kp, kp = fi rounded
// up to 64) and W packed as [W | W] (fo x K', zeros past fi), so one BF16 GEMM over K' gives
// x_hi W + x_lo W in FP32 accumulators: the activations keep ~16 bits beyond BF16 and the
// weights are the BF16 copy the SIMT layers read too.  The kernel is the linear model's
// persistent tcgen05 structure (TMA ring of 128B-swizzled K-major tiles, one thread issuing
// tcgen05.mma into one of two TMEM accumulators, epilogue warps reading the other with
// tcgen05.ld); the epilogue adds the bias, applies GELU and writes the next layer's split
// BF16 input directly, plus the FP32 pre-activation Z and output Y where asked.
// The epilogue is what a layer cannot hide: ~35 instructions an element, most of them the error
// function's.  Tiles of 64 columns, two CTAs per SM with eight epilogue warps each, leave the last
// wave nearly full (32,768 rows: 7 tiles per SM where the mean is 6.7; of 256 columns 2 where it is
// 1.7).  They read X four times, so a CTA keeps to one block of columns and holds its weights (up to
// kMlpHeld inputs; both halves of K' use the same ones), which leaves X alone to stream from L2.
// Layers of 10-256-256-256-256-64, from tiles of 256 columns and one CTA per SM with 16 epilogue
// warps: 256 rows 60 -> 33 µs, 8,192 64 -> 44, 32,768 110 -> 101, 65,536 233 -> 177 (tiles of 128 columns:
// 37, 42, 105, 185); 10-64-128-64 loses 8% at 65,536 (43 -> 46).
constexpr int kMlpCols = 64;                                 // columns of a tile
constexpr int kMlpEpi = 8;                                   // epilogue warps, 32 columns each
constexpr int kMlpThreads = 64 + 32 * kMlpEpi;
constexpr int kMlpCtas = 2;                                  // per SM
constexpr uint32_t kMlpW = kMlpCols * TC_BK * 2;             // bytes of a K-block of weights
constexpr int kMlpHeld = TC_STAGES * TC_BK;                  // the held weights take the ring's place for them
constexpr uint32_t kMlpSmem = TC_STAGES * (TC_A_BYTES + kMlpW) + 1024 + 256;

__global__ void __launch_bounds__(kMlpThreads, kMlpCtas)
mlp_layer_tc_kernel(const __grid_constant__ CUtensorMap map_x,   // n  x K' split BF16 activations
                    const __grid_constant__ CUtensorMap map_w,   // fo x K' packed BF16 weights
                    int n, int fo, int kblocks, int mtiles, int ntiles, const float* __restrict__ bias,
                    int gelu_on, float* __restrict__ Z, float* __restrict__ Y,
                    __nv_bfloat16* __restrict__ xnext, int kp_next, uint32_t* __restrict__ flags) {
    constexpr uint32_t STAGE = TC_A_BYTES + kMlpW;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_addr(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + TC_STAGES * STAGE);
    uint64_t* full = bars;
    uint64_t* empty = bars + TC_STAGES;
    uint64_t* tfull = bars + 2 * TC_STAGES;
    uint64_t* tempty = bars + 2 * TC_STAGES + 2;
    uint64_t* drain = bars + 2 * TC_STAGES + 4;
    uint64_t* wfull = bars + 2 * TC_STAGES + 5;
    constexpr int EPI = kMlpEpi, COLS = 32, BN = kMlpCols;   // COLS: columns per epilogue warp
    // held weights: K-blocks behind the ring's A tiles; else next to each A tile
    const bool held = kblocks * TC_BK <= 2 * kMlpHeld;
    const uint32_t astep = held ? TC_A_BYTES : STAGE;
    const uint32_t wbase = base + TC_STAGES * TC_A_BYTES;
    const int nt = blockIdx.x % ntiles, m0 = blockIdx.x / ntiles, mstep = gridDim.x / ntiles;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ __align__(16) float s_bias[EPI][COLS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int st = 0; st < TC_STAGES; ++st) {
            mbar_init(&full[st], 1);
            mbar_init(&empty[st], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], EPI);
        }
        mbar_init(drain, 1);
        mbar_init(wfull, 1);
        fence_mbar_init();
        s_abort = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&s_tmem)), "r"(2 * BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    auto aborted = [&]() { return *(volatile int*)&s_abort != 0; };
    // the weights were packed at least two launches back (the rows are split in between), so they may be
    // read before the wait
    if (held && threadIdx.x == 0) {
        mbar_arrive_expect_tx(wfull, kblocks / 2 * kMlpW);
        for (int kb = 0; kb < kblocks / 2; ++kb)
            tma_load_2d(wbase + kb * kMlpW, &map_w, kb * TC_BK, nt * BN, smem_addr(wfull));
    }
    after_previous();

    int issued = 0;
    if (warp == 0 && lane == 0) {
        for (int mt = m0; mt < mtiles && !aborted(); mt += mstep) {
            for (int kb = 0; kb < kblocks; ++kb, ++issued) {
                const int st = issued % TC_STAGES;
                if (issued >= TC_STAGES &&
                    !mbar_wait_bounded(&empty[st], (uint32_t)((issued / TC_STAGES) - 1) & 1u, TC_WAIT)) {
                    atomicExch(&s_abort, 1);
                    break;
                }
                if (aborted()) break;
                const uint32_t sa = base + st * astep;
                mbar_arrive_expect_tx(&full[st], astep);
                tma_load_2d(sa, &map_x, kb * TC_BK, mt * TC_BM, smem_addr(&full[st]));
                if (!held) tma_load_2d(sa + TC_A_BYTES, &map_w, kb * TC_BK, nt * BN, smem_addr(&full[st]));
            }
        }
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = idesc_bf16(TC_BM, BN);
        int it = 0, local = 0;
        if (held && !mbar_wait_bounded(wfull, 0, TC_WAIT)) atomicExch(&s_abort, 1);
        for (int mt = m0; mt < mtiles && !aborted(); mt += mstep, ++local) {
            const int b = local & 1;
            if (local >= 2 && !mbar_wait_bounded(&tempty[b], (uint32_t)((local >> 1) - 1) & 1u, TC_WAIT)) {
                atomicExch(&s_abort, 1);
                break;
            }
            tc_fence_after();
            const uint32_t acc_addr = tmem + (uint32_t)(b * BN);
            bool ok = true;
            for (int kb = 0; kb < kblocks; ++kb, ++it) {
                const int st = it % TC_STAGES;
                if (!mbar_wait_bounded(&full[st], (uint32_t)(it / TC_STAGES) & 1u, TC_WAIT)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t sa = base + st * astep;
                const uint64_t adesc = sw128_desc(sa);
                const uint64_t bdesc = sw128_desc(held ? wbase + kb % (kblocks / 2) * kMlpW : sa + TC_A_BYTES);
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)
                    mma_bf16(acc_addr, adesc + 2 * k, bdesc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                mma_commit(smem_addr(&empty[st]));
            }
            if (!ok) {
                atomicExch(&s_abort, 1);
                break;
            }
            mma_commit(smem_addr(&tfull[b]));
        }
        mma_commit(smem_addr(drain));
    } else if (warp >= 2) {
        // epilogue: thread = row of the tile (TMEM lane quarter of this warp), the warps of a
        // quarter share the columns
        const int quarter = warp & 3, first = (warp - 2) / 4 * COLS;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        float* bs = s_bias[warp - 2];
        int local = 0;
        const int n0 = nt * BN + first;                                // fo is a multiple of BN
        bs[lane] = __ldg(bias + n0 + lane);
        __syncwarp();
        for (int mt = m0; mt < mtiles; mt += mstep, ++local) {
            const int b = local & 1;
            const bool ok = __all_sync(0xffffffffu,
                                       mbar_wait_bounded(&tfull[b], (uint32_t)(local >> 1) & 1u, TC_WAIT));
            if (!ok || aborted()) {
                if (lane == 0) atomicExch(&s_abort, 1);
                break;
            }
            __syncwarp();
            tc_fence_after();
            const int row = mt * TC_BM + quarter * 32 + lane;
            const bool live = row < n;
            uint32_t r[32];
            tmem_ld32_nowait(tmem + lane_base + (uint32_t)(b * BN + first), r);
            tmem_wait_ld();
            // the accumulator is free for the next tile but one
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[b]);
            const size_t o = (size_t)row * fo + n0;
            __nv_bfloat16* hi = xnext + (size_t)row * (2 * kp_next) + n0;
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
                float z[8], y[8];
#pragma unroll
                for (int q = 0; q < 8; q += 4) {
                    const float4 bb = *reinterpret_cast<const float4*>(bs + i + q);
                    z[q] = __uint_as_float(r[i + q]) + bb.x;
                    z[q + 1] = __uint_as_float(r[i + q + 1]) + bb.y;
                    z[q + 2] = __uint_as_float(r[i + q + 2]) + bb.z;
                    z[q + 3] = __uint_as_float(r[i + q + 3]) + bb.w;
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) y[q] = gelu_on ? gelu(z[q]) : z[q];
                if (live && Z) {
#pragma unroll
                    for (int q = 0; q < 8; q += 4)
                        *reinterpret_cast<float4*>(Z + o + i + q) = make_float4(z[q], z[q + 1], z[q + 2], z[q + 3]);
                }
                if (live && Y) {
#pragma unroll
                    for (int q = 0; q < 8; q += 4)
                        *reinterpret_cast<float4*>(Y + o + i + q) = make_float4(y[q], y[q + 1], y[q + 2], y[q + 3]);
                }
                if (live && xnext) {
                    __align__(16) __nv_bfloat162 h2[4], l2[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        h2[q] = __floats2bfloat162_rn(y[2 * q], y[2 * q + 1]);
                        l2[q] = __floats2bfloat162_rn(y[2 * q] - __low2float(h2[q]),
                                                      y[2 * q + 1] - __high2float(h2[q]));
                    }
                    *reinterpret_cast<uint4*>(hi + i) = *reinterpret_cast<const uint4*>(h2);
                    *reinterpret_cast<uint4*>(hi + kp_next + i) = *reinterpret_cast<const uint4*>(l2);
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && aborted()) raise_flag(flags, DEV_ERR_TIMEOUT);
    if (warp == 0 && lane == 0 && aborted()) {
        for (int k = (issued > TC_STAGES ? issued - TC_STAGES : 0); k < issued; ++k)
            mbar_wait_bounded(&full[k % TC_STAGES], (uint32_t)(k / TC_STAGES) & 1u, TC_WAIT);
    }
    if (warp == 0 && held) mbar_wait_bounded(wfull, 0, TC_WAIT);
    if (warp == 1) mbar_wait_bounded(drain, 0, TC_WAIT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
    }
}

// x (n x fi FP32) -> split BF16 rows [x_hi | 0 .. | x_lo | 0 ..] of width 2 kp; a thread per 8
// columns of a row
__global__ void split_rows_kernel(const float* __restrict__ x, int n, int fi, int kp,
                                  __nv_bfloat16* __restrict__ xs) {
    after_previous();
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int groups = kp >> 3;
    const long r = e / groups;
    const int k0 = (int)(e - r * groups) * 8;
    if (r >= n) return;
    __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float v = (k0 + q < fi) ? __ldg(x + r * fi + k0 + q) : 0.f;
        hi[q] = __float2bfloat16_rn(v);
        lo[q] = __float2bfloat16_rn(v - __bfloat162float(hi[q]));
    }
    *reinterpret_cast<uint4*>(xs + r * 2 * kp + k0) = *reinterpret_cast<const uint4*>(hi);
    *reinterpret_cast<uint4*>(xs + r * 2 * kp + kp + k0) = *reinterpret_cast<const uint4*>(lo);
}

// W (fo x fi BF16) -> [W | W] of width 2 kp, zeros past fi
__global__ void pack_weights_kernel(const __nv_bfloat16* __restrict__ w, int fo, int fi, int kp,
                                    __nv_bfloat16* __restrict__ out) {
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long)fo * kp) return;
    const int o = (int)(e / kp), k = (int)(e % kp);
    const __nv_bfloat16 v = (k < fi) ? w[(size_t)o * fi + k] : __float2bfloat16_rn(0.f);
    out[(size_t)o * 2 * kp + k] = v;
    out[(size_t)o * 2 * kp + kp + k] = v;
}

// θ (FP64, N x p) -> x = 2 (θ - lo)/(hi - lo) - 1 (FP32).  A thread keeps to one parameter j and
// walks the rows, so that the division (~20 FP64 instructions) is made once for its rows; the FP32
// result differs from the division's by its last bit at most, once in 2^28 elements.
constexpr int kNormRows = 8;
__global__ void normalize_kernel(const double* __restrict__ theta, int n, int p,
                                 const double* __restrict__ lo, const double* __restrict__ hi,
                                 float* __restrict__ x) {
    after_previous();
    const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const long band = e / p;
    const int j = (int)(e - band * p);
    const long i0 = band * kNormRows;
    if (i0 >= n) return;
    const double l = lo[j], s = 2.0 / (hi[j] - l);
    double v[kNormRows];
#pragma unroll
    for (int q = 0; q < kNormRows; ++q) v[q] = i0 + q < n ? __ldg(theta + (i0 + q) * p + j) : 0.0;
#pragma unroll
    for (int q = 0; q < kNormRows; ++q)
        if (i0 + q < n) x[(i0 + q) * p + j] = (float)fma(v[q] - l, s, -1.0);
}

// dZ = dY ⊙ GELU'(Z)
__global__ void gelu_back_kernel(long n, const float* __restrict__ Z, float* __restrict__ dY) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) dY[e] *= gelu_grad(Z[e]);
}

// db[j] = Σ_i dZ[i, j] (fixed order: one thread per column, strided rows)
__global__ void colsum_kernel(int rows, int cols, const float* __restrict__ dZ, float* __restrict__ db) {
    __shared__ float part[256];
    const int j = blockIdx.x;
    float s = 0.f;
    for (int i = threadIdx.x; i < rows; i += blockDim.x) s += dZ[(long)i * cols + j];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) db[j] = part[0];
}

// mean-squared error: dY = (out - y)/n, per-row squared error for the loss.  A CTA reads its rows in
// lines and a thread per row forms that row's sum, one chain, from shared memory: 7.8 µs for
// 1,024 x 64, where a thread per row of global memory (no two lanes on one line) took 42
constexpr int kMseRows = 16;
constexpr int kMseCols = 64;
__global__ void __launch_bounds__(128) mse_kernel(int n, int k, const float* __restrict__ out,
                                                  const float* __restrict__ y, float* __restrict__ dY,
                                                  float* __restrict__ row_loss) {
    after_previous();
    __shared__ float s_d[kMseRows][kMseCols + 1];
    const long r0 = (long)blockIdx.x * kMseRows;
    const int rows = n - r0 < kMseRows ? (int)(n - r0) : kMseRows, tid = threadIdx.x;
    float s = 0.f;
    for (int c = 0; c < k; c += kMseCols) {
        const int cols = min(kMseCols, k - c);
#pragma unroll
        for (int e = tid; e < kMseRows * kMseCols; e += 128) {
            const int r = e / kMseCols, j = e % kMseCols;
            if (r >= rows || j >= cols) continue;
            const long at = (r0 + r) * k + c + j;
            const float d = out[at] - y[at];
            dY[at] = d / (float)n;
            s_d[r][j] = d;
        }
        __syncthreads();
        if (tid < rows)
            for (int j = 0; j < cols; ++j) s = fmaf(s_d[tid][j], s_d[tid][j], s);
        __syncthreads();
    }
    if (tid < rows && row_loss) row_loss[r0 + tid] = 0.5f * s;
}

// Adam with bias correction (Kingma & Ba 2015); refreshes the BF16 weight copy
__global__ void adam_kernel(long count, float* __restrict__ p, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                            float eps, float c1, float c2, __nv_bfloat16* __restrict__ pbf) {
    after_previous();
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= count) return;
    const float gi = g[e];
    const float mi = b1 * m[e] + (1.f - b1) * gi;
    const float vi = b2 * v[e] + (1.f - b2) * gi * gi;
    m[e] = mi;
    v[e] = vi;
    const float w = p[e] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[e] = w;
    if (pbf) pbf[e] = __float2bfloat16_rn(w);
}

__global__ void to_bf16_kernel(long count, const float* __restrict__ p, __nv_bfloat16* __restrict__ q) {
    long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < count) q[e] = __float2bfloat16_rn(p[e]);
}

// llk_s = norm - ½ (q0 - 2 hᵀ c̃ + c̃ᵀ G c̃), c̃ = scale ⊙ c.  A CTA takes 16 PER chains; a thread
// forms kSurRows rows of G c̃ for PER chains, eight of them so that four 16-byte shared-memory loads feed 64 FMAs
// (shared-memory wavefronts bound it otherwise: with eight FMAs per three loads 34 µs for 32,768
// chains and 64 coefficients).  Its FP32 terms are added exactly in float-float and the threads
// of a chain in order (FP64 products and sums in a warp per chain took 61 µs at the FP64
// pipe's rate).  Measured: 24 µs; staging the operands by 4-byte loads, 58 µs.
constexpr int kSurMaxK = 96;
constexpr int kSurLanes = 16;                // threads over the chains of a CTA
__host__ __device__ constexpr int sur_stride(int chains) { return chains + 4; }   // row of c̃: 16-byte aligned, spread over the banks
constexpr int kSurRows = 8;
// chains per SM up to which a thread takes two of them (a fourth of the work in the chain of FMAs, four
// times the CTAs): 1,000 x 64 7.4 µs against 13.4 with eight (10.4 with a warp per chain), 9,728 x 8
// 7.0 against 10.4 (12.4), 9,728 x 64 8.8 against 13.9, 9,728 x 96 15.8 against 20.5; but 12,000 x 96
// 28.2 against 21.2
constexpr int kSurFew = 64;
static int sur_groups(int k) { return (k + kSurRows - 1) / kSurRows; }
static size_t sur_smem(int k, int chains) {
    return ((size_t)k * kSurRows * sur_groups(k) + (size_t)k * sur_stride(chains) + 2 * (size_t)sur_groups(k) * chains) *
           sizeof(float);
}

template <int PER>
__global__ void __launch_bounds__(kSurLanes * (kSurMaxK / kSurRows))
surrogate_llk_kernel(int n, int k, const float* __restrict__ coeff, const float* __restrict__ scale,
                     const float* __restrict__ G, const float* __restrict__ h, double q0, double norm,
                     double* __restrict__ llk) {
    after_previous();
    extern __shared__ __align__(16) float s_mem[];
    constexpr int kChains = kSurLanes * PER, kStride = sur_stride(kChains);
    const int groups = (k + kSurRows - 1) / kSurRows, rows = groups * kSurRows;
    float* sGT = s_mem;                                  // [k][rows], sGT[b][a] = G[a][b]
    float* sc = sGT + k * rows;                          // [k][kStride]
    float2* s_part = reinterpret_cast<float2*>(sc + k * kStride);     // [groups][kChains]
    const int tid = threadIdx.x, threads = kSurLanes * groups;
    const int c0 = tid % kSurLanes * PER, a0 = tid / kSurLanes * kSurRows;
    const long i0 = (long)blockIdx.x * kChains;
    const int chains = n - i0 < kChains ? (int)(n - i0) : kChains;
    // staged by 16-byte loads, eight in flight per thread, where the rows allow
    if (k % 4 == 0 && ((size_t)G | (size_t)coeff | (size_t)scale) % 16 == 0) {
        const int kq = k / 4;
#pragma unroll 8
        for (int e = tid; e < k * kq; e += threads) {
            const int a = e / kq, b = 4 * (e - a * kq);
            const float4 v = __ldg(reinterpret_cast<const float4*>(G) + e);
            float* to = sGT + b * rows + a;
            to[0] = v.x; to[rows] = v.y; to[2 * rows] = v.z; to[3 * rows] = v.w;
        }
#pragma unroll 8
        for (int e = tid; e < chains * kq; e += threads) {
            const int q = e / kq, b = 4 * (e - q * kq);
            const float4 v = __ldg(reinterpret_cast<const float4*>(coeff + i0 * k) + e);
            const float4 f = __ldg(reinterpret_cast<const float4*>(scale + b));
            float* to = sc + b * kStride + q;
            to[0] = v.x * f.x; to[kStride] = v.y * f.y; to[2 * kStride] = v.z * f.z; to[3 * kStride] = v.w * f.w;
        }
    } else {
        for (int e = tid; e < k * k; e += threads) {
            const int a = e / k, b = e - a * k;
            sGT[b * rows + a] = __ldg(G + e);
        }
        for (int e = tid; e < chains * k; e += threads) {
            const int q = e / k, b = e - q * k;
            sc[b * kStride + q] = __ldg(coeff + i0 * k + e) * __ldg(scale + b);
        }
    }
    // rows past k and chains past n: zeros
    for (int e = tid; e < (rows - k) * k; e += threads) sGT[e / (rows - k) * rows + k + e % (rows - k)] = 0.f;
    for (int e = tid; e < (kChains - chains) * k; e += threads)
        sc[e % k * kStride + chains + e / k] = 0.f;
    __syncthreads();
    float row[kSurRows][PER] = {};
#pragma unroll 2
    for (int b = 0; b < k; ++b) {
        float g[kSurRows], v[PER];
        *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(sGT + b * rows + a0);
        *reinterpret_cast<float4*>(g + 4) = *reinterpret_cast<const float4*>(sGT + b * rows + a0 + 4);
        if constexpr (PER == 8) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(sc + b * kStride + c0);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(sc + b * kStride + c0 + 4);
        } else {
            *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(sc + b * kStride + c0);
        }
#pragma unroll
        for (int q = 0; q < kSurRows; ++q)
#pragma unroll
            for (int c = 0; c < PER; ++c) row[q][c] = fmaf(g[q], v[c], row[q][c]);
    }
    ff acc[PER] = {};
#pragma unroll
    for (int q = 0; q < kSurRows; ++q) {
        if (a0 + q < k) {
            const float h2 = -2.0f * __ldg(h + a0 + q);
#pragma unroll
            for (int c = 0; c < PER; ++c) {
                const float ca = sc[(a0 + q) * kStride + c0 + c];
                float t = ca * row[q][c];
                ff_add(acc[c], t, fmaf(ca, row[q][c], -t));
                t = h2 * ca;
                ff_add(acc[c], t, fmaf(h2, ca, -t));
            }
        }
    }
#pragma unroll
    for (int c = 0; c < PER; ++c) s_part[a0 / kSurRows * kChains + c0 + c] = make_float2(acc[c].hi, acc[c].lo);
    __syncthreads();
    for (int c = tid; c < chains; c += threads) {
        ff t{0.f, 0.f};
        for (int g = 0; g < groups; ++g) {
            const float2 p = s_part[g * kChains + c];
            ff_add(t, p.x, p.y);
        }
        double acc = ff_to_double(t);
        if (!isfinite(acc)) {
            // a product or the sum left FP32's range (a NaN would be accepted as a sample): in FP64
            acc = 0.0;
            for (int a = 0; a < k; ++a) {
                float z = 0.f;
                for (int b = 0; b < k; ++b) z = fmaf(sGT[b * rows + a], sc[b * kStride + c], z);
                const double ca = (double)sc[a * kStride + c];
                acc += ca * (double)z - 2.0 * (double)h[a] * ca;
            }
        }
        llk[i0 + c] = norm - 0.5 * (q0 + acc);
    }
}

// Stage 1 of delayed acceptance: surrogate Metropolis test and compaction of survivors
__global__ void da_screen_kernel(int n, const double* __restrict__ beta, uint64_t seed, uint32_t step,
                                 const uint32_t* __restrict__ epoch, const uint32_t* __restrict__ mask,
                                 const double* __restrict__ cprior, const double* __restrict__ csur,
                                 const double* __restrict__ prior, const double* __restrict__ sur,
                                 int32_t* __restrict__ pass, int32_t* __restrict__ index,
                                 int32_t* __restrict__ count) {
    after_previous();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int ok = 0;
    if (!mask[i]) {
        const double b = *beta;
        const double d1 = (cprior[i] + b * csur[i]) - (prior[i] + b * sur[i]);
        u32x4 r = draw(seed, (uint32_t)i, 1u, STREAM_ACCEPT, step, *epoch);
        ok = log(u01_open_closed(r.x, r.y)) <= d1;
    }
    pass[i] = ok;
    if (ok) index[atomicAdd(count, 1)] = i;
}

// Stage 2: exact correction for the survivors; counters: accepted, rejected (support), unlikely
__global__ void da_accept_kernel(int n, int p, const double* __restrict__ beta, uint64_t seed,
                                 uint32_t step, const uint32_t* __restrict__ epoch,
                                 const uint32_t* __restrict__ mask, const int32_t* __restrict__ pass,
                                 const double* __restrict__ cand, const double* __restrict__ cprior,
                                 const double* __restrict__ cdata, const double* __restrict__ csur,
                                 double* __restrict__ theta, double* __restrict__ prior,
                                 double* __restrict__ data, double* __restrict__ post,
                                 double* __restrict__ sur, unsigned long long* __restrict__ counters,
                                 unsigned long long* __restrict__ screened) {
    after_previous();
    __shared__ unsigned int s_cnt[4];
    if (threadIdx.x < 4) s_cnt[threadIdx.x] = 0u;
    __syncthreads();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        if (mask[i]) {
            atomicAdd(&s_cnt[1], 1u);
        } else if (!pass[i]) {
            atomicAdd(&s_cnt[2], 1u);
        } else {
            atomicAdd(&s_cnt[3], 1u);
            const double b = *beta;
            const double cp = cprior[i] + b * cdata[i];
            const double dsur = (cprior[i] + b * csur[i]) - (prior[i] + b * sur[i]);
            u32x4 r = draw(seed, (uint32_t)i, 2u, STREAM_ACCEPT, step, *epoch);
            if (log(u01_open_closed(r.x, r.y)) > (cp - post[i]) - dsur) {
                atomicAdd(&s_cnt[2], 1u);
            } else {
                atomicAdd(&s_cnt[0], 1u);
                for (int j = 0; j < p; ++j) theta[(size_t)i * p + j] = cand[(size_t)i * p + j];
                prior[i] = cprior[i];
                data[i] = cdata[i];
                post[i] = cp;
                sur[i] = csur[i];
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_cnt[threadIdx.x])
        atomicAdd(&counters[threadIdx.x], (unsigned long long)s_cnt[threadIdx.x]);
    if (threadIdx.x == 3 && s_cnt[3] && screened) atomicAdd(screened, (unsigned long long)s_cnt[3]);
}

// The exact log-likelihood below which the stage-2 test of da_accept_kernel certainly
// rejects chain i (early rejection of the exact correction): the test rejects when
// log u > (cprior + β cdata − post) − dsur, so below (log u + post − cprior + dsur)/β, lowered
// by a relative 1e-9 for the rounding of the test; -inf where no evaluation is made.
__global__ void da_floor_kernel(int n, const double* __restrict__ beta, uint64_t seed, uint32_t step,
                                const uint32_t* __restrict__ epoch, const uint32_t* __restrict__ mask,
                                const int32_t* __restrict__ pass, const double* __restrict__ cprior,
                                const double* __restrict__ csur, const double* __restrict__ prior,
                                const double* __restrict__ sur, const double* __restrict__ post,
                                double* __restrict__ floor) {
    after_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double b = *beta;
    double f = -INFINITY;
    if (!mask[i] && pass[i] && b > 0.0) {
        const double dsur = (cprior[i] + b * csur[i]) - (prior[i] + b * sur[i]);
        u32x4 r = draw(seed, (uint32_t)i, 2u, STREAM_ACCEPT, step, *epoch);
        f = (log(u01_open_closed(r.x, r.y)) + post[i] - cprior[i] + dsur) / b;
        f -= (fabs(f) + 1.0) * 1e-9;
        if (!(f == f)) f = -INFINITY;
    }
    floor[i] = f;
}

// chains whose surrogate-chain state moved away from the exact state go to the exact
// correction: pass[i] = (θ_s ≠ θ) and no support violation, compacted into index
__global__ void da_moved_kernel(int n, int p, const double* __restrict__ theta,
                                const double* __restrict__ theta_s, int32_t* __restrict__ pass,
                                int32_t* __restrict__ index, int32_t* __restrict__ count) {
    after_previous();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int moved = 0;
    for (int j = 0; j < p; ++j) moved |= (theta[(size_t)i * p + j] != theta_s[(size_t)i * p + j]);
    pass[i] = moved;
    if (moved) index[atomicAdd(count, 1)] = i;
}

}  // namespace ag

// ---------------------------------------------------------------------------
// C ABI
using namespace ag;

static inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

extern "C" int ag_da_moved(int32_t n, int32_t p, const double* theta, const double* theta_s, int32_t* pass,
                           int32_t* index, int32_t* count, void* stream) {
    AG_REQUIRE(n > 0 && p > 0 && theta && theta_s && pass && index && count, "invalid arguments");
    cudaStream_t s = as_stream(stream);
    int rc = cuda_status(cudaMemsetAsync(count, 0, sizeof(int32_t), s), "memset count");
    if (rc) return rc;
    launch_after(da_moved_kernel, nblk(n, 256), 256, 0, s, n, p, theta, theta_s, pass, index, count);
    return launch_status("da_moved_kernel");
}

static int check_net(const ag_mlp* net) {
    AG_REQUIRE(net && net->nlayers >= 1 && net->nlayers <= kMaxLayers, "invalid network");
    for (int l = 0; l <= net->nlayers; ++l) AG_REQUIRE(net->sizes[l] > 0, "layer size must be positive");
    return AG_OK;
}

extern "C" int64_t ag_mlp_param_count(const ag_mlp* net) {
    if (check_net(net)) return -1;
    int64_t c = 0;
    for (int l = 0; l < net->nlayers; ++l) c += (int64_t)net->sizes[l + 1] * net->sizes[l] + net->sizes[l + 1];
    return c;
}

// parameter layout: for each layer W (out x in) then b (out)
static void offsets(const ag_mlp* net, int64_t* w, int64_t* b) {
    int64_t c = 0;
    for (int l = 0; l < net->nlayers; ++l) {
        w[l] = c;
        c += (int64_t)net->sizes[l + 1] * net->sizes[l];
        b[l] = c;
        c += net->sizes[l + 1];
    }
}

extern "C" int64_t ag_mlp_activation_floats(const ag_mlp* net, int32_t n) {
    if (check_net(net) || n <= 0) return -1;
    int64_t c = 0;
    for (int l = 1; l <= net->nlayers; ++l) c += 2 * (int64_t)n * net->sizes[l];   // Z and Y per layer
    return c;
}

// the shares of K (product_split) on a cluster of up to 8 CTAs
static int gemm(cudaStream_t s, int M, int N, int K, const float* A, long sam, long sak, const void* B,
                bool bbf16, long sbk, long sbn, float* C, long ldc, const float* bias, int epi, float* Z) {
    const int split = product_split(M, N, K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblk(N, BN), nblk(M, BM), split);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = split;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = bbf16 ? cudaLaunchKernelEx(&cfg, gemm_kernel<true>, M, N, K, A, sam, sak, B, sbk, sbn, C, ldc,
                                               bias, epi, Z)
                          : cudaLaunchKernelEx(&cfg, gemm_kernel<false>, M, N, K, A, sam, sak, B, sbk, sbn, C, ldc,
                                               bias, epi, Z);
    int rc = cuda_status(e, "cudaLaunchKernelEx(gemm_kernel)");
    if (rc) return rc;
    return launch_status("gemm_kernel");
}

// whether the row-wise kernels take n rows of a network: a layer's outputs fit a CTA's threads with all
// their shares of K, and the weights can be read in words of eight (four behind layer 0's odd size)
static bool rows_net(const ag_mlp* net, int n, const void* wbf16) {
    if (!aligned(wbf16, 16)) return false;
    for (int l = 0; l <= net->nlayers; ++l)
        if (net->sizes[l] > kRowWidth || (l > 0 && net->sizes[l] % 8)) return false;
    for (int l = 0; l < net->nlayers; ++l) {
        if (!net_split(n, net->sizes[l + 1], net->sizes[l]).row_groups) return false;
        if (l > 0 && !net_split(n, net->sizes[l], net->sizes[l + 1]).row_groups) return false;
    }
    return true;
}

extern "C" int ag_normalize_inputs(const double* theta, int32_t n, int32_t p, const double* lo,
                                   const double* hi, float* x, void* stream) {
    AG_REQUIRE(theta && lo && hi && x && n > 0 && p > 0, "invalid arguments");
    launch_after(normalize_kernel, nblk((long)nblk(n, kNormRows) * p, 128), 128, 0, as_stream(stream), theta, n, p,
                 lo, hi, x);
    return launch_status("normalize_kernel");
}

extern "C" int ag_mlp_forward(const ag_mlp* net, const float* params, const uint16_t* wbf16,
                              const float* x, int32_t n, float* out, float* acts, void* stream) {
    int rc = check_net(net);
    if (rc) return rc;
    AG_REQUIRE(params && wbf16 && x && out && acts && n > 0, "invalid arguments");
    cudaStream_t s = as_stream(stream);
    int64_t wo[kMaxLayers], bo[kMaxLayers];
    offsets(net, wo, bo);
    if (n <= kNetMost && rows_net(net, n, wbf16)) {
        NetLayers L;
        L.nlayers = net->nlayers;
        for (int l = 0; l < net->nlayers; ++l) {
            L.sizes[l] = net->sizes[l];
            L.w[l] = wo[l];
            L.b[l] = bo[l];
        }
        L.sizes[net->nlayers] = net->sizes[net->nlayers];
        rc = cuda_status(cudaFuncSetAttribute(net_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kNetSmem),
                         "cudaFuncSetAttribute(net_forward_kernel)");
        if (rc) return rc;
        launch_after(net_forward_kernel, nblk(n, kNetRows), kNetThreads, kNetSmem, s, L, params,
                     reinterpret_cast<const __nv_bfloat16*>(wbf16), x, n, out, acts);
        return launch_status("net_forward_kernel");
    }
    const float* in = x;
    float* a = acts;
    for (int l = 0; l < net->nlayers; ++l) {
        const int fi = net->sizes[l], fo = net->sizes[l + 1];
        const bool last = (l == net->nlayers - 1);
        float* Z = a;
        float* Y = last ? out : a + (int64_t)n * fo;
        rc = gemm(s, n, fo, fi, in, fi, 1, wbf16 + wo[l], true, 1, fi, Y, fo, params + bo[l],
                  last ? EPI_BIAS : EPI_BIAS_GELU, Z);
        if (rc) return rc;
        in = Y;
        a += 2 * (int64_t)n * fo;
    }
    return AG_OK;
}

// ---- tensor-core forward (inference)
static int mlp_kp(int f) { return (f + 63) / 64 * 64; }

static int check_net_tc(const ag_mlp* net) {
    int rc = check_net(net);
    if (rc) return rc;
    for (int l = 1; l <= net->nlayers; ++l)
        AG_REQUIRE(net->sizes[l] % 64 == 0, "the tensor-core layers need widths that are multiples of 64 "
                                            "(layer %d has %d)", l, net->sizes[l]);
    return AG_OK;
}

extern "C" size_t ag_mlp_tc_pack_bytes(const ag_mlp* net) {
    if (check_net_tc(net)) return 0;
    size_t c = 0;
    for (int l = 0; l < net->nlayers; ++l) c += (size_t)net->sizes[l + 1] * 2 * mlp_kp(net->sizes[l]) * 2;
    return c;
}

extern "C" int ag_mlp_tc_pack(const ag_mlp* net, const uint16_t* wbf16, uint16_t* wpack, void* stream) {
    int rc = check_net_tc(net);
    if (rc) return rc;
    AG_REQUIRE(wbf16 && wpack && aligned(wpack, 256), "invalid arguments (wpack must be 256-byte aligned)");
    cudaStream_t s = as_stream(stream);
    int64_t wo[kMaxLayers], bo[kMaxLayers];
    offsets(net, wo, bo);
    size_t off = 0;
    for (int l = 0; l < net->nlayers; ++l) {
        const int fi = net->sizes[l], fo = net->sizes[l + 1], kp = mlp_kp(fi);
        pack_weights_kernel<<<nblk((long)fo * kp, 256), 256, 0, s>>>(
            reinterpret_cast<const __nv_bfloat16*>(wbf16) + wo[l], fo, fi, kp,
            reinterpret_cast<__nv_bfloat16*>(wpack) + off);
        rc = launch_status("pack_weights_kernel");
        if (rc) return rc;
        off += (size_t)fo * 2 * kp;
    }
    return AG_OK;
}

extern "C" size_t ag_mlp_tc_workspace_bytes(const ag_mlp* net, int32_t n) {
    if (check_net_tc(net) || n <= 0) return 0;
    int kmax = 0;
    for (int l = 0; l < net->nlayers; ++l) kmax = max(kmax, mlp_kp(net->sizes[l]));
    const size_t one = ((size_t)n * 2 * kmax * 2 + 255) / 256 * 256;
    return 2 * one;
}

static int mlp_layer_launch(cudaStream_t s, const __nv_bfloat16* xs, int n, int kp, const __nv_bfloat16* w,
                            int fo, const float* bias, int gelu_on, float* Z, float* Y, __nv_bfloat16* xnext,
                            int kp_next, uint32_t* flags) {
    CUtensorMap mx, mw;
    int rc = make_map(&mx, xs, n, 2 * kp, TC_BM);
    if (rc) return rc;
    rc = make_map(&mw, w, fo, 2 * kp, kMlpCols);
    if (rc) return rc;
    rc = cuda_status(cudaFuncSetAttribute(mlp_layer_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kMlpSmem),
                     "cudaFuncSetAttribute(mlp_layer_tc_kernel)");
    if (rc) return rc;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    // as many CTAs per block of columns as there are places for, or tiles
    const int mtiles = (n + TC_BM - 1) / TC_BM, ntiles = fo / kMlpCols;
    const int places = kMlpCtas * sms / ntiles, per_block = places < 1 ? 1 : places < mtiles ? places : mtiles;
    launch_after(mlp_layer_tc_kernel, ntiles * per_block, kMlpThreads, kMlpSmem, s, mx, mw, n, fo,
                 2 * kp / TC_BK, mtiles, ntiles, bias, gelu_on, Z, Y, xnext, kp_next, flags);
    return launch_status("mlp_layer_tc_kernel");
}

extern "C" int ag_mlp_forward_tc(const ag_mlp* net, const float* params, const uint16_t* wpack, const float* x,
                                 int32_t n, float* out, float* acts, void* workspace, size_t workspace_bytes,
                                 uint32_t* flags, void* stream) {
    int rc = check_net_tc(net);
    if (rc) return rc;
    AG_REQUIRE(params && wpack && x && out && flags && n > 0, "invalid arguments");
    AG_REQUIRE(aligned(out, 16) && (acts == nullptr || aligned(acts, 16)) && aligned(wpack, 256),
               "out and acts must be 16-byte aligned, wpack 256-byte aligned");
    const size_t need = ag_mlp_tc_workspace_bytes(net, n);
    AG_REQUIRE(workspace && workspace_bytes >= need && aligned(workspace, 256),
               "the tensor-core forward needs %zu bytes of 256-byte aligned workspace", need);
    cudaStream_t s = as_stream(stream);
    int64_t wo[kMaxLayers], bo[kMaxLayers];
    offsets(net, wo, bo);
    __nv_bfloat16* buf[2] = {reinterpret_cast<__nv_bfloat16*>(workspace),
                             reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(workspace) + need / 2)};
    const int fi0 = net->sizes[0], kp0 = mlp_kp(fi0);
    // also what keeps the first layer's early read of wpack behind the packing: it may start once this kernel,
    // which waits for everything before it, has
    launch_after(split_rows_kernel, nblk((long)n * (kp0 / 8), 256), 256, 0, s, x, n, fi0, kp0, buf[0]);
    rc = launch_status("split_rows_kernel");
    if (rc) return rc;
    const __nv_bfloat16* w = reinterpret_cast<const __nv_bfloat16*>(wpack);
    float* a = acts;
    for (int l = 0; l < net->nlayers; ++l) {
        const int fi = net->sizes[l], fo = net->sizes[l + 1], kp = mlp_kp(fi);
        const bool last = (l == net->nlayers - 1);
        float* Z = (a && !last) ? a : nullptr;
        float* Y = last ? out : (a ? a + (int64_t)n * fo : nullptr);
        __nv_bfloat16* xnext = last ? nullptr : buf[(l + 1) & 1];
        const int kp_next = last ? 0 : mlp_kp(fo);
        rc = mlp_layer_launch(s, buf[l & 1], n, kp, w, fo, params + bo[l], last ? 0 : 1, Z, Y, xnext, kp_next, flags);
        if (rc) return rc;
        w += (size_t)fo * 2 * kp;
        if (a) a += 2 * (int64_t)n * fo;
    }
    return AG_OK;
}

extern "C" int ag_mlp_backward(const ag_mlp* net, const float* params, const uint16_t* wbf16,
                               const float* x, int32_t n, const float* acts, float* dout, float* grads,
                               float* scratch, void* stream) {
    int rc = check_net(net);
    if (rc) return rc;
    AG_REQUIRE(params && wbf16 && x && acts && dout && grads && scratch && n > 0, "invalid arguments");
    cudaStream_t s = as_stream(stream);
    int64_t wo[kMaxLayers], bo[kMaxLayers], ao[kMaxLayers];
    offsets(net, wo, bo);
    int64_t c = 0;
    int maxw = 0;
    for (int l = 0; l < net->nlayers; ++l) {
        ao[l] = c;
        c += 2 * (int64_t)n * net->sizes[l + 1];
        maxw = max(maxw, net->sizes[l + 1]);
        maxw = max(maxw, net->sizes[l]);
    }
    // dY of the current layer lives in dout (last layer) or in scratch (n x maxw, ping-pong)
    float* cur = dout;
    float* bufs[2] = {scratch, scratch + (int64_t)n * maxw};
    const bool by_rows = rows_net(net, n, wbf16);
    if (by_rows) {
        rc = cuda_status(cudaFuncSetAttribute(net_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)kBackSmem),
                         "cudaFuncSetAttribute(net_backward_kernel)");
        if (rc) return rc;
    }
    for (int l = net->nlayers - 1; l >= 0; --l) {
        const int fi = net->sizes[l], fo = net->sizes[l + 1];
        const bool last = (l == net->nlayers - 1);
        if (by_rows) {
            // cur holds this layer's dZ
            const float* hin = (l == 0) ? x : acts + ao[l - 1] + (int64_t)n * fi;
            const int row_ctas = l > 0 ? nblk(nblk(n, kNetRows), kBackSplit) * kBackSplit : 0;
            const int sum_ctas = nblk(fo, 8 * kBackSplit) * kBackSplit;
            const int htiles = nblk(fi, kBackTile), tiles = nblk(fo, kBackTile) * htiles;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(row_ctas + sum_ctas + tiles * kBackSplit);
            cfg.blockDim = dim3(kNetThreads);
            cfg.dynamicSmemBytes = kBackSmem;
            cfg.stream = s;
            cudaLaunchAttribute attr[2];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = kBackSplit;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[1].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 2;
            float* nxt = bufs[l & 1];
            rc = cuda_status(cudaLaunchKernelEx(&cfg, net_backward_kernel, n, fi, fo, (const float*)cur,
                                                reinterpret_cast<const __nv_bfloat16*>(wbf16) + wo[l],
                                                l > 0 ? acts + ao[l - 1] : nullptr, nxt, row_ctas, sum_ctas, hin, htiles,
                                                grads + wo[l], grads + bo[l]),
                             "cudaLaunchKernelEx(net_backward_kernel)");
            if (rc) return rc;
            cur = nxt;
            continue;
        }
        if (!last) {
            gelu_back_kernel<<<nblk((long)n * fo, 256), 256, 0, s>>>((long)n * fo, acts + ao[l], cur);
            rc = launch_status("gelu_back_kernel");
            if (rc) return rc;
        }
        const float* hin = (l == 0) ? x : acts + ao[l - 1] + (int64_t)n * fi;   // Y of layer l-1
        // dW (fo x fi) = dZᵀ (fo x n) · h (n x fi)
        rc = gemm(s, fo, fi, n, cur, 1, fo, hin, false, fi, 1, grads + wo[l], fi, nullptr, EPI_NONE, nullptr);
        if (rc) return rc;
        colsum_kernel<<<fo, 256, 0, s>>>(n, fo, cur, grads + bo[l]);
        rc = launch_status("colsum_kernel");
        if (rc) return rc;
        if (l > 0) {
            float* nxt = bufs[l & 1];
            // dX (n x fi) = dZ (n x fo) · W (fo x fi)
            rc = gemm(s, n, fi, fo, cur, fo, 1, wbf16 + wo[l], true, fi, 1, nxt, fi, nullptr, EPI_NONE, nullptr);
            if (rc) return rc;
            cur = nxt;
        }
    }
    return AG_OK;
}

extern "C" int ag_mse_grad(int32_t n, int32_t k, const float* out, const float* target, float* dout,
                           float* row_loss, void* stream) {
    AG_REQUIRE(n > 0 && k > 0 && out && target && dout, "invalid arguments");
    launch_after(mse_kernel, nblk(n, kMseRows), 128, 0, as_stream(stream), n, k, out, target, dout, row_loss);
    return launch_status("mse_kernel");
}

extern "C" int ag_adam_step(int64_t count, float* params, const float* grads, float* m, float* v,
                            int32_t t, float lr, float b1, float b2, float eps, uint16_t* wbf16,
                            void* stream) {
    AG_REQUIRE(count > 0 && params && grads && m && v && t >= 1, "invalid arguments");
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    launch_after(adam_kernel, nblk(count, 256), 256, 0, as_stream(stream), count, params, grads, m, v, lr, b1, b2,
                 eps, c1, c2, reinterpret_cast<__nv_bfloat16*>(wbf16));
    return launch_status("adam_kernel");
}

extern "C" int ag_to_bf16(int64_t count, const float* src, uint16_t* dst, void* stream) {
    AG_REQUIRE(count > 0 && src && dst, "invalid arguments");
    to_bf16_kernel<<<nblk(count, 256), 256, 0, as_stream(stream)>>>(count, src,
                                                                     reinterpret_cast<__nv_bfloat16*>(dst));
    return launch_status("to_bf16_kernel");
}

extern "C" int ag_surrogate_llk(int32_t n, int32_t k, const float* coeff, const float* scale,
                                const float* gram, const float* h, double q0, double norm, double* llk,
                                void* stream) {
    AG_REQUIRE(n > 0 && k > 0 && coeff && scale && gram && h && llk, "invalid arguments");
    AG_REQUIRE(k <= kSurMaxK, "at most %d surrogate coefficients are supported (got %d)", kSurMaxK, k);
    int sms = 0;
    int rc = sm_count(&sms);
    if (rc) return rc;
    const bool few = n <= kSurFew * sms;
    const int chains = kSurLanes * (few ? 2 : 8);
    const auto kernel = few ? surrogate_llk_kernel<2> : surrogate_llk_kernel<8>;
    const size_t smem = sur_smem(k, chains);
    if (smem > 48 * 1024) {
        rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                         "cudaFuncSetAttribute(surrogate_llk_kernel)");
        if (rc) return rc;
    }
    launch_after(kernel, nblk(n, chains), kSurLanes * sur_groups(k), smem, as_stream(stream), n, k, coeff, scale, gram,
                 h, q0, norm, llk);
    return launch_status("surrogate_llk_kernel");
}

extern "C" int ag_da_screen(const ag_stage_state* st, int32_t n, uint64_t seed, uint32_t step,
                            const uint32_t* mask, const double* cprior, const double* csur,
                            const double* prior, const double* sur, int32_t* pass, int32_t* index,
                            int32_t* count, void* stream) {
    AG_REQUIRE(st && n > 0 && mask && cprior && csur && prior && sur && pass && index && count,
               "invalid arguments");
    cudaStream_t s = as_stream(stream);
    int rc = cuda_status(cudaMemsetAsync(count, 0, sizeof(int32_t), s), "memset count");
    if (rc) return rc;
    launch_after(da_screen_kernel, nblk(n, 256), 256, 0, s, n,
                 st->beta, seed, step, st->epoch, mask, cprior, csur, prior, sur, pass, index, count);
    return launch_status("da_screen_kernel");
}

extern "C" int ag_da_floor(const ag_stage_state* st, int32_t n, uint64_t seed, uint32_t step, const uint32_t* mask,
                           const int32_t* pass, const double* cprior, const double* csur, const double* prior,
                           const double* sur, const double* post, double* llk_floor, void* stream) {
    AG_REQUIRE(st && n > 0 && mask && pass && cprior && csur && prior && sur && post && llk_floor,
               "invalid arguments");
    launch_after(da_floor_kernel, nblk(n, 256), 256, 0, as_stream(stream), n,
                 st->beta, seed, step, st->epoch, mask, pass, cprior, csur, prior, sur, post, llk_floor);
    return launch_status("da_floor_kernel");
}

extern "C" int ag_da_accept(const ag_stage_state* st, int32_t n, int32_t p, uint64_t seed, uint32_t step,
                            const uint32_t* mask, const int32_t* pass, const double* cand,
                            const double* cprior, const double* cdata, const double* csur, double* theta,
                            double* prior, double* data, double* post, double* sur,
                            unsigned long long* screened, void* stream) {
    AG_REQUIRE(st && n > 0 && p > 0 && mask && pass && cand && cprior && cdata && csur && theta && prior &&
                   data && post && sur,
               "invalid arguments");
    launch_after(da_accept_kernel, nblk(n, 256), 256, 0, as_stream(stream), n, p,
                 st->beta, seed, step, st->epoch, mask, pass, cand, cprior, cdata, csur, theta, prior, data, post, sur, st->counters, screened);
    return launch_status("da_accept_kernel");
}
