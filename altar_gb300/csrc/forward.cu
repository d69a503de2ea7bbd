// Fused batched forward models + diagonal-Cd misfit + per-chain log-likelihood.
//
// CDM (Compound Dislocation Model, Nikkhoo et al. 2016), following the
// reference numpy CDM models/cdm/cdm/libcdm.py:39-430, and the Mogi point
// source, following models/mogi/lib/libmogi/Source.cc:65-154.
//
// CDM evaluation strategy.  The reference sums, over the 12 sides of three
// rectangles, the difference v(B) - v(A) of two angular dislocations
// (libcdm.py:310-372).  Evaluated in FP32 as written, that difference loses
// up to ~4 digits: each term is O(1) while the side's contribution is
// O(side length / distance).  Here every quantity of the angular-dislocation
// formula is carried as a pair (value at A, difference B - A), with the
// difference propagated by exact identities (product rule
// Δ(uv) = Δu·v_B + u_A·Δv, Δ(1/u) = -Δu/(u_A u_B),
// Δr = Δ(r²)/(r_A + r_B), Δlog u = log1p(Δu/u_A), and the Burgers-function
// difference as a single atan2 of the rotation from A to B), so the
// cancellation never happens in floating point.
//
// Work decomposition: cdm_setup_kernel computes each chain's per-side
// constants and per-rectangle quadrature parameters in FP64 and lists the
// chains that have work (not masked, not above the free surface) in
// consecutive slots; the likelihood kernel runs one warp per slot (several for
// few chains, each over a share of the stations), lanes over
// stations; a CTA holds WARPS chains whose constants live in shared memory and
// are read with broadcast vector loads; station tiles stream through a ring of
// shared-memory buffers filled by 1-D bulk copies (cp.async.bulk + mbarrier)
// and shared by the CTA's warps.  For each tile a warp decides, from the
// tile's bounding box, which rectangles it integrates by quadrature and with
// how many nodes (generated into shared memory), and evaluates the sides of the
// others.  Each lane accumulates w·r² in float-float; the warp's sum is reduced
// in FP64 in a fixed order.
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "cdm_side.cuh"

namespace ag {

constexpr int kMaxOffsets = 16;      // datasets with their own offset parameter
constexpr int kTile = AG_STATION_TILE;
constexpr uint32_t kWaitLimit = 1u << 24;

// ---------------------------------------------------------------------------
// per-chain constants: stations are taken relative to the source centre (x0, y0)
struct __align__(16) ChainC {
    float4 hdr;                 // x0_hi, x0_lo, y0_hi, y0_lo
    uint32_t side_mask;         // active sides; 0 = chain inactive
    int32_t chain;              // row of θ, llk and the residuals
    uint32_t pad0, pad1;
    float off[kMaxOffsets];     // per-dataset offsets θ[offset_idx + k]
    float pad2[8];
    SideC side[kSides];
    RectQ rect[3];              // every rectangle that takes part, parametric quadrature
};
static_assert(sizeof(ChainC) % 16 == 0, "ChainC must be a whole number of float4");

// Set-up.  A block takes kSetupChains chains and gives every step to as many threads as it has
// parts: a thread per rotation (sine and cosine), per corner, per side and rectangle of the plan, per
// side and rectangle of the constants.  Each part is 50 to 150 dependent FP64 instructions at ~67
// cycles; one thread per chain took them one after another (159 µs for a set-up of 2,000
// chains, whatever their number, and the plan twice), sixteen lanes per chain with every lane
// repeating the corners issued twice the FP64 instructions.  Here lanes are full and nothing is
// repeated: 31 µs for 2,000 chains (210 µs), 23 µs for 256 (248 µs).
//
// Chain slots ordered by cost (ORDERED).  The chains of one CTA share its ring of station tiles, so a
// CTA advances at the pace of its most expensive chain; with rectangles integrated by
// quadrature, with node counts that depend on each tile's distance, the work of a chain
// ranges over several times its minimum.  The set-up counts the chains per cost bucket (the work
// of their plan averaged over a sample of the tiles); cdm_slot_kernel gives each chain the next
// slot of its bucket, buckets in decreasing cost, so the CTAs hold chains of similar cost and the
// expensive ones are scheduled first (which also shortens the tail of the launch for one-chain
// CTAs).  Few chains, whose stations are split over several CTAs, take slots as they come.
constexpr int kCostBuckets = 64;
constexpr int kCostBucketFlop = 96;      // FLOP per station per bucket
constexpr int kSetupChains = 8;
constexpr int kSetupThreads = 128;

struct SetupHdr {                        // in the workspace, cleared before each set-up
    int32_t nslots;
    int32_t pad[31];
    int32_t hist[kCostBuckets];          // chains per cost bucket
    int32_t fill[kCostBuckets];          // slots handed out per bucket
};

// All requested chains (n, or the first *count_in of index_in): the constants of each chain with
// work in row t of out, t its position among the requested; the status bit for one above the
// free surface.
template <bool ORDERED>
__global__ void __launch_bounds__(kSetupThreads)
cdm_setup_kernel(ag_layout L, const double* __restrict__ theta, int n, const uint32_t* __restrict__ mask_in,
                 uint32_t* __restrict__ chain_status, const int32_t* __restrict__ index_in,
                 const int32_t* __restrict__ count_in, int noffsets, const float4* __restrict__ tile_box, int ntiles,
                 ChainC* __restrict__ out, int8_t* __restrict__ key, int32_t* __restrict__ slot_row,
                 SetupHdr* __restrict__ hdr) {
    __shared__ ChainC s_chain[kSetupChains];
    __shared__ Vec3 s_V[kSetupChains][3][4], s_slip[kSetupChains][3];
    __shared__ double s_sc[kSetupChains][6];
    __shared__ int s_idx[kSetupChains], s_nq[kSetupChains][3];
    __shared__ uint32_t s_above[kSetupChains], s_bits[kSetupChains], s_flop[kSetupChains];
    const int tid = threadIdx.x, t0 = blockIdx.x * kSetupChains;
    const int requested = index_in ? min(n, *count_in) : n;
    if (t0 >= requested) return;
    if (tid < kSetupChains) {
        const int t = t0 + tid;
        int i = -1;
        if (t < requested) {
            i = index_in ? index_in[t] : t;
            if (mask_in && mask_in[i]) {
                i = -1;
                if (ORDERED) key[t] = -1;
            }
        }
        s_idx[tid] = i;
        s_above[tid] = 0u;
        s_bits[tid] = 0u;
        s_flop[tid] = 0u;
    }
    __syncthreads();
    if (tid < 3 * kSetupChains) {
        const int c = tid / 3, w = tid - 3 * c;
        if (s_idx[c] >= 0) {
            const double omega = theta[(size_t)s_idx[c] * L.nparams + L.omega_idx + w];
            sincospi(omega / 180.0, &s_sc[c][2 * w], &s_sc[c][2 * w + 1]);
        }
    }
    __syncthreads();
    // threads 0-95: a corner, then a side, of one chain; threads 96-119: a rectangle
    const bool on_side = tid < kSides * kSetupChains;
    const int c = on_side ? tid / kSides : min((tid - kSides * kSetupChains) / 3, kSetupChains - 1);
    const int e = on_side ? tid - kSides * c : 0;
    const int r = on_side ? e >> 2 : tid - kSides * kSetupChains - 3 * c;        // >= 3: no rectangle
    const double* th = theta + (size_t)(s_idx[c] < 0 ? 0 : s_idx[c]) * L.nparams;
    if (on_side && s_idx[c] >= 0) {
        const Vec3 p = cdm_corner(th, L, s_sc[c], r, e & 3);
        s_V[c][r][e & 3] = p;
        if (p.z > 0.0) atomicOr(&s_above[c], 1u);
    }
    __syncthreads();
    const bool live = s_idx[c] >= 0 && !s_above[c];
    const uint32_t use = live ? rects_used(th[L.axes_idx], th[L.axes_idx + 1], th[L.axes_idx + 2]) : 0u;
    if (tid < kSetupChains && s_idx[tid] >= 0 && s_above[tid]) {
        if (chain_status) chain_status[s_idx[tid]] |= CHAIN_ABOVE_SURFACE;
        if (ORDERED) key[t0 + tid] = -2;
    }
    // the plan (cdm_plan): far rectangles, sides that take part and near-vertical ones
    if (r < 3 && (use >> r & 1u)) {
        if (on_side) {
            bool act, steep;
            side_class(s_V[c][r][e & 3], s_V[c][r][(e + 1) & 3], act, steep);
            if (act) atomicOr(&s_bits[c], (1u << e) | (steep ? 1u << (kSides + e) : 0u));
        } else {
            int n1 = 0, n2 = 0;
            const bool far = far_rect(s_V[c][r], n1, n2);
            if (far) atomicOr(&s_bits[c], 1u << (24 + r));
            s_nq[c][r] = far ? n1 | (n2 << 8) : 0;
            Vec3 nrm = v_cross(v_sub(s_V[c][r][1], s_V[c][r][0]), v_sub(s_V[c][r][3], s_V[c][r][0]));
            nrm = v_scale(nrm, 1.0 / sqrt(v_dot(nrm, nrm)));
            s_slip[c][r] = v_scale(nrm, th[L.strength_idx]);
        }
    }
    __syncthreads();
    uint32_t mask = s_bits[c];
    for (int q = 0; q < 3; ++q) {
        if (mask >> (24 + q) & 1u) mask &= ~((0xFu << (4 * q)) | (0xFu << (kSides + 4 * q)));
        if ((mask >> (24 + q) & 1u) || (mask >> (4 * q) & 0xFu)) mask |= 1u << (27 + q);
    }
    ChainC& C = s_chain[c];
    const double x0 = th[L.x_idx], y0 = th[L.x_idx + 1];
    if (live && on_side && (mask >> e & 1u))
        fill_side(C.side[e], s_V[c][r][e & 3], s_V[c][r][(e + 1) & 3], s_slip[c][r], L.nu, x0, y0,
                  (mask >> (kSides + e)) & 1u);
    if (live && !on_side && r < 3 && (mask >> (27 + r) & 1u)) {
        int sf, su;
        rect_side_work(mask, r, sf, su);
        const int nq = s_nq[c][r];
        fill_rect(C.rect[r], s_V[c][r], th[L.strength_idx], L.nu, x0, y0, sf, nq & 255, nq >> 8);
    }
    if (tid >= kSetupThreads - kSetupChains) {
        const int k = tid - (kSetupThreads - kSetupChains), i = s_idx[k];
        if (i >= 0 && !s_above[k]) {
            const double* p = theta + (size_t)i * L.nparams;
            uint32_t m = s_bits[k];
            for (int q = 0; q < 3; ++q) {
                if (m >> (24 + q) & 1u) m &= ~((0xFu << (4 * q)) | (0xFu << (kSides + 4 * q)));
                if ((m >> (24 + q) & 1u) || (m >> (4 * q) & 0xFu)) m |= 1u << (27 + q);
            }
            ChainC& K = s_chain[k];
            split_hilo(p[L.x_idx], K.hdr.x, K.hdr.y);
            split_hilo(p[L.x_idx + 1], K.hdr.z, K.hdr.w);
            for (int o = 0; o < kMaxOffsets; ++o) K.off[o] = (o < noffsets) ? (float)p[L.offset_idx + o] : 0.f;
            K.side_mask = m | 0x80000000u;      // a chain with no active side still needs a llk
            K.chain = i;
        }
    }
    __syncthreads();
    if (ORDERED) {
        // work per station averaged over every stride-th station tile (tile boxes relative to the
        // source centre as the likelihood kernel forms them)
        const int stride = ntiles > 16 ? ntiles / 16 : 1;
        const int first = stride / 2, samples = first < ntiles ? (ntiles - 1 - first) / stride + 1 : 0;
        for (int k = tid; k < kSetupChains * samples; k += kSetupThreads) {
            const int q = k / samples;
            if (s_idx[q] < 0 || s_above[q]) continue;
            const ChainC& K = s_chain[q];
            const float4 tb = __ldg(tile_box + first + (k - q * samples) * stride);
            uint32_t fl, su;
            tile_work(K.rect, K.side_mask, __fsub_rn(__fsub_rn(tb.x, K.hdr.x), K.hdr.y),
                      __fsub_rn(__fsub_rn(tb.y, K.hdr.x), K.hdr.y), __fsub_rn(__fsub_rn(tb.z, K.hdr.z), K.hdr.w),
                      __fsub_rn(__fsub_rn(tb.w, K.hdr.z), K.hdr.w), fl, su);
            atomicAdd(&s_flop[q], fl);
        }
        __syncthreads();
        if (tid < kSetupChains && s_idx[tid] >= 0 && !s_above[tid]) {
            const int b = (int)(s_flop[tid] / (uint32_t)(samples * kCostBucketFlop));
            key[t0 + tid] = (int8_t)(b < kCostBuckets ? b : kCostBuckets - 1);
            atomicAdd(&hdr->hist[b < kCostBuckets ? b : kCostBuckets - 1], 1);
        }
    } else if (tid < kSetupChains && s_idx[tid] >= 0 && !s_above[tid]) {
        slot_row[atomicAdd(&hdr->nslots, 1)] = t0 + tid;
    }
    // the rows of chains with work, by 16-byte stores
    constexpr int nvec = sizeof(ChainC) / 16;
    for (int k = tid; k < kSetupChains * nvec; k += kSetupThreads) {
        const int q = k / nvec;
        if (s_idx[q] < 0 || s_above[q]) continue;
        reinterpret_cast<float4*>(out + t0)[k] = reinterpret_cast<const float4*>(s_chain)[k];
    }
}

// Every chain with work takes the next slot of its cost bucket (buckets in decreasing cost;
// the order inside a bucket is that of the atomic, which does not affect any chain's result), so
// the likelihood kernel's CTAs hold only chains with work.
__global__ void cdm_slot_kernel(int n, const int8_t* __restrict__ key, const int32_t* __restrict__ count_in,
                                int32_t* __restrict__ slot_row, SetupHdr* __restrict__ hdr) {
    __shared__ int s_start[kCostBuckets];
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int b = kCostBuckets - 1; b >= 0; --b) {
            s_start[b] = acc;
            acc += hdr->hist[b];
        }
        if (blockIdx.x == 0) hdr->nslots = acc;
    }
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (count_in ? min(n, *count_in) : n)) return;
    const int b = key[t];
    if (b >= 0) slot_row[s_start[b] + atomicAdd(&hdr->fill[b], 1)] = t;
}

__global__ void cdm_check_kernel(ag_layout L, const double* __restrict__ theta, int n,
                                 uint32_t* __restrict__ chain_status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Vec3 V[3][4];
    if (cdm_corners(theta + (size_t)i * L.nparams, L, V)) chain_status[i] |= CHAIN_ABOVE_SURFACE;
}

// FP32 operations the likelihood kernel executes for each chain over the m stations (its
// plan per station tile: sides and quadrature nodes); 0 for chains above the free surface,
// which it skips
__global__ void cdm_work_kernel(ag_layout L, const double* __restrict__ theta, int n,
                                const float4* __restrict__ tile_box, int m, double* __restrict__ flop,
                                double* __restrict__ sfu) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* th = theta + (size_t)i * L.nparams;
    Vec3 V[3][4];
    double f = 0.0, u = 0.0;
    if (!cdm_corners(th, L, V)) {
        const double x0 = th[L.x_idx], y0 = th[L.x_idx + 1];
        float x0h, x0l, y0h, y0l;
        split_hilo(x0, x0h, x0l);
        split_hilo(y0, y0h, y0l);
        RectQ rect[3];
        const uint32_t mask = cdm_rects(th, L, V, x0, y0, rect);
        const int ntiles = (m + kTile - 1) / kTile;
        for (int t = 0; t < ntiles; ++t) {
            const float4 tb = __ldg(tile_box + t);
            uint32_t fl, su;
            tile_work(rect, mask, __fsub_rn(__fsub_rn(tb.x, x0h), x0l), __fsub_rn(__fsub_rn(tb.y, x0h), x0l),
                      __fsub_rn(__fsub_rn(tb.z, y0h), y0l), __fsub_rn(__fsub_rn(tb.w, y0h), y0l), fl, su);
            const int cnt = min(kTile, m - t * kTile);
            f += (double)fl * cnt;
            u += (double)su * cnt;
        }
    }
    flop[i] = f;
    if (sfu) sfu[i] = u;
}

// Bounding box of each tile of AG_STATION_TILE stations (coordinates hi + lo), rounded
// outwards to FP32; padding stations (index >= m) are left out.  One warp per tile.
__global__ void station_boxes_kernel(const float4* __restrict__ xy, int m, int ntiles, float4* __restrict__ box) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= ntiles) return;
    double x0 = INFINITY, x1 = -INFINITY, y0 = INFINITY, y1 = -INFINITY;
    for (int j = t * kTile + lane; j < min(m, (t + 1) * kTile); j += 32) {
        const float4 a = xy[j];
        const double x = (double)a.x + (double)a.y, y = (double)a.z + (double)a.w;
        x0 = fmin(x0, x); x1 = fmax(x1, x);
        y0 = fmin(y0, y); y1 = fmax(y1, y);
    }
    for (int o = 16; o > 0; o >>= 1) {
        x0 = fmin(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        x1 = fmax(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y0 = fmin(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        y1 = fmax(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    }
    if (lane == 0) box[t] = make_float4(f32_down(x0), f32_up(x1), f32_down(y0), f32_up(y1));
}

// ---------------------------------------------------------------------------
// CDM likelihood.  One warp per compacted chain slot, lanes over stations.
// Station tiles stream through a ring of STAGES shared-memory buffers filled
// by 1-D bulk copies: each warp waits on the buffer's full barrier, works
// through the tile and counts itself done; the warp that finishes a tile last
// refills that buffer with the tile STAGES ahead.  No CTA-wide barrier is
// taken per tile, so warps drift apart by up to STAGES - 1 tiles instead of
// waiting for the slowest one at every tile.
//
// The misfit is summed in kParts fixed parts of the tiles: each lane adds its stations of a part
// in float-float, the warp adds the lanes in FP64, and the parts are added in order, so a chain's
// log-likelihood has the same bits whoever computes its parts.  SPLIT (one warp per CTA): the
// CTAs (slot, y) of one chain take consecutive parts each and the last to finish adds them up.
// One warp per chain leaves most of the GPU idle below ~1,800 chains (12 resident CTAs on 152
// SMs) and ends in a ragged last wave up to a few times that (figures at kSplitChains).
constexpr int kParts = 32;

__host__ __device__ constexpr int part_begin(int k, int ntiles) { return (int)((long)k * ntiles / kParts); }
// first tile of share y of splits: whole parts, or whole tiles where a part has at most one
__host__ __device__ constexpr int split_begin(int y, int splits, int ntiles) {
    return ntiles <= kParts ? y * ntiles / splits : part_begin(y * kParts / splits, ntiles);
}

template <int WARPS, int MINB, int SPL, int STAGES, bool SPLIT = false>
__global__ void __launch_bounds__(WARPS * 32, MINB)
cdm_llk_kernel(const ChainC* __restrict__ chains, const int32_t* __restrict__ slot_row,
               const int32_t* __restrict__ nslots_ptr, int n, const float4* __restrict__ xy,
               const float4* __restrict__ losd, const float* __restrict__ wt,
               const int32_t* __restrict__ oid, const float4* __restrict__ tile_box,
               const int32_t* __restrict__ order, int m, int m_padded, double norm,
               const double* __restrict__ llk_floor, double* __restrict__ llk, float* __restrict__ resid,
               uint32_t* __restrict__ flags, double* __restrict__ parts, int* __restrict__ done) {
    static_assert(!SPLIT || WARPS == 1, "the stations of a chain are split over CTAs of one warp");
    const int nslots = min(n, *nslots_ptr);
    if ((int)(blockIdx.x * WARPS) >= nslots) return;       // whole CTA past the active chains
    __shared__ ChainC s_chain[WARPS];
    __shared__ float4 s_xy[STAGES][kTile];
    __shared__ float4 s_ld[STAGES][kTile];
    __shared__ __align__(16) float s_w[STAGES][kTile];
    __shared__ __align__(16) int32_t s_oid[STAGES][kTile];
    __shared__ float4 s_box[STAGES];                  // each tile's bounding box, with the tile
    __shared__ __align__(8) uint64_t full[STAGES];
    __shared__ int s_done[STAGES];
    __shared__ int s_issued;
    // each warp's quadrature nodes: one buffer per rectangle (one shared by the three where
    // shared memory is short), regenerated only when a tile needs other node counts
    constexpr int kNodeBufs = WARPS <= 4 ? 3 : 1;
    // (several stations per lane: packed nodes)
    typedef typename std::conditional<(SPL > 1), PackedNode, float4>::type Node;
    __shared__ __align__(16) Node s_node[WARPS][kNodeBufs][kQuadBudget];
    __shared__ float s_gx[136], s_gw[136];             // Gauss-Legendre rules (FP32)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = blockIdx.x * WARPS + warp;
    const bool active = slot < nslots;
    const int ntiles = m_padded / kTile;
    const int tile0 = SPLIT ? split_begin(blockIdx.y, gridDim.y, ntiles) : 0;
    const int tile1 = SPLIT ? split_begin(blockIdx.y + 1, gridDim.y, ntiles) : ntiles;
    const bool with_oid = (oid != nullptr);
    const uint32_t tile_bytes = kTile * (16u + 16u + 4u) + (with_oid ? kTile * 4u : 0u) + 16u;

    for (int k = threadIdx.x; k < 136; k += blockDim.x) {
        s_gx[k] = kGaussXf[k];
        s_gw[k] = kGaussWf[k];
    }
    // this warp's chain constants
    if (active) {
        const float4* src = reinterpret_cast<const float4*>(chains + slot_row[slot]);
        float4* dst = reinterpret_cast<float4*>(&s_chain[warp]);
        constexpr int nvec = sizeof(ChainC) / 16;
        for (int k = lane; k < nvec; k += 32) dst[k] = src[k];
    }
    auto issue = [&](int t, int buf) {
        const size_t base = (size_t)t * kTile;
        mbar_arrive_expect_tx(&full[buf], tile_bytes);
        bulk_g2s(&s_xy[buf][0], xy + base, kTile * 16u, &full[buf]);
        bulk_g2s(&s_ld[buf][0], losd + base, kTile * 16u, &full[buf]);
        bulk_g2s(&s_w[buf][0], wt + base, kTile * 4u, &full[buf]);
        if (with_oid) bulk_g2s(&s_oid[buf][0], oid + base, kTile * 4u, &full[buf]);
        bulk_g2s(&s_box[buf], tile_box + t, 16u, &full[buf]);
    };
    if (threadIdx.x == 0) {
        for (int b = 0; b < STAGES; ++b) {
            mbar_init(&full[b], 1);
            s_done[b] = 0;
        }
        fence_mbar_init();
        const int first = tile1 - tile0 < STAGES ? tile1 - tile0 : STAGES;
        for (int t = 0; t < first; ++t) issue(tile0 + t, t);
        s_issued = first;
    }
    __syncthreads();
    const ChainC& C = s_chain[warp];
    const int chain = active ? C.chain : n;
    const uint32_t smask = active ? C.side_mask : 0u;
    const float x0h = C.hdr.x, x0l = C.hdr.y, y0h = C.hdr.z, y0l = C.hdr.w;
    ff acc{0.f, 0.f};
    bool failed = false;
    uint64_t node_keys = ~0ull;       // 12 bits per buffer: rectangle, n1, n2 of the nodes it holds
    // early rejection: the misfit only grows with the stations, so once the partial
    // log-likelihood is below the chain's floor the proposal is certainly rejected and its
    // remaining stations are skipped (the llk is then reported as -inf)
    const double floor_llk = (llk_floor && active && !resid) ? llk_floor[chain] : -INFINITY;
    bool stopped = false;
    int u_stop = tile1 - tile0;
    // the finished parts' sum and the part at work, kept out of the registers of the tile loop
    __shared__ double s_sum[WARPS];
    __shared__ int s_part[WARPS];
    if (lane == 0) {
        s_sum[warp] = 0.0;
        s_part[warp] = 0;
    }
    __syncwarp();
    for (int t = tile0; t < tile1; ++t) {
        const int u = t - tile0, buf = u % STAGES;
        const uint32_t phase = (uint32_t)(u / STAGES) & 1u;
        const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[buf], phase, kWaitLimit));
        if (!ok) {
            failed = true;
            break;
        }
        if (smask && !stopped) {
            // this tile's plan: the rectangles it integrates (node counts packed 5 + 5 bits per
            // rectangle) and the sides of the others
            const float4 tb = s_box[buf];
            const float bx0 = __fsub_rn(__fsub_rn(tb.x, x0h), x0l), bx1 = __fsub_rn(__fsub_rn(tb.y, x0h), x0l);
            const float by0 = __fsub_rn(__fsub_rn(tb.z, y0h), y0l), by1 = __fsub_rn(__fsub_rn(tb.w, y0h), y0l);
            uint32_t sides = smask & 0x0FFFu, qrect = 0u, qpack = 0u;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                int n1, n2;
                if ((smask >> (27 + r) & 1u) &&
                    tile_quad(C.rect[r], (smask >> (24 + r)) & 1u, bx0, bx1, by0, by1, n1, n2)) {
                    qrect |= 1u << r;
                    qpack |= (uint32_t)(n1 | (n2 << 5)) << (10 * r);
                    sides &= ~(0xFu << (4 * r));
                }
            }
            // one rectangle's nodes in this warp's buffer (every lane reads all of them); the
            // buffer is refilled only when it holds other nodes
            auto load_nodes = [&](int r) -> const Node* {
                const int n1 = (qpack >> (10 * r)) & 31, n2 = (qpack >> (10 * r + 5)) & 31;
                const int b = kNodeBufs == 3 ? r : 0;
                const uint64_t key = (uint64_t)(r | (n1 << 2) | (n2 << 7));
                if (((node_keys >> (12 * b)) & 0xFFFull) != key) {
                    __syncwarp();
                    if (lane < n1 * n2) {
                        const float4 q = rect_node(C.rect[r], n1, n2, lane, s_gx, s_gw);
                        if constexpr (SPL > 1)
                            s_node[warp][b][lane] =
                                PackedNode{make_float4(-q.x, -q.x, -q.y, -q.y), make_float4(q.z, q.z, q.w, q.w)};
                        else
                            s_node[warp][b][lane] = q;
                    }
                    __syncwarp();
                    node_keys = (node_keys & ~(0xFFFull << (12 * b))) | (key << (12 * b));
                }
                return s_node[warp][b];
            };
            // u projected on the LOS, minus data and offset; accumulate w r² and store r
            auto finish = [&](float e_, float n_, float v_, int j) {
                const float4 B = s_ld[buf][j];
                const float w = s_w[buf][j];
                const float u = fmaf(e_, B.x, fmaf(n_, B.y, v_ * B.z));
                float r = u - B.w;
                if (with_oid) r -= C.off[s_oid[buf][j] & (kMaxOffsets - 1)];
                if (w != 0.f) ff_add_wsq(acc, r, w);
                if (resid) {
                    const int col = t * kTile + j;
                    resid[(size_t)chain * m_padded + (order ? __ldg(order + col) : col)] = (col < m) ? r : 0.f;
                }
            };
            if constexpr (SPL > 1) {
                // stations j, j + 32, ... together; accumulation order as in the one-station loop
                for (int j0 = lane; j0 < kTile; j0 += 32 * SPL) {
                    SV<SPL> Xr, Yr;
#pragma unroll
                    for (int q = 0; q < SPL; ++q) {
                        const float4 A = s_xy[buf][j0 + 32 * q];
                        Xr.v[q] = (A.x - x0h) + (A.y - x0l);
                        Yr.v[q] = (A.z - y0h) + (A.w - y0l);
                    }
                    SV<SPL> ue(0.f), un(0.f), uv(0.f);
                    uint32_t msk = sides;
#pragma unroll 1
                    while (msk) {
                        const int sidx = __ffs(msk) - 1;
                        msk &= msk - 1;
                        side_pair<SV<SPL>>(ScalarSide(C.side[sidx]), Xr, Yr, ue, un, uv, (smask >> (kSides + sidx)) & 1u);
                    }
                    uint32_t qm = qrect;
#pragma unroll 1
                    while (qm) {
                        const int r = __ffs(qm) - 1;
                        qm &= qm - 1;
                        const Node* nodes = load_nodes(r);
                        const int nn = ((qpack >> (10 * r)) & 31) * ((qpack >> (10 * r + 5)) & 31);
                        rect_quad_packed<SPL>(C.rect[r], nodes, nn, Xr, Yr, ue, un, uv);
                    }
#pragma unroll
                    for (int q = 0; q < SPL; ++q) finish(ue.v[q], un.v[q], uv.v[q], j0 + 32 * q);
                }
            } else {
                for (int j = lane; j < kTile; j += 32) {
                    const float4 A = s_xy[buf][j];
                    const float Xr = (A.x - x0h) + (A.y - x0l);
                    const float Yr = (A.z - y0h) + (A.w - y0l);
                    float ue = 0.f, un = 0.f, uv = 0.f;
                    uint32_t msk = sides;
#pragma unroll 1
                    while (msk) {
                        const int sidx = __ffs(msk) - 1;
                        msk &= msk - 1;
                        side_pair<float>(ScalarSide(C.side[sidx]), Xr, Yr, ue, un, uv, (smask >> (kSides + sidx)) & 1u);
                    }
                    uint32_t qm = qrect;
#pragma unroll 1
                    while (qm) {
                        const int r = __ffs(qm) - 1;
                        qm &= qm - 1;
                        const float4* nodes = load_nodes(r);
                        rect_quad<float>(C.rect[r], nodes, ((qpack >> (10 * r)) & 31) * ((qpack >> (10 * r + 5)) & 31),
                                         Xr, Yr, ue, un, uv);
                    }
                    finish(ue, un, uv, j);
                }
            }
            if (floor_llk > -INFINITY && norm - 0.5 * (s_sum[warp] + warp_sum(ff_to_double(acc))) < floor_llk) stopped = true;
            // the end of a part (parts without a tile are left out)
            int part = s_part[warp];
            while (part_begin(part + 1, ntiles) <= t) ++part;
            if (t + 1 == part_begin(part + 1, ntiles)) {
                const double p = warp_sum(ff_to_double(acc));
                if (lane == 0) {
                    if (SPLIT) __stcg(parts + (size_t)slot * kParts + part, p);
                    s_sum[warp] += p;
                    s_part[warp] = part + 1;
                }
                __syncwarp();
                acc = ff{0.f, 0.f};
            }
        }
        // done with this buffer: the last warp of the CTA to get here refills it
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            if (atomicAdd(&s_done[buf], 1) == WARPS - 1) {
                __threadfence_block();
                s_done[buf] = 0;
                if (t + STAGES < tile1) {
                    fence_proxy_async_smem();
                    issue(t + STAGES, buf);
                    atomicAdd(&s_issued, 1);
                }
            }
        }
        // a CTA of one stopped warp leaves the ring; CTAs of several warps keep counting tiles
        // (the stopped warp's share of each tile's completion) without computing
        if (WARPS == 1 && stopped) {
            u_stop = u;
            break;
        }
    }
    if (WARPS == 1 && stopped && !failed) {
        // wait (bounded) for the copies already issued into this CTA's ring before it exits
        if (lane == 0) {
            const int last = s_issued;
            for (int u = u_stop + 1; u < last; ++u)
                mbar_wait_bounded(&full[u % STAGES], (uint32_t)(u / STAGES) & 1u, kWaitLimit);
        }
        __syncwarp();
    }
    if (__syncthreads_or(failed)) {
        // a wait gave up: drain the copies still in flight (bounded) before the CTA exits
        if (threadIdx.x == 0) {
            raise_flag(flags, DEV_ERR_TIMEOUT);
            const int last = s_issued;
            for (int t = (last > STAGES ? last - STAGES : 0); t < last; ++t)
                mbar_wait_bounded(&full[t % STAGES], (uint32_t)(t / STAGES) & 1u, kWaitLimit);
        }
        return;
    }
    if (!SPLIT) {
        if (lane == 0 && active) llk[chain] = stopped ? -INFINITY : norm - 0.5 * s_sum[warp];
        return;
    }
    // the chain's last CTA adds its parts; a CTA that stopped below the floor says so in the count
    int total = 0;
    if (lane == 0) {
        __threadfence();
        total = atomicAdd(done + slot, stopped ? 0x10001 : 1) + (stopped ? 0x10001 : 1);
        __threadfence();
    }
    total = __shfl_sync(0xffffffffu, total, 0);
    if ((total & 0xFFFF) != (int)gridDim.y) return;
    static_assert(kParts == 32, "one part per lane");
    const bool full_part = part_begin(lane, ntiles) < part_begin(lane + 1, ntiles);
    const double p = full_part && (total >> 16) == 0 ? __ldcg(parts + (size_t)slot * kParts + lane) : 0.0;
    double sum = 0.0;
    for (int k = 0; k < kParts; ++k) sum += __shfl_sync(0xffffffffu, p, k);
    if (lane == 0) {
        const double v = norm - 0.5 * sum;
        llk[chain] = (total >> 16) != 0 || v < floor_llk ? -INFINITY : v;
    }
}

// ---------------------------------------------------------------------------
// Mogi: one thread per station, CH chains per CTA held in shared memory, two chains per packed
// FP32 instruction (every element rounded as by the scalar one).  The FMA pipe bounds it: per pair
// 15 operations per source, 18 for the residual and the float-float sum w r², and one reciprocal
// square root.  Beside the scalar instructions' issue slots, FP64 took a sixth of the former
// kernel: 128 conversions and additions per warp at 64 cycles each to add the lanes' sums.  These
// are now added in three FP32 parts, which leave out less than FP64 does, each step halving the
// chains a lane holds, and only the warps' sums in FP64.  16,384 chains x 10,007 stations
// 334 -> 201 µs, 40,000 x 300 219 -> 50 µs, two sources with residual rows, 16,384 x 4,950, 303 -> 187 µs
// (L2 cold; two float-float parts between the lanes took 193, 46 and 183 but lost up to 5 bits against
// FP64; FP64 additions shared out over the lanes took 207, 107 and 191; two CTAs per SM instead of four
// 10% longer).
struct __align__(16) MogiPair {       // a source of two chains
    float4 x;      // x0 hi, hi, lo, lo
    float4 y;
    float4 d;      // depth²,  depth², -depth, -depth
    float2 c;      // C = (nu - 1) ΔV / π
    float2 pad;
};

// a sum in three FP32 parts, each below the last places of the one before: what an addition leaves out
// is below 2^-60 of it (FP64 leaves 2^-53, at 64 cycles per warp instruction)
struct fff { float hi, mid, lo; };
AG_DEVICE_INLINE fff fff_sum(fff a, fff b) {
    float s, e, t, f, u, g;
    two_sum(a.hi, b.hi, s, e);
    two_sum(a.mid, b.mid, t, f);
    two_sum(e, t, u, g);
    return fff{s, u, (a.lo + b.lo) + (f + g)};
}

// sum over the warp of each of N (a power of two from 4 to 32) float-float values per lane, the additions of
// a butterfly shared out over the lanes; on return lane l holds value l / (32 / N)
template <int N>
__device__ __forceinline__ fff warp_sum_ff(const ff (&v)[N], int lane) {
    fff w[N / 2];
    const bool top = lane & 16;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const ff keep = top ? v[i + N / 2] : v[i], send = top ? v[i] : v[i + N / 2];
        const float h = __shfl_xor_sync(0xffffffffu, send.hi, 16), l = __shfl_xor_sync(0xffffffffu, send.lo, 16);
        w[i] = fff_sum(fff{keep.hi, keep.lo, 0.f}, fff{h, l, 0.f});
    }
    int held = N / 2;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const bool split = held > 1, up = split && (lane & o);
        if (split) held >>= 1;
#pragma unroll
        for (int i = 0; i < N / 4; ++i) {
            if (i >= held) break;
            const fff keep = up ? w[i + held] : w[i], send = up || !split ? w[i] : w[i + held];
            fff got;
            got.hi = __shfl_xor_sync(0xffffffffu, send.hi, o);
            got.mid = __shfl_xor_sync(0xffffffffu, send.mid, o);
            got.lo = __shfl_xor_sync(0xffffffffu, send.lo, o);
            w[i] = fff_sum(keep, got);
        }
    }
    return w[0];
}

template <int CH, int NSRC>
__global__ void __launch_bounds__(256, CH <= 16 ? 4 : 2)
mogi_llk_kernel(ag_layout L, const double* __restrict__ theta, int n,
                const uint32_t* __restrict__ mask_in, const float4* __restrict__ xy,
                const float4* __restrict__ losd, const float* __restrict__ wt,
                const int32_t* __restrict__ oid, const int32_t* __restrict__ order, int noffsets, int m,
                int m_padded, double norm, double* __restrict__ llk, float* __restrict__ resid,
                const int32_t* __restrict__ index, const int32_t* __restrict__ count) {
    if (index && (int)(blockIdx.x * CH) >= *count) return;
    constexpr int CP = CH / 2;
    __shared__ MogiPair s_src[CP][NSRC];
    __shared__ int s_chain[CH];
    __shared__ float2 s_off[CP][kMaxOffsets];
    __shared__ int s_act[CH];
    __shared__ fff s_part[CH][8];
    const int c0 = blockIdx.x * CH;
    const double PI = 3.14159265358979323846;
    const int nslots = index ? min(n, *count) : n;
    for (int c = threadIdx.x; c < CH; c += blockDim.x) {
        const int slot = c0 + c;
        const int i = (slot < nslots) ? (index ? index[slot] : slot) : n;
        s_chain[c] = i;
        s_act[c] = (i < n) && !(mask_in && mask_in[i]);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < CH * NSRC; k += blockDim.x) {
        const int c = k / NSRC, src = k % NSRC, i = s_chain[c], h = c & 1;
        float xh = 0.f, xl = 0.f, yh = 0.f, yl = 0.f, d = 0.f, C = 0.f;
        if (i < n) {
            const double* th = theta + (size_t)i * L.nparams + src * L.source_stride;
            split_hilo(th[L.x_idx], xh, xl);
            split_hilo(th[L.x_idx + 1], yh, yl);
            const double dv = L.log_strength ? pow(10.0, th[L.strength_idx]) : th[L.strength_idx];
            d = (float)th[L.depth_idx];
            C = (float)((L.nu - 1.0) * dv / PI);
        }
        float* S = reinterpret_cast<float*>(&s_src[c >> 1][src]);
        S[h] = xh; S[2 + h] = xl;
        S[4 + h] = yh; S[6 + h] = yl;
        S[8 + h] = __fmul_rn(d, d); S[10 + h] = -d;
        S[12 + h] = C;
    }
    if (oid) {
        for (int k = threadIdx.x; k < CH * kMaxOffsets; k += blockDim.x) {
            const int c = k / kMaxOffsets, o = k % kMaxOffsets, i = s_chain[c];
            reinterpret_cast<float*>(&s_off[c >> 1][o])[c & 1] =
                (i < n && o < noffsets) ? (float)theta[(size_t)i * L.nparams + L.offset_idx + o] : 0.f;
        }
    }
    __syncthreads();
    f32x2 hi[CP], lo[CP];
#pragma unroll
    for (int c = 0; c < CP; ++c) hi[c] = lo[c] = 0ull;
    for (int j = threadIdx.x; j < m_padded; j += blockDim.x) {
        const float4 A = __ldg(xy + j);
        const float4 B = __ldg(losd + j);
        const float w = __ldg(wt + j);
        const int o = oid ? (__ldg(oid + j) & (kMaxOffsets - 1)) : 0;
        const int col = order ? __ldg(order + j) : j;
        const f32x2 nax = pack2(-A.x, -A.x), nay = pack2(-A.y, -A.y), naz = pack2(-A.z, -A.z), naw = pack2(-A.w, -A.w);
        const f32x2 bx = pack2(B.x, B.x), by = pack2(B.y, B.y), bz = pack2(B.z, B.z), nd = pack2(-B.w, -B.w);
        const f32x2 w2 = pack2(w, w), nw2 = pack2(-w, -w);
#pragma unroll
        for (int c = 0; c < CP; ++c) {
            f32x2 u = 0ull;
#pragma unroll
            for (int src = 0; src < NSRC; ++src) {
                const MogiPair& S = s_src[c][src];
                const ulonglong2 sx = *reinterpret_cast<const ulonglong2*>(&S.x);
                const ulonglong2 sy = *reinterpret_cast<const ulonglong2*>(&S.y);
                const ulonglong2 sd = *reinterpret_cast<const ulonglong2*>(&S.d);
                const f32x2 sc = *reinterpret_cast<const f32x2*>(&S.c);
                // source minus observation point (libmogi/Source.cc:86-88)
                const f32x2 dx = add2(add2(sx.x, nax), add2(sx.y, nay));
                const f32x2 dy = add2(add2(sy.x, naz), add2(sy.y, naw));
                const f32x2 R2 = fma2(dx, dx, fma2(dy, dy, sd.x));
                float r0, r1;
                unpack2(R2, r0, r1);
                const f32x2 iR = pack2(rsqrtf(r0), rsqrtf(r1));
                const f32x2 iR3 = mul2(mul2(iR, iR), iR);
                const f32x2 proj = fma2(dx, bx, fma2(dy, by, mul2(sd.y, bz)));
                u = fma2(mul2(sc, proj), iR3, u);
            }
            f32x2 r = add2(u, nd);
            if (oid) r = sub2(r, *reinterpret_cast<const f32x2*>(&s_off[c][o]));
            if (w != 0.f) ff2_add_wsq(hi[c], lo[c], r, w2, nw2);
            if (resid) {
                float r0, r1;
                unpack2(r, r0, r1);
                if (s_chain[2 * c] < n) resid[(size_t)s_chain[2 * c] * m_padded + col] = (j < m) ? r0 : 0.f;
                if (s_chain[2 * c + 1] < n) resid[(size_t)s_chain[2 * c + 1] * m_padded + col] = (j < m) ? r1 : 0.f;
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // 1/32 of the lanes' sums, so that the warp's stays below FP32's largest value where they do
    ff v[CH];
    const f32x2 part = pack2(0.03125f, 0.03125f);
#pragma unroll
    for (int c = 0; c < CP; ++c) {
        unpack2(mul2(hi[c], part), v[2 * c].hi, v[2 * c + 1].hi);
        unpack2(mul2(lo[c], part), v[2 * c].lo, v[2 * c + 1].lo);
    }
    const fff sum = warp_sum_ff(v, lane);
    if (lane % (32 / CH) == 0) s_part[lane / (32 / CH)][warp] = sum;
    __syncthreads();
    // eight lanes per chain, in FP64 over the warps
    if (threadIdx.x < 8 * CH) {
        const int c = threadIdx.x >> 3;
        const fff q = s_part[c][threadIdx.x & 7];
        double s = (double)q.hi + ((double)q.mid + (double)q.lo);
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 7) == 0 && s_act[c]) llk[s_chain[c]] = norm - 0.5 * (32.0 * s);
    }
}

}  // namespace ag

// ---------------------------------------------------------------------------
// C ABI
using namespace ag;

// CDM launch variants: warps (= chains) per CTA and resident CTAs per SM the
// register allocation targets; 0, the default, splits the stations of few chains over CTAs and is
// variant 11, the fastest of them at 32,768 x 40,000, for many; the others are chosen per problem by the autotuner
struct CdmVariant { int warps; };
static constexpr CdmVariant kCdmVariants[] = {{1}, {4}, {4}, {2}, {4}, {4}, {2}, {4}, {4}, {4}, {4}, {1}, {1}, {1}, {2}};
static constexpr int kCdmVariantCount = 15;
// Mogi launch variants: chains per CTA held in registers (16, 8, 32)
static constexpr int kMogiChainsOf[] = {16, 8, 32};
static constexpr int kMogiVariantCount = 3;

extern "C" int32_t ag_forward_variants(int model) {
    return model == AG_MODEL_CDM ? kCdmVariantCount : model == AG_MODEL_MOGI ? kMogiVariantCount : 0;
}

// Chains up to which a launch of the default variant splits the stations of a chain over CTAs, and
// the CTAs it aims at: 152 SMs x 12 resident CTAs, eight times over, so that the last wave is a small
// share.  Split against one CTA per chain, slots ordered by cost (chains x stations): 64 x 577
// 45 against 79 µs, 256 x 40,000 665 against 1,928, 1,024 x 5,000 422 against 492, 3,000 x 12,000
// 2,189 against 2,211, but 4,096 x 2,500 756 against 689 and 8,100 x 10,000 4,151 against 3,986:
// the order by cost then does more for the last wave.
constexpr int kSplitChains = 3072;
constexpr int kSplitCtas = 8 * 152 * 12;
static int station_splits(int n, int ntiles) {
    int s = (kSplitCtas - 1) / n + 1;
    if (s > kParts) s = kParts;
    return s < ntiles ? s : ntiles;
}

// CDM workspace: chain constants, the row of each slot, the set-up header (slot count and cost
// histogram), each requested chain's cost bucket; the finished CTAs and the partial misfits of each
// slot of a split launch, which has up to kSplitChains: a population of more takes as much, so that
// its workspace serves every smaller call
struct CdmWorkspace {
    ChainC* chains;
    int32_t* slot_row;
    SetupHdr* hdr;
    int32_t* done;
    int8_t* key;
    double* parts;
};
static size_t al256(size_t b) { return (b + 255) / 256 * 256; }
static size_t cdm_workspace(char* base, int n, CdmWorkspace* w) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        char* p = base + at;
        at += al256(bytes);
        return p;
    };
    const size_t split = n <= kSplitChains ? n : kSplitChains;
    CdmWorkspace ws;
    ws.chains = reinterpret_cast<ChainC*>(take((size_t)n * sizeof(ChainC)));
    ws.slot_row = reinterpret_cast<int32_t*>(take((size_t)n * sizeof(int32_t)));
    ws.hdr = reinterpret_cast<SetupHdr*>(take(sizeof(SetupHdr)));
    ws.done = reinterpret_cast<int32_t*>(take(split * sizeof(int32_t)));     // cleared with the header
    ws.key = reinterpret_cast<int8_t*>(take((size_t)n));
    ws.parts = reinterpret_cast<double*>(take(split * kParts * sizeof(double)));
    if (w) *w = ws;
    return at;
}

extern "C" size_t ag_forward_workspace_bytes(int model, int32_t n) {
    return model == AG_MODEL_CDM && n > 0 ? cdm_workspace(nullptr, n, nullptr) : 0;
}

static int check_stations(const ag_station_set* st) {
    AG_REQUIRE(st != nullptr, "stations is NULL");
    AG_REQUIRE(st->xy && st->losd && st->weight, "station arrays must not be NULL");
    AG_REQUIRE(st->m > 0 && st->m_padded >= st->m && st->m_padded % AG_STATION_TILE == 0,
               "m=%d m_padded=%d: m_padded must be a multiple of %d and >= m", st->m,
               st->m_padded, AG_STATION_TILE);
    AG_REQUIRE(aligned(st->xy, 16) && aligned(st->losd, 16) && aligned(st->weight, 16) &&
                   (st->oid == nullptr || aligned(st->oid, 16)) && (st->order == nullptr || aligned(st->order, 4)),
               "station arrays must be 16-byte aligned (order 4-byte)");
    return AG_OK;
}

static int forward_llk(int model, const ag_layout* layout, const double* theta, int32_t n,
                       const ag_station_set* st, double norm, const uint32_t* mask_in,
                       const int32_t* index, const int32_t* count, const double* llk_floor, double* llk,
                       uint32_t* chain_status, float* residuals, void* workspace,
                       size_t workspace_bytes, void* stream) {
    AG_REQUIRE(layout != nullptr && theta != nullptr && llk != nullptr, "null argument");
    AG_REQUIRE(n > 0, "n must be positive (got %d)", n);
    int rc = check_stations(st);
    if (rc) return rc;
    const ag_layout L = *layout;
    AG_REQUIRE(L.nparams > 0 && L.x_idx >= 0 && L.x_idx + 1 < L.nparams && L.depth_idx >= 0 &&
                   L.depth_idx < L.nparams && L.strength_idx >= 0 && L.strength_idx < L.nparams,
               "invalid parameter layout");
    int noffsets = 0;
    if (st->oid) {
        AG_REQUIRE(L.offset_idx >= 0, "stations carry dataset ids but the layout has no offsets");
        noffsets = L.nparams - L.offset_idx;
        AG_REQUIRE(noffsets > 0 && noffsets <= kMaxOffsets,
                   "between 1 and %d offset parameters are supported", kMaxOffsets);
    }
    cudaStream_t s = as_stream(stream);
    const float4* xy = reinterpret_cast<const float4*>(st->xy);
    const float4* ld = reinterpret_cast<const float4*>(st->losd);
    if (model == AG_MODEL_CDM) {
        AG_REQUIRE(L.axes_idx >= 0 && L.axes_idx + 2 < L.nparams && L.omega_idx >= 0 &&
                       L.omega_idx + 2 < L.nparams,
                   "invalid CDM layout");
        const size_t need = ag_forward_workspace_bytes(model, n);
        AG_REQUIRE(workspace != nullptr && workspace_bytes >= need && aligned(workspace, 256),
                   "CDM needs %zu bytes of 256-byte aligned workspace", need);
        AG_REQUIRE(st->tile_box != nullptr && aligned(st->tile_box, 16),
                   "the CDM needs the stations' tile boxes (ag_station_boxes), 16-byte aligned");
        const float4* tile_box = reinterpret_cast<const float4*>(st->tile_box);
        const int ntiles = st->m_padded / AG_STATION_TILE;
        CdmWorkspace ws;
        cdm_workspace(static_cast<char*>(workspace), n, &ws);
        int32_t* nslots = &ws.hdr->nslots;
        const int v = L.variant;
        AG_REQUIRE(v >= 0 && v < kCdmVariantCount, "CDM variant %d out of range [0, %d)", v, kCdmVariantCount);
        const bool split = v == 0 && n <= kSplitChains;
        rc = cuda_status(cudaMemsetAsync(ws.hdr, 0, al256(sizeof(SetupHdr)) + (split ? (size_t)n * sizeof(int32_t) : 0),
                                         s),
                         "cudaMemsetAsync(set-up header)");
        if (rc) return rc;
        const int setup_ctas = (n + kSetupChains - 1) / kSetupChains;
        if (split) {
            cdm_setup_kernel<false><<<setup_ctas, kSetupThreads, 0, s>>>(L, theta, n, mask_in, chain_status, index,
                                                                        count, noffsets, tile_box, ntiles, ws.chains,
                                                                        ws.key, ws.slot_row, ws.hdr);
        } else {
            cdm_setup_kernel<true><<<setup_ctas, kSetupThreads, 0, s>>>(L, theta, n, mask_in, chain_status, index,
                                                                       count, noffsets, tile_box, ntiles, ws.chains,
                                                                       ws.key, ws.slot_row, ws.hdr);
            cdm_slot_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, ws.key, count, ws.slot_row, ws.hdr);
        }
        rc = launch_status("cdm set-up kernels");
        if (rc) return rc;
        if (split) {
            const dim3 grid(n, station_splits(n, ntiles));
            cdm_llk_kernel<1, 12, 4, 2, true><<<grid, 32, 0, s>>>(
                ws.chains, ws.slot_row, nslots, n, xy, ld, st->weight, st->oid, tile_box, st->order, st->m,
                st->m_padded, norm, llk_floor, llk, residuals, nullptr, ws.parts, ws.done);
            return launch_status("cdm_llk_kernel (split)");
        }
        const int warps = kCdmVariants[v].warps;
        const int grid = (n + warps - 1) / warps;
#define AG_CDM_LAUNCH(W, B, SPL, ST)                                                                             \
    cdm_llk_kernel<W, B, SPL, ST><<<grid, W * 32, 0, s>>>(ws.chains, ws.slot_row, nslots, n, xy, ld, st->weight, \
                                                          st->oid, tile_box, st->order, st->m, st->m_padded,     \
                                                          norm, llk_floor, llk, residuals, nullptr, nullptr,     \
                                                          nullptr)
        // warps per CTA, CTAs per SM, stations per lane, ring depth; a CTA of one warp has its
        // own ring, so its chain never waits for another chain's tiles
        switch (v) {
            case 0: AG_CDM_LAUNCH(1, 12, 4, 2); break;
            case 1: AG_CDM_LAUNCH(4, 4, 1, 4); break;
            case 2: AG_CDM_LAUNCH(4, 5, 1, 4); break;
            case 3: AG_CDM_LAUNCH(2, 8, 1, 4); break;
            case 4: AG_CDM_LAUNCH(4, 3, 2, 4); break;
            case 5: AG_CDM_LAUNCH(4, 4, 2, 4); break;
            case 6: AG_CDM_LAUNCH(2, 6, 2, 4); break;
            case 7: AG_CDM_LAUNCH(4, 2, 4, 4); break;
            case 8: AG_CDM_LAUNCH(4, 3, 4, 4); break;
            case 9: AG_CDM_LAUNCH(4, 4, 4, 4); break;
            case 10: AG_CDM_LAUNCH(4, 5, 4, 4); break;
            case 11: AG_CDM_LAUNCH(1, 12, 4, 2); break;
            case 12: AG_CDM_LAUNCH(1, 12, 4, 3); break;
            case 13: AG_CDM_LAUNCH(1, 10, 4, 3); break;
            default: AG_CDM_LAUNCH(2, 6, 4, 3); break;
        }
#undef AG_CDM_LAUNCH
        return launch_status("cdm_llk_kernel");
    }
    if (model == AG_MODEL_MOGI) {
        AG_REQUIRE(L.nsources == 1 || L.nsources == 2, "1 or 2 Mogi sources are supported");
        AG_REQUIRE(L.variant >= 0 && L.variant < kMogiVariantCount, "Mogi variant %d out of range [0, %d)",
                   L.variant, kMogiVariantCount);
        // the default takes fewer chains per CTA where sixteen would leave SMs
        // with fewer than two: 4,096 x 3,000 27.0 µs with 8 and 32.9 with 32, 1,024 x 1,024 10.6 with 4
        // and 16.6 with 32
        const int ch = L.variant != 0 ? kMogiChainsOf[L.variant] : n >= 16 * 304 ? 16 : n >= 8 * 304 ? 8 : 4;
        const int grid = (n + ch - 1) / ch;
#define AG_MOGI_LAUNCH(CH, NS)                                                                               \
    mogi_llk_kernel<CH, NS><<<grid, 256, 0, s>>>(L, theta, n, mask_in, xy, ld, st->weight, st->oid, st->order, \
                                                 noffsets, st->m, st->m_padded, norm, llk, residuals, index, count)
        if (L.nsources == 1) {
            if (ch == 4) AG_MOGI_LAUNCH(4, 1);
            else if (ch == 8) AG_MOGI_LAUNCH(8, 1);
            else if (ch == 32) AG_MOGI_LAUNCH(32, 1);
            else AG_MOGI_LAUNCH(16, 1);
        } else {
            if (ch == 4) AG_MOGI_LAUNCH(4, 2);
            else if (ch == 8) AG_MOGI_LAUNCH(8, 2);
            else if (ch == 32) AG_MOGI_LAUNCH(32, 2);
            else AG_MOGI_LAUNCH(16, 2);
        }
#undef AG_MOGI_LAUNCH
        return launch_status("mogi_llk_kernel");
    }
    return set_error(AG_ERR_ARG, "unknown model %d", model);
}

extern "C" int ag_forward_llk(int model, const ag_layout* layout, const double* theta, int32_t n,
                              const ag_station_set* st, double norm, const uint32_t* mask_in,
                              double* llk, uint32_t* chain_status, float* residuals,
                              void* workspace, size_t workspace_bytes, void* stream) {
    return forward_llk(model, layout, theta, n, st, norm, mask_in, nullptr, nullptr, nullptr, llk, chain_status,
                       residuals, workspace, workspace_bytes, stream);
}

extern "C" int ag_forward_llk_floor(int model, const ag_layout* layout, const double* theta, int32_t n,
                                    const ag_station_set* st, double norm, const uint32_t* mask_in,
                                    const double* llk_floor, double* llk, uint32_t* chain_status,
                                    void* workspace, size_t workspace_bytes, void* stream) {
    AG_REQUIRE(llk_floor != nullptr, "llk_floor must not be NULL (ag_forward_llk evaluates without one)");
    return forward_llk(model, layout, theta, n, st, norm, mask_in, nullptr, nullptr, llk_floor, llk, chain_status,
                       nullptr, workspace, workspace_bytes, stream);
}

extern "C" int ag_forward_llk_subset_floor(int model, const ag_layout* layout, const double* theta, int32_t n,
                                           const ag_station_set* st, double norm, const int32_t* index,
                                           const int32_t* count, const double* llk_floor, double* llk,
                                           uint32_t* chain_status, void* workspace, size_t workspace_bytes,
                                           void* stream) {
    AG_REQUIRE(index != nullptr && count != nullptr && llk_floor != nullptr,
               "index, count and llk_floor must not be NULL");
    return forward_llk(model, layout, theta, n, st, norm, nullptr, index, count, llk_floor, llk, chain_status,
                       nullptr, workspace, workspace_bytes, stream);
}

extern "C" int ag_forward_llk_subset(int model, const ag_layout* layout, const double* theta,
                                     int32_t n, const ag_station_set* st, double norm,
                                     const int32_t* index, const int32_t* count, double* llk,
                                     uint32_t* chain_status, float* residuals, void* workspace,
                                     size_t workspace_bytes, void* stream) {
    AG_REQUIRE(index != nullptr && count != nullptr, "index and count must not be NULL");
    return forward_llk(model, layout, theta, n, st, norm, nullptr, index, count, nullptr, llk, chain_status,
                       residuals, workspace, workspace_bytes, stream);
}

extern "C" int ag_cdm_work(const ag_layout* layout, const double* theta, int32_t n, const ag_station_set* st,
                           double* flop, double* sfu, void* stream) {
    AG_REQUIRE(layout && theta && flop && n > 0, "invalid arguments");
    int rc = check_stations(st);
    if (rc) return rc;
    AG_REQUIRE(st->tile_box != nullptr && aligned(st->tile_box, 16),
               "the CDM needs the stations' tile boxes (ag_station_boxes), 16-byte aligned");
    const ag_layout L = *layout;
    AG_REQUIRE(L.nparams > 0 && L.axes_idx >= 0 && L.axes_idx + 2 < L.nparams && L.omega_idx >= 0 &&
                   L.omega_idx + 2 < L.nparams,
               "invalid CDM layout");
    cdm_work_kernel<<<(n + 127) / 128, 128, 0, as_stream(stream)>>>(
        L, theta, n, reinterpret_cast<const float4*>(st->tile_box), st->m, flop, sfu);
    return launch_status("cdm_work_kernel");
}

extern "C" int ag_station_boxes(const float* xy, int32_t m, int32_t m_padded, float* tile_box, void* stream) {
    AG_REQUIRE(xy && tile_box && m > 0 && m_padded >= m && m_padded % AG_STATION_TILE == 0,
               "invalid arguments (m=%d, m_padded=%d must be a multiple of %d)", m, m_padded, AG_STATION_TILE);
    AG_REQUIRE(aligned(xy, 16) && aligned(tile_box, 16), "xy and tile_box must be 16-byte aligned");
    const int ntiles = m_padded / AG_STATION_TILE;
    station_boxes_kernel<<<(ntiles + 7) / 8, 256, 0, as_stream(stream)>>>(
        reinterpret_cast<const float4*>(xy), m, ntiles, reinterpret_cast<float4*>(tile_box));
    return launch_status("station_boxes_kernel");
}

extern "C" int ag_cdm_check(const ag_layout* layout, const double* theta, int32_t n,
                            uint32_t* chain_status, void* stream) {
    AG_REQUIRE(layout && theta && chain_status && n > 0, "invalid arguments");
    cdm_check_kernel<<<(n + 127) / 128, 128, 0, as_stream(stream)>>>(*layout, theta, n, chain_status);
    return launch_status("cdm_check_kernel");
}
