// Reverso two-reservoir magma model (Reverso et al. 2014): predicted GPS
// displacements, residuals and the diagonal-Cd data log-likelihood of a batch
// of samples, in FP64.
//
// Reference: models/reverso/lib/libreverso/reverso.cc:37-142 (the forward model
// the default strategy calls, Source.cc:56-88), Source.cc:92-123 (residuals) and
// Fast.py:52-90 (llk = norm - |L r|²/2, L = chol(Cd⁻¹), per sample on the host).
// The reference's algebra is kept, quirks included: τ uses H_c^γ_s
// (reverso.cc:60-61) and the pressures 1 - exp(-t/τ) (reverso.cc:79).  The E/N
// split u_r·(cos φ, sin φ) with φ = atan2(y, x) is evaluated as (x, y)·F with
// u_r = r F, which is the same quantity without the angle (and is 0 at r = 0,
// where the reference's atan2(0, 0) = 0 also gives 0).
//
// What bounds it is FP64 issue (a warp instruction takes an SM quarter 64 cycles) and, before
// that, the ~200 dependent FP64 instructions of a sample's constants.  A block takes up to 32
// samples: four warps form their constants, a lane per sample and a part of the constants per
// warp, then the threads take the (sample, point) pairs of kRevTile points at a time, whatever
// the number of points, so no lane idles and no constant is computed twice; the pairs'
// contributions are added per sample in an order that depends on the points alone, so results do
// not depend on the launch (or on how a population is split).  Blocks are sized to a whole number
// per SM.  A pair takes ~70 FP64 instructions: r² is formed once per block and point, r^-5 from one
// reciprocal square root, exp(-t/τ) without the division.  Measured, 4,096 samples of 35 points:
// 26 µs (118 µs with a warp per sample: its constants in every lane, 35 points on 64 lanes).
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "internal.h"

namespace ag {

constexpr int kRevThreads = 256;
constexpr int kRevSamples = 32;        // most samples per block
constexpr int kRevTile = 128;          // observation points per pass

// a sample's constants (reverso.cc:44-68)
enum : int { R_POW, R_IPRE, R_A, R_C1, R_CD, R_HS, R_HD, R_KS, R_KD, R_COUNT };

// k R^-5 (or k R^-3) from R².  With i ≈ 1/R and i² rounded, 1 - R² i² (one FMA, exact to its own
// rounding) is the relative error of i², and so, times 5/2 (3/2), that of the power.  An infinite R² (a
// squared distance or depth beyond FP64) gives 0 as the division does, not 0 times that error's NaN.
__device__ __forceinline__ double inverse_power(double k, double R2, bool cube) {
    const double i = rsqrt(R2), i2 = i * i;
    const double err = __double2hiint(R2) >= 0x7ff00000 ? 0.0 : fma(-R2, i2, 1.0);
    const double p = k * (cube ? i2 * i : i2 * i2 * i);
    return fma(p, (cube ? 1.5 : 2.5) * err, p);
}

__global__ void __launch_bounds__(kRevThreads)
reverso_llk_kernel(ag_reverso_model M, const double* __restrict__ theta, int n, int per_block, double norm,
                   const uint32_t* __restrict__ mask, double* __restrict__ llk,
                   double* __restrict__ predicted) {
    const double PI = 3.14159265358979323846;
    __shared__ double s_c[R_COUNT][kRevSamples];
    __shared__ double s_r2[kRevTile];
    __shared__ double s_part[kRevSamples * kRevTile];
    __shared__ uint32_t s_skip[kRevSamples];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = blockIdx.x * per_block;
    const int samples = n - i0 < per_block ? n - i0 : per_block;
    const double gamma_s = 8.0 * (1.0 - M.v) / (3.0 * PI), gamma_d = gamma_s;
    if (warp < 4 && lane < samples) {
        const double* th = theta + (size_t)(i0 + lane) * M.nparams;
        const double Qin = th[M.qin_idx], H_s = th[M.hs_idx], H_d = th[M.hd_idx];
        const double a_s = th[M.as_idx], a_d = th[M.ad_idx], a_c = th[M.ac_idx];
        const double H_c = H_d - H_s;
        if (warp == 0) {
            s_c[R_POW][lane] = pow(H_c, -gamma_s);
            s_skip[lane] = mask ? mask[i0 + lane] : 0u;
        } else {
            const double q = a_d / a_s;
            const double k = q * q * q;
            const double gamma_r = gamma_s + gamma_d * k;
            const double as3 = a_s * a_s * a_s, ad3 = a_d * a_d * a_d, ac4 = a_c * a_c * a_c * a_c;
            if (warp == 1) {
                // τ = 8 μ H_c^γ_s γ_d k a_s³/(G a_c⁴ γ_r): 1/τ without the power
                s_c[R_IPRE][lane] = (M.G * ac4 * gamma_r) / (8.0 * M.mu * gamma_d * k * as3);
                s_c[R_HS][lane] = H_s;
                s_c[R_HD][lane] = H_d;
            } else if (warp == 2) {
                s_c[R_A][lane] = gamma_d * k / gamma_r *
                                 (M.drho * M.g * H_c - 8.0 * gamma_s * M.mu * Qin * H_c / (PI * ac4 * gamma_r));
                s_c[R_CD][lane] = gamma_s / (gamma_d * k);
            } else {
                s_c[R_C1][lane] = M.G * Qin / (PI * as3 * gamma_r);
                const double ks = as3 * (1.0 - M.v) / M.G, kd = ad3 * (1.0 - M.v) / M.G;
                s_c[R_KS][lane] = gamma_s == 1.0 ? ks : ks * (4.0 * H_s * H_s / PI);
                s_c[R_KD][lane] = gamma_d == 1.0 ? kd : kd * (4.0 * H_d * H_d / PI);
            }
        }
    }
    double acc = 0.0;                          // thread 8 c + k: its share of sample c's misfit
    for (int j0 = 0; j0 < M.n_obs; j0 += kRevTile) {
        const int tile = M.n_obs - j0 < kRevTile ? M.n_obs - j0 : kRevTile;
        if (warp >= 4) {                       // while the other warps form the constants
            for (int j = tid - 128; j < tile; j += kRevThreads - 128) {
                const double x = M.txy[3 * (j0 + j) + 1], y = M.txy[3 * (j0 + j) + 2];
                s_r2[j] = x * x + y * y;
            }
        }
        __syncthreads();
        for (int e = tid; e < samples * tile; e += kRevThreads) {
            const int c = e / tile, jt = e - c * tile, j = j0 + jt;
            if (s_skip[c]) continue;
            const double t = M.txy[3 * j], x = M.txy[3 * j + 1], y = M.txy[3 * j + 2];
            // pressures (reverso.cc:78-83)
            const double A = s_c[R_A][c];
            const double f0 = A * (1.0 - exp(-t * (s_c[R_IPRE][c] * s_c[R_POW][c])));
            const double f1 = s_c[R_C1][c] * t;
            const double dP_s = f1 + f0;
            const double dP_d = f1 - f0 * s_c[R_CD][c];
            // Green's functions of the two reservoirs (reverso.cc:109-142): a³ (1 - ν)/G · 4 H²/(π R²)/R³
            const double H_s = s_c[R_HS][c], H_d = s_c[R_HD][c];
            const double f_s = inverse_power(s_c[R_KS][c], s_r2[jt] + H_s * H_s, gamma_s == 1.0);
            const double f_d = inverse_power(s_c[R_KD][c], s_r2[jt] + H_d * H_d, gamma_d == 1.0);
            const double us = f_s * dP_s, ud = f_d * dP_d;
            const double F = us + ud;                            // u_r / r
            const double* d = M.d + 3 * j;
            const double* w = M.w + 3 * j;
            const double xe = M.east_cos ? x : y, xn = M.east_cos ? y : x;
            if (predicted) {
                double* out = predicted + (size_t)(i0 + c) * 3 * M.n_obs + 3 * j;
                out[0] = xe * F;
                out[1] = xn * F;
                out[2] = fma(H_s, us, H_d * ud);
            }
            const double re = fma(xe, F, -d[0]), rn = fma(xn, F, -d[1]), rz = fma(H_s, us, fma(H_d, ud, -d[2]));
            s_part[c * kRevTile + jt] = fma(w[0] * re, re, fma(w[1] * rn, rn, w[2] * rz * rz));
        }
        __syncthreads();
        const int c = tid >> 3;
        if (c < samples)
            for (int jt = tid & 7; jt < tile; jt += 8) acc += s_part[c * kRevTile + jt];
    }
    for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int c = tid >> 3;
    if ((tid & 7) == 0 && c < samples && !s_skip[c]) llk[i0 + c] = norm - 0.5 * acc;
}

}  // namespace ag

using namespace ag;

extern "C" int ag_reverso_llk(const ag_reverso_model* model, const double* theta, int32_t n, double norm,
                              const uint32_t* mask, double* llk, double* predicted, void* stream) {
    AG_REQUIRE(model != nullptr && theta != nullptr && llk != nullptr, "null argument");
    AG_REQUIRE(n > 0, "n must be positive (got %d)", n);
    const ag_reverso_model M = *model;
    AG_REQUIRE(M.txy && M.d && M.w && M.n_obs > 0, "observation arrays must be given (n_obs=%d)", M.n_obs);
    const int idx[6] = {M.qin_idx, M.hs_idx, M.hd_idx, M.as_idx, M.ad_idx, M.ac_idx};
    for (int k = 0; k < 6; ++k)
        AG_REQUIRE(idx[k] >= 0 && idx[k] < M.nparams, "parameter index %d out of range [0, %d)", idx[k],
                   M.nparams);
    AG_REQUIRE(M.G > 0.0, "shear modulus must be positive");
    int dev = 0, sms = 0;
    int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    rc = cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "multiProcessorCount");
    if (rc) return rc;
    // samples per block: at most kRevSamples, in a whole number of blocks per SM
    const int per_sm = (n - 1) / sms + 1;
    const int waves = (per_sm - 1) / kRevSamples + 1;
    const int per_block = (per_sm - 1) / waves + 1;
    reverso_llk_kernel<<<(n - 1) / per_block + 1, kRevThreads, 0, as_stream(stream)>>>(M, theta, n, per_block, norm,
                                                                                      mask, llk, predicted);
    return launch_status("reverso_llk_kernel");
}
