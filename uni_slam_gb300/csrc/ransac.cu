// ransac.cu — batched RANSAC hypothesis scoring: the step after matching.
//
// The reference's RansacCPU (wslam/src/pose_estimate_cpu/ransac_cpu.cpp)
// fits a fundamental matrix to 8 random matches per iteration and classifies
// every match by its Sampson distance (SampsonDistance, :183-196;
// ClassifyInliers, :198-210).  The fit (an SVD) stays on the host; this file
// scores many hypotheses against all matches at once on the GPU.
//
// Arithmetic: binary64, no contraction (--fmad=false), in this order:
//   Fx  = F xp            component r: (F[r][0] x_p + F[r][1] y_p) + F[r][2]
//   Ftx = F^T xc          component c: (F[0][c] x_c + F[1][c] y_c) + F[2][c]
//   num = (x_c Fx0 + y_c Fx1) + Fx2
//   den = ((Fx0^2 + Fx1^2) + Ftx0^2) + Ftx1^2
//   d   = den < 1e-12 ? +inf : num^2 / den;   inlier iff d < threshold.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

#include "runtime_internal.h"

namespace {

constexpr int KR_THREADS = 256;  // matches of a CTA
constexpr int KR_HYPS = 8;       // hypotheses of a CTA

__device__ __forceinline__ bool sampson_inlier(const double* F, double xp, double yp, double xc, double yc,
                                               double thr) {
    const double fx0 = (F[0] * xp + F[1] * yp) + F[2];
    const double fx1 = (F[3] * xp + F[4] * yp) + F[5];
    const double fx2 = (F[6] * xp + F[7] * yp) + F[8];
    const double ft0 = (F[0] * xc + F[3] * yc) + F[6];
    const double ft1 = (F[1] * xc + F[4] * yc) + F[7];
    const double num = (xc * fx0 + yc * fx1) + fx2;
    const double den = ((fx0 * fx0 + fx1 * fx1) + ft0 * ft0) + ft1 * ft1;
    if (den < 1e-12) return false;  // infinite distance
    return (num * num) / den < thr;
}

// A hypothesis in binary32: the matrix times a power of two (an exact step
// that leaves num^2 / den as it is) so that its largest entry is in [1, 2).
struct HypF {
    float f[9];
    float den_min;  // 1e-12 on the scaled matrix
    int sane;       // the decision below applies
};

// The inlier decision in binary32 where it is certain: 1 inlier, 0 outlier, -1
// too close to tell.  Every value carries a bound of its distance from the
// exact one: a component of F x or F^T x is a sum of three products of rounded
// inputs, off by at most 6 units of 2^-24 of the sum of its terms' magnitudes,
// and num by at most 10; 2^-20 (16 units) covers both and the rounding of the
// bounds themselves.  The binary64 evaluation differs from the exact values by
// 2^-49 of the same sums, far inside what is left.  NaN and infinities compare
// false and are not certain.  The bounds are relative, so they miss what a
// matrix entry or a product below binary32's normal range loses: at most 2^-150
// each, and 9 (1 + c)^2 2^-150 in num for coordinates up to c.  For c < 1e9
// (the caller sees to that) this is below 1e-26, against en > 1e-20 and
// components whose squares add up to lo > 1e-20.
__device__ __forceinline__ int sampson_certain(const HypF& H, float xp, float yp, float xc, float yc, float thr) {
    constexpr float g = 9.5367431640625e-07f;  // 2^-20
    const float* F = H.f;
    const float fx0 = F[0] * xp + F[1] * yp + F[2], ax0 = fabsf(F[0] * xp) + fabsf(F[1] * yp) + fabsf(F[2]);
    const float fx1 = F[3] * xp + F[4] * yp + F[5], ax1 = fabsf(F[3] * xp) + fabsf(F[4] * yp) + fabsf(F[5]);
    const float fx2 = F[6] * xp + F[7] * yp + F[8], ax2 = fabsf(F[6] * xp) + fabsf(F[7] * yp) + fabsf(F[8]);
    const float ft0 = F[0] * xc + F[3] * yc + F[6], at0 = fabsf(F[0] * xc) + fabsf(F[3] * yc) + fabsf(F[6]);
    const float ft1 = F[1] * xc + F[4] * yc + F[7], at1 = fabsf(F[1] * xc) + fabsf(F[4] * yc) + fabsf(F[7]);
    const float num = fabsf(xc * fx0 + yc * fx1 + fx2);
    const float en = g * (fabsf(xc) * ax0 + fabsf(yc) * ax1 + ax2);
    // den between lo and hi, with a relative 2^-20 for their own rounding
    const float c0 = fabsf(fx0), c1 = fabsf(fx1), c2 = fabsf(ft0), c3 = fabsf(ft1);
    const float e0 = g * ax0, e1 = g * ax1, e2 = g * at0, e3 = g * at1;
    const float l0 = fmaxf(c0 - e0, 0.0f), l1 = fmaxf(c1 - e1, 0.0f), l2 = fmaxf(c2 - e2, 0.0f), l3 = fmaxf(c3 - e3, 0.0f);
    const float h0 = c0 + e0, h1 = c1 + e1, h2 = c2 + e2, h3 = c3 + e3;
    const float lo = (l0 * l0 + l1 * l1 + l2 * l2 + l3 * l3) * (1.0f - g);
    const float hi = (h0 * h0 + h1 * h1 + h2 * h2 + h3 * h3) * (1.0f + g);
    // (values far from the range's ends, so no product above lost bits to underflow or overflow)
    if (!H.sane || !(lo > H.den_min && lo > 1e-20f && hi < 1e30f && en > 1e-20f)) return -1;
    const float far = num + en, near = num - en;
    if (far * far * (1.0f + g) < thr * lo) return 1;
    if (near > 0.0f && near * near * (1.0f - g) > thr * hi) return 0;
    return -1;
}

// A CTA scores KR_HYPS hypotheses on KR_THREADS matches, a thread one match:
// in binary32 where that decides (all but about one match in a thousand), else
// in binary64 as the definition above.  FP64 runs at 1/64 of the FP32 rate on
// this GPU: the binary64 evaluation of every pair took 83 us for 500 x 1640.
__global__ void __launch_bounds__(KR_THREADS)
k_sampson(const double* __restrict__ fmats, int n_hyp, const double2* __restrict__ prev,
          const double2* __restrict__ curr, int n, double thr, int* __restrict__ counts,
          uint32_t* __restrict__ masks) {
    __shared__ HypF s_h[KR_HYPS];
    __shared__ int s_cnt[KR_HYPS];
    const int h0 = blockIdx.y * KR_HYPS, nh = min(KR_HYPS, n_hyp - h0);
    if (threadIdx.x < nh) {
        const double* F = fmats + (size_t)(h0 + threadIdx.x) * 9;
        double m = 0.0;
        bool finite = true;
        for (int k = 0; k < 9; ++k) {
            m = fmax(m, fabs(F[k]));
            finite = finite && isfinite(F[k]);
        }
        HypF H;
        // the scale 2^-e and its square stay normal numbers for e within +-400
        const int e = finite && m > 0.0 ? ilogb(m) : 9999;
        H.sane = e > -400 && e < 400 && thr > 1e-6 && thr < 1e6 ? 1 : 0;
        const double s = H.sane ? scalbn(1.0, -e) : 0.0;
        for (int k = 0; k < 9; ++k) H.f[k] = (float)(F[k] * s);
        // rounded up, and one too large for binary32 leaves nothing certain
        H.den_min = __double2float_ru(fmin(1e-12 * s * s, 1e38) * 1.001);
        s_h[threadIdx.x] = H;
        s_cnt[threadIdx.x] = 0;
    }
    __syncthreads();
    const int i = blockIdx.x * KR_THREADS + threadIdx.x, lane = threadIdx.x & 31;
    const int words = (n + 31) / 32;
    double2 p = make_double2(0.0, 0.0), q = p;
    if (i < n) {
        p = prev[i];
        q = curr[i];
    }
    const float yp = (float)p.y, xc = (float)q.x, yc = (float)q.y, t = (float)thr;
    float xp = (float)p.x;
    // far coordinates are not certain: not a number here
    if (!(fabsf(xp) < 1e9f && fabsf(yp) < 1e9f && fabsf(xc) < 1e9f && fabsf(yc) < 1e9f)) xp = __int_as_float(0x7fc00000);
    for (int k = 0; k < nh; ++k) {
        bool in = false;
        if (i < n) {
            const int c = sampson_certain(s_h[k], xp, yp, xc, yc, t);
            in = c > 0;
            if (c < 0) {
                double F[9];
#pragma unroll
                for (int m = 0; m < 9; ++m) F[m] = __ldg(fmats + (size_t)(h0 + k) * 9 + m);
                in = sampson_inlier(F, p.x, p.y, q.x, q.y, thr);
            }
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, in);
        if (lane == 0) {
            if (bal) atomicAdd(&s_cnt[k], __popc(bal));
            if (masks && (i >> 5) < words) masks[(size_t)(h0 + k) * words + (i >> 5)] = bal;
        }
    }
    __syncthreads();
    if (threadIdx.x < nh && s_cnt[threadIdx.x]) atomicAdd(counts + h0 + threadIdx.x, s_cnt[threadIdx.x]);
}

}  // namespace

extern "C" {

uslam_status uslam_ransac_score(uslam_ctx* ctx, const double* fmats, int n_hyp, const double* prev_xy,
                                const double* curr_xy, int n_matches, double threshold, int* counts,
                                uint32_t* masks) {
    if (!ctx || n_hyp < 0 || n_matches < 0 || !counts || (n_hyp > 0 && !fmats) ||
        (n_matches > 0 && (!prev_xy || !curr_xy)))
        return set_err(ctx ? &ctx->err : nullptr, USLAM_INVALID_ARG, "ransac_score: bad arguments");
    if (n_hyp == 0) return USLAM_OK;
    cudaError_t e = cudaSetDevice(ctx->device);
    const int words = (n_matches + 31) / 32;
    const size_t f_b = uslam_rt::round_up(sizeof(double) * 9 * static_cast<size_t>(n_hyp), 256);
    const size_t m_b = uslam_rt::round_up(sizeof(double) * 2 * static_cast<size_t>(std::max(n_matches, 1)), 256);
    const size_t c_b = uslam_rt::round_up(sizeof(int) * static_cast<size_t>(n_hyp), 256);
    const size_t k_b = masks ? uslam_rt::round_up(sizeof(uint32_t) * words * static_cast<size_t>(n_hyp), 256) : 0;
    const size_t need = f_b + 2 * m_b + c_b + k_b;
    std::lock_guard<std::mutex> lk(ctx->ransac_mu);
    if (e == cudaSuccess && need > ctx->ransac_bytes) {
        if (ctx->ransac_buf) cudaFree(ctx->ransac_buf);
        ctx->ransac_buf = nullptr;
        ctx->ransac_bytes = 0;
        e = cudaMalloc(&ctx->ransac_buf, need);
        if (e == cudaSuccess) ctx->ransac_bytes = need;
    }
    if (e != cudaSuccess) return ctx->cuda_fail(e, "ransac_score: scratch");
    const bool pinned = ctx->ransac_pin.reserve(need);
    char* base = static_cast<char*>(ctx->ransac_buf);
    double* d_f = reinterpret_cast<double*>(base);
    double2* d_p = reinterpret_cast<double2*>(base + f_b);
    double2* d_q = reinterpret_cast<double2*>(base + f_b + m_b);
    int* d_c = reinterpret_cast<int*>(base + f_b + 2 * m_b);
    uint32_t* d_k = masks ? reinterpret_cast<uint32_t*>(base + f_b + 2 * m_b + c_b) : nullptr;
    // one copy each way through pinned staging laid out as the scratch (the
    // counts start at zero in it)
    const size_t in_b = f_b + 2 * m_b + c_b, f_n = sizeof(double) * 9 * n_hyp, m_n = sizeof(double) * 2 * n_matches;
    char* const pin = pinned ? ctx->ransac_pin.p : nullptr;
    if (pin) {
        std::memcpy(pin, fmats, f_n);
        if (n_matches > 0) {
            std::memcpy(pin + f_b, prev_xy, m_n);
            std::memcpy(pin + f_b + m_b, curr_xy, m_n);
        }
        std::memset(pin + f_b + 2 * m_b, 0, c_b);
        e = cudaMemcpyAsync(base, pin, in_b, cudaMemcpyHostToDevice, 0);
    } else {
        e = cudaMemcpy(d_f, fmats, f_n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess && n_matches > 0) e = cudaMemcpy(d_p, prev_xy, m_n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess && n_matches > 0) e = cudaMemcpy(d_q, curr_xy, m_n, cudaMemcpyHostToDevice);
        if (e == cudaSuccess) e = cudaMemset(d_c, 0, c_b);
    }
    if (e == cudaSuccess && n_matches > 0) {
        const int hyps = 65535 * KR_HYPS;  // of one launch
        for (int h = 0; h < n_hyp && e == cudaSuccess; h += hyps) {
            const int m = std::min(hyps, n_hyp - h);
            const dim3 grid((n_matches + KR_THREADS - 1) / KR_THREADS, (m + KR_HYPS - 1) / KR_HYPS);
            k_sampson<<<grid, KR_THREADS>>>(d_f + static_cast<size_t>(h) * 9, m, d_p, d_q, n_matches, threshold, d_c + h,
                                            d_k ? d_k + static_cast<size_t>(h) * words : nullptr);
            e = cudaGetLastError();
        }
    }
    const size_t c_n = sizeof(int) * n_hyp, k_n = masks ? sizeof(uint32_t) * words * static_cast<size_t>(n_hyp) : 0;
    if (pin) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(pin + in_b - c_b, d_c, c_b + k_b, cudaMemcpyDeviceToHost, 0);
        if (e == cudaSuccess) e = cudaStreamSynchronize(0);
        if (e == cudaSuccess) std::memcpy(counts, pin + in_b - c_b, c_n);
        if (e == cudaSuccess && masks) std::memcpy(masks, pin + in_b, k_n);
    } else {
        if (e == cudaSuccess) e = cudaMemcpy(counts, d_c, c_n, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && masks) e = cudaMemcpy(masks, d_k, k_n, cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) return ctx->cuda_fail(e, "ransac_score");
    return USLAM_OK;
}

}  // extern "C"
