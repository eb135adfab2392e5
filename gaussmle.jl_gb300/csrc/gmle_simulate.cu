// gmle_simulate.cu - synthetic ROIs on the device (gmle_simulate_device).
//
// The reference simulator (src/simulator.jl:228-307, `_generate_single_roi!`)
// draws, per pixel (i, j) of a ROI, Poisson(mu) photo-electrons with
// mu = bg + N psf_x(j) psf_y(i) (`_evaluate_psf_pixel`, src/simulator.jl:
// 312-346); an sCMOS camera adds Normal(0, readnoise) and converts to ADU,
// total / gain + offset.  This kernel makes the same stacks at GPU rates, as
// benchmark input and as a check of the noise model against the fits.  Its
// random streams are its own (the reference's Julia RNG and Poisson sampler
// cannot be reproduced):
//
// * Philox4x32-10 (Salmon, Moraes, Dror and Shaw, "Parallel random numbers:
//   as easy as 1, 2, 3", SC 2011): key = the 64-bit seed, counter = (pixel
//   index, ROI index low word, high word, block), so a pixel's draws depend
//   only on (seed, ROI, pixel), whatever the launch shape; a 32-bit word w
//   gives the uniform ((w >> 8) + 0.5) / 2^24 in float;
// * Poisson(lam): lam < 10 by inversion in float (sequential search of the
//   CDF from expf(-lam)), lam >= 10 by Hormann's transformed rejection with
//   squeeze (PTRS, "The transformed rejection method for generating Poisson
//   random variables", 1993), in float but for the exact acceptance test at
//   lam >= 64, in double (and only where a float estimate of it does not
//   decide); lam <= 0 gives 0 as in the reference;
// * read noise by Box-Muller in float from its own counter block;
// * mu in float from erf-integrated 1-D Gaussians (src/gausslib/
//   baselibrary.jl:8-14; astigmatic widths sigma0 sqrt(alpha(z -+ gamma)),
//   baselibrary.jl:75-83), the camera arithmetic in float in the
//   reference's order, every operation rounded on its own (no contraction).
//
// Maps are indexed like the fitting kernel, row = y (the reference simulator
// indexes its maps transposed, src/simulator.jl:292-304).  Layout: ROI k's
// pixel (i, j) at (i-1) + box (j-1) + box^2 k, true parameters (P, n)
// column-major in the fitted parameter order.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "gmle_fit_kernel.cuh"
#include "gmle_internal.h"

using gmle::log_approx;
using gmle::rcp_approx;

namespace {

constexpr int kSimThreads = 256;
constexpr int kSimPixels = 2048;  // output pixels per block (whole ROIs)
constexpr int kSimMaxRois = 64;   // ROIs per block (axis tables in shared memory)
constexpr int kSimMaxBox = 32;
constexpr uint32_t kNoiseBlock = 0xFFFF;  // counter block of the read-noise draw

struct Words {
    uint32_t w[4];
};

// Philox4x32-10 of counter c with key (k0, k1).
__device__ __forceinline__ Words philox4x32_10(Words c, uint32_t k0, uint32_t k1)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.w[0]), lo0 = 0xD2511F53u * c.w[0];
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.w[2]), lo1 = 0xCD9E8D57u * c.w[2];
        c = Words{{hi1 ^ c.w[1] ^ k0, lo1, hi0 ^ c.w[3] ^ k1, lo0}};
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ float to_uniform_f(uint32_t w)
{
    return ((float)(w >> 8) + 0.5f) * 0x1p-24f;
}

// ln k! for integer k >= 0: a table below 10, else the Stirling series
// (k + 1/2) ln(k + 1) - (k + 1) + ln(2 pi)/2 + 1/(12 (k+1)) - 1/(360 (k+1)^3)
// for ln Gamma(k + 1), good to 1e-10 there.  Every operation rounded on its
// own, in float or in double.
__device__ __forceinline__ double log_factorial_table(int i)
{
    return i <= 1 ? 0.0 : i == 2 ? 0.6931471805599453 : i == 3 ? 1.791759469228055
         : i == 4 ? 3.1780538303479458 : i == 5 ? 4.787491742782046 : i == 6 ? 6.579251212010101
         : i == 7 ? 8.525161361065415 : i == 8 ? 10.60460290274525 : 12.801827480081469;
}
__device__ __forceinline__ float log_factorial_f(float k)
{
    if (k < 10.f) return (float)log_factorial_table((int)k);
    const float x = __fadd_rn(k, 1.0f), rx = __fdiv_rn(1.0f, x);
    const float corr = __fmul_rn(rx, __fadd_rn(0.0833333333f, -__fmul_rn(__fmul_rn(rx, rx), 0.00277777778f)));
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(__fadd_rn(k, 0.5f), logf(x)), -x), 0.918938533f), corr);
}
__device__ __forceinline__ double log_factorial_d(double k)
{
    if (k < 10.0) return log_factorial_table((int)k);
    const double x = __dadd_rn(k, 1.0), rx = __ddiv_rn(1.0, x);
    const double corr = __dmul_rn(rx, __dadd_rn(0.083333333333333333,
                                                -__dmul_rn(__dmul_rn(rx, rx), 0.0027777777777777778)));
    return __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(__dadd_rn(k, 0.5), log(x)), -x), 0.9189385332046728),
                     corr);
}

// PTRS's exact acceptance test,
//   log(v invalpha / (a / us^2 + b)) <= -lam + k log lam - ln k!,
// in float while its terms stay small, else in double.
__device__ __noinline__ bool accept_exactly(float lf, float a, float b, float invalpha, float us,
                                            float v, float k)
{
    if (lf < 64.f) {
        const float lhs = __fadd_rn(__fadd_rn(logf(v), logf(invalpha)),
                                    -logf(__fadd_rn(__fdiv_rn(a, __fmul_rn(us, us)), b)));
        const float rhs = __fadd_rn(__fadd_rn(-lf, __fmul_rn(k, logf(lf))), -log_factorial_f(k));
        return lhs <= rhs;
    }
    const double usd = us, kd = k, ld = lf;
    const double lhs = __dadd_rn(__dadd_rn(log((double)v), log((double)invalpha)),
                                 -log(__dadd_rn(__ddiv_rn((double)a, __dmul_rn(usd, usd)), (double)b)));
    const double rhs = __dadd_rn(__dadd_rn(-ld, __dmul_rn(kd, log(ld))), -log_factorial_d(kd));
    return lhs <= rhs;
}

// The same decision, by an FP32 estimate of both sides where it is clear.  With
// m = k + 1, t = (m - lam) / lam and L = log(1 + t) the right side is
//   lam (t - (1 + t) L) + (L - log lam) / 2 - ln(2 pi) / 2 - 1/(12 m) + 1/(360 m^3)
// (Stirling's series for ln k!), whose terms are no larger than the result:
// t - (1 + t) L is summed as its power series for |t| < 1/4.  The estimate, and
// below lam = 64 the float test itself, are off by less than a third of `sure` for
// every lam in 10..1e7 (3 10^7 random attempts against FP64); 0.15 % of the
// tests are closer than that and are evaluated exactly.  The FP64 logarithms (1/64
// of the FP32 rate) of every attempt at lam >= 64 bound the generator: 200 000
// 11x11 sCMOS ADU ROIs 5913 us with them, 773 us so, every draw the same.
__device__ __forceinline__ bool accept(float lf, float rl, float half_log_lam, float a, float b,
                                       float invalpha, float us, float v, float k)
{
    const float m = k + 1.0f, t = (m - lf) * rl;
    const float L = log_approx(m * rl);
    float phi;
    const bool near = fabsf(t) < 0.25f;
    if (near) {
        float c = 1.0f / 156.0f;
#pragma unroll
        for (int n = 12; n >= 2; n--) c = fmaf(-t, c, 1.0f / (float)(n * (n - 1)));
        phi = -(t * t) * c;
    } else {
        phi = fmaf(-(1.0f + t), L, t);
    }
    const float rm = rcp_approx(m);
    const float rhs = fmaf(lf, phi, 0.5f * L - half_log_lam - 0.918938533f) -
                      rm * fmaf(-rm * rm, 0.00277777778f, 0.0833333333f);
    const float lhs = log_approx(v * invalpha * rcp_approx(fmaf(a, rcp_approx(us * us), b)));
    const float diff = lhs - rhs;
    const float sure = (lf < 64.f ? 5e-4f : 5e-5f) + (near ? 4e-6f : 4e-5f) * fabsf(rhs);
    if (k >= 3.f && fabsf(diff) > sure) return diff < 0.f;  // (NaN: exactly)
    return accept_exactly(lf, a, b, invalpha, us, v, k);
}

// Poisson(lf) for 0 < lf < 10 by inversion from the pixel's first word.  rk[k] is
// 1/k to nearest: q = lf rk, corrected by its residual, is lf / k to nearest
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990; checked for every mantissa and k = 1..64).
constexpr int kRecips = 65;
__device__ __forceinline__ float poisson_inversion(float lf, uint32_t word, const float *rk)
{
    const float u = to_uniform_f(word);
    float p = expf(-lf), f = p;
    int k = 0;
    while (u > f && k < 1000) {
        k++;
        const float kf = (float)k;
        float q;
        if (k < kRecips) {
            const float r = rk[k];
            q = __fmul_rn(lf, r);
            q = fmaf(fmaf(-kf, q, lf), r, q);
        } else {
            q = __fdiv_rn(lf, kf);
        }
        p = __fmul_rn(p, q);
        f = __fadd_rn(f, p);
    }
    return (float)k;
}

// One PTRS attempt for Poisson(lf), lf >= 10, from two words of the pixel's
// counter blocks: whether it is accepted, and the count.
__device__ __forceinline__ bool poisson_attempt(float lf, uint32_t wu, uint32_t wv, float &k)
{
    const float slam = __fsqrt_rn(lf);
    const float b = __fadd_rn(0.931f, __fmul_rn(2.53f, slam));
    const float a = __fadd_rn(-0.059f, __fmul_rn(0.02483f, b));
    const float vr = __fadd_rn(0.9277f, -__fdiv_rn(3.6224f, __fadd_rn(b, -2.0f)));
    const float u = __fadd_rn(to_uniform_f(wu), -0.5f);
    const float v = to_uniform_f(wv);
    const float us = __fadd_rn(0.5f, -fabsf(u));
    k = floorf(__fadd_rn(__fadd_rn(__fmul_rn(__fadd_rn(__fdiv_rn(__fmul_rn(2.0f, a), us), b), u), lf),
                         0.43f));
    if (us >= 0.07f && v <= vr) return true;
    if (k < 0.f || (us < 0.013f && v > us)) return false;
    const float invalpha = __fadd_rn(1.1239f, __fdiv_rn(1.1328f, __fadd_rn(b, -3.4f)));
    return accept(lf, rcp_approx(lf), 0.5f * log_approx(lf), a, b, invalpha, us, v, k);
}

// erf-integrated 1-D Gaussian of pixel t (1-based) around c with width s.
__device__ __forceinline__ float integral_1d(int t, float c, float s)
{
    const float k = __fdiv_rn(1.0f, __fmul_rn(1.41421356f, s));
    const float d = __fadd_rn((float)t, -c);
    return __fmul_rn(0.5f, __fadd_rn(erff(__fmul_rn(__fadd_rn(d, 0.5f), k)),
                                     -erff(__fmul_rn(__fadd_rn(d, -0.5f), k))));
}

__device__ __forceinline__ float astig_width(float s0, float u, float a, float b)
{
    const float u2 = __fmul_rn(u, u);
    return __fmul_rn(s0, __fsqrt_rn(__fadd_rn(__fadd_rn(__fadd_rn(1.0f, u2), __fmul_rn(a, __fmul_rn(u2, u))),
                                              __fmul_rn(b, __fmul_rn(u2, u2)))));
}

struct SimArgs {
    int model, box, camera, P;
    float psf[8];
    const float *truth;
    const int32_t *xc, *yc;
    int64_t n;
    uint32_t k0, k1;
    const float *var, *gain, *offset;
    int32_t ny, nx;
    float *out;
    unsigned long long *bad;
};

// Append e to a list of `count` entries (growing up from list[0] with dir 1, down
// from list[0] with dir -1) where `add`; one counter update per warp.
__device__ __forceinline__ void push(bool add, int e, uint16_t *list, int dir, int *count)
{
    const unsigned m = __activemask(), who = __ballot_sync(m, add);
    if (who == 0) return;
    const int lane = threadIdx.x & 31, leader = __ffs(who) - 1;
    int at = 0;
    if (lane == leader) at = atomicAdd(count, __popc(who));
    at = __shfl_sync(m, at, leader);
    if (add) list[dir * (at + __popc(who & ((1u << lane) - 1u)))] = (uint16_t)e;
}

// A block makes whole ROIs, up to kSimPixels pixels.  A
// pixel's cost depends on its rate and on how many attempts its draw takes, so
// that a warp that drew its 32 pixels one by one waited for the slowest
// branch and the longest rejection run among them.  The block therefore sorts
// its pixels into two lists, rates below 10 (inversion) and from 10 on (PTRS),
// works each list off with full warps, and gives the rejected attempts of a
// round (a quarter) to full warps again in the next, twice; the few pixels left
// then are drawn to the end by a thread each.  200 000 11x11 sCMOS ADU
// ROIs: 773 -> 621 us, every draw the same.  (Bound: issue, 65 % of the slots busy, at
// about 700 instructions per pixel and lane, two Philox blocks among them.)
__global__ void __launch_bounds__(kSimThreads, 5) simulate_kernel(const SimArgs a, int rois_per_block)
{
    __shared__ float s_ax[kSimMaxRois][2][kSimMaxBox];  // [roi][x, y][pixel]
    __shared__ float s_n[kSimMaxRois], s_bg[kSimMaxRois];
    __shared__ long long s_base[kSimMaxRois];  // map offset of the ROI's first pixel; -1: bad
    __shared__ float s_val[kSimPixels];        // a pixel's rate, then its count
    // pixels still to draw: rates from 10 on at the front of a round's list, and
    // in the first round's, rates below 10 at its end
    __shared__ uint16_t s_list[2][kSimPixels];
    __shared__ int s_small, s_large[2];
    __shared__ float s_rk[kRecips];
    const int box = a.box, b2 = box * box;
    const int64_t k0 = (int64_t)blockIdx.x * rois_per_block;
    const int64_t left = a.n - k0;
    const int nk = left < rois_per_block ? (int)left : rois_per_block;
    if (nk <= 0) return;
    // per ROI: photons, background and (sCMOS) the map offset
    for (int q = threadIdx.x; q < nk; q += blockDim.x) {
        const float *th = a.truth + (int64_t)a.P * (k0 + q);
        const int in = a.model == 3 ? 3 : 2, ib = a.model == 3 ? 4 : 3;
        s_n[q] = th[in];
        s_bg[q] = th[ib];
        long long base = 0;
        if (a.camera != GMLE_CAMERA_POISSON) {
            const int32_t x0 = a.xc[k0 + q], y0 = a.yc[k0 + q];
            const bool ok = x0 >= 1 && y0 >= 1 && (int64_t)x0 + box - 1 <= a.nx &&
                            (int64_t)y0 + box - 1 <= a.ny;
            if (!ok) atomicAdd(a.bad, 1ull);
            base = ok ? (long long)(y0 - 1) + (long long)a.ny * (x0 - 1) : -1;
        }
        s_base[q] = base;
    }
    // axis tables: entry (roi, axis, pixel index)
    for (int e = threadIdx.x; e < nk * 2 * box; e += blockDim.x) {
        const int q = e / (2 * box), r = e - q * 2 * box, ax = r / box, t = r - ax * box;
        const float *th = a.truth + (int64_t)a.P * (k0 + q);
        const float c = ax == 0 ? th[0] : th[1];
        float s;
        if (a.model == 0) {
            s = a.psf[0];
        } else if (a.model == 1) {
            s = th[4];
        } else if (a.model == 2) {
            s = ax == 0 ? th[4] : th[5];
        } else {
            const float z = th[2], gam = a.psf[6], d = a.psf[7];
            s = ax == 0 ? astig_width(a.psf[0], __fdiv_rn(__fadd_rn(z, -gam), d), a.psf[2], a.psf[4])
                        : astig_width(a.psf[1], __fdiv_rn(__fadd_rn(z, gam), d), a.psf[3], a.psf[5]);
        }
        s_ax[q][ax][t] = integral_1d(t + 1, c, s);
    }
    for (int k = threadIdx.x; k < kRecips; k += blockDim.x) s_rk[k] = __fdiv_rn(1.0f, (float)k);
    if (threadIdx.x == 0) s_small = s_large[0] = s_large[1] = 0;
    __syncthreads();

    const float qnan = __int_as_float(0x7fc00000);
    const int cnt = nk * b2;
    // e / b2 and p / box for the block's pixel numbers (below 2^11) by
    // multiplication: exact while e b2 and p box stay below 2^32
    const uint32_t m_b2 = 0xffffffffu / (uint32_t)b2 + 1u, m_box = 0xffffffffu / (uint32_t)box + 1u;
    auto roi_of = [&](int e) { return b2 == 1 ? e : (int)__umulhi((uint32_t)e, m_b2); };
    auto col_of = [&](int p) { return box == 1 ? p : (int)__umulhi((uint32_t)p, m_box); };
    auto words = [&](int e, uint32_t block) {
        const int q = roi_of(e);
        const int64_t k = k0 + q;
        return philox4x32_10(Words{{(uint32_t)(e - q * b2), (uint32_t)k,
                                    (uint32_t)((uint64_t)k >> 32), block}}, a.k0, a.k1);
    };
    // rates: mu = bg + N (psf_y[i] psf_x[j])
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
        const int q = roi_of(e), p = e - q * b2, j = col_of(p), i = p - j * box;
        const float mu = __fadd_rn(s_bg[q], __fmul_rn(s_n[q], __fmul_rn(s_ax[q][1][i], s_ax[q][0][j])));
        const bool draw = s_base[q] >= 0 && mu > 0.f;
        s_val[e] = draw ? mu : 0.f;
        push(draw && mu < 10.f, e, &s_list[0][kSimPixels - 1], -1, &s_small);
        push(draw && !(mu < 10.f), e, &s_list[0][0], 1, &s_large[0]);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < s_small; t += blockDim.x) {
        const int e = s_list[0][kSimPixels - 1 - t];
        s_val[e] = poisson_inversion(s_val[e], words(e, 0u).w[0], s_rk);
    }
    // attempt `it` of pixel e: two words per attempt, two attempts per counter
    // block; the 10 000th is taken as it comes
    auto attempt = [&](int e, int it) {
        const Words w = words(e, (uint32_t)it >> 1);
        const float lf = s_val[e];
        float k;
        bool ok = poisson_attempt(lf, it & 1 ? w.w[2] : w.w[0], it & 1 ? w.w[3] : w.w[1], k);
        if (it == 9999 && !ok) {
            k = floorf(lf);
            ok = true;
        }
        if (ok) s_val[e] = k;
        return ok;
    };
    constexpr int kRounds = 2;
#pragma unroll 1
    for (int it = 0; it < kRounds; it++) {
        const int cur = it & 1, n = s_large[cur];
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int e = s_list[cur][t];
            push(!attempt(e, it), e, &s_list[cur ^ 1][0], 1, &s_large[cur ^ 1]);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_large[cur] = 0;
        __syncthreads();
    }
    for (int t = threadIdx.x; t < s_large[kRounds & 1]; t += blockDim.x) {
        const int e = s_list[kRounds & 1][t];
#pragma unroll 1
        for (int it = kRounds; !attempt(e, it); it++) {}
    }
    __syncthreads();
    // read noise and camera, written coalesced
    float *dst = a.out + k0 * b2;
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
        const int q = roi_of(e), p = e - q * b2;
        const long long base = s_base[q];
        float v = s_val[e];
        if (base < 0) {
            v = qnan;
        } else if (a.camera != GMLE_CAMERA_POISSON) {
            const int j = col_of(p), i = p - j * box;
            const long long m = base + i + (long long)a.ny * j;
            const Words w = words(e, kNoiseBlock);
            const float u1 = to_uniform_f(w.w[0]), u2 = to_uniform_f(w.w[1]);
            const float z = __fmul_rn(__fsqrt_rn(__fmul_rn(-2.0f, logf(u1))),
                                      cosf(__fmul_rn(6.28318530717958648f, u2)));
            v = __fadd_rn(v, __fmul_rn(z, __fsqrt_rn(a.var[m])));
            if (a.camera == GMLE_CAMERA_SCMOS_ADU)
                v = __fadd_rn(__fdiv_rn(v, a.gain[m]), a.offset[m]);
        }
        dst[e] = v;
    }
}

}  // namespace

extern "C" gmle_status gmle_simulate_device(gmle_ctx *ctx, const gmle_fit_desc *d,
                                            const float *d_truth, const int32_t *d_x_corners,
                                            const int32_t *d_y_corners, int64_t n, uint64_t seed,
                                            float *d_rois, void *stream)
{
    if (!ctx) return GMLE_INVALID_ARG;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (!d) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "desc is NULL");
    if (d->model < 0 || d->model > 3)
        return gmle_rt::fail(ctx, GMLE_UNSUPPORTED_MODEL, "unknown model id %d", d->model);
    if (d->box < 1 || d->box > kSimMaxBox)
        return gmle_rt::fail(ctx, GMLE_UNSUPPORTED_BOX, "box %d outside 1..%d", d->box, kSimMaxBox);
    if (d->camera < 0 || d->camera > 2)
        return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "unknown camera id %d", d->camera);
    if (n < 0) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "n < 0");
    if (n == 0) return GMLE_OK;
    if (!d_truth || !d_rois) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "truth and output are required");
    if (d->camera != GMLE_CAMERA_POISSON) {
        if (!d_x_corners || !d_y_corners)
            return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "sCMOS ROIs need their corners");
        if (!ctx->d_var) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "sCMOS ROIs without calibration maps");
        if (d->camera == GMLE_CAMERA_SCMOS_ADU && (!ctx->d_gain || !ctx->d_offset))
            return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "ADU ROIs need gain and offset maps");
    }
    SimArgs a{};
    a.model = d->model;
    a.box = d->box;
    a.camera = d->camera;
    a.P = gmle_rt::nparams(d->model);
    std::copy(d->psf, d->psf + 8, a.psf);
    a.truth = d_truth;
    a.xc = d_x_corners;
    a.yc = d_y_corners;
    a.n = n;
    a.k0 = (uint32_t)seed;
    a.k1 = (uint32_t)(seed >> 32);
    a.var = ctx->d_var;
    a.gain = ctx->d_gain;
    a.offset = ctx->d_offset;
    a.ny = ctx->ny;
    a.nx = ctx->nx;
    a.out = d_rois;
    a.bad = ctx->d_bad;
    cudaSetDevice(ctx->device);
    const int rpb = std::min(kSimMaxRois, std::max(1, kSimPixels / (d->box * d->box)));
    const int64_t blocks = (n + rpb - 1) / rpb;
    if (blocks > 0x7fffffffLL) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "too many ROIs");
    ctx->launches++;
    simulate_kernel<<<(unsigned)blocks, kSimThreads, 0, static_cast<cudaStream_t>(stream)>>>(a, rpb);
    GMLE_CK(cudaGetLastError(), "ROI generator launch");
    return GMLE_OK;
}
