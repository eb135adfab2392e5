// gmle_pvalue.cu - goodness-of-fit p-values of the fits, on the device.
//
// The reference computes them on the host after every fit, one ROI at a time
// (src/interface.jl:265-275, :459-468):
//     chi2 = -2 llr            (Float32)
//     p    = 1 - Float32(cdf(Chisq(df), chi2)),   df = box^2 - P.
// cdf(Chisq(df), x) is the regularised lower incomplete gamma function
// P(a, x/2) with a = df/2, evaluated by Distributions.jl in Float64 (the Float32
// chi2 is promoted and halved exactly).  A launch has one a, so P(a, .) is one
// smooth function of x there:
//
// * a >= 8 (boxes of 5 pixels and more): every block builds a table of Taylor
//   polynomials of P at nodes k D in FP64 (one node per thread), and each ROI
//   costs one lookup and a polynomial of degree 10 in FP32 whose leading terms
//   are kept in pairs of floats.  D is a power of two, so that x / D and its
//   distance from the nearest node are exact.
// * smaller a: P(a, x) in FP64 per ROI by the classical scheme (Numerical
//   Recipes, 2nd ed., sec. 6.2; Abramowitz & Stegun 6.5.29 and 6.5.31): the
//   power series
//     P = x^a e^-x / Gamma(a) * sum_n x^n / (a (a+1) ... (a+n))      (x < a + 1)
//   and otherwise the continued fraction of Q = 1 - P, evaluated with the
//   modified Lentz method, both up to a relative term below 1e-16 or 1000 terms.
//
// The p-value is rounded to Float32 as the reference does; the table's P is
// within 1e-9 of the FP64 one, so that at most 0.5 % of the rounded values differ,
// by one ulp of 1 (df 16..4092; the root mean square error against 64 bits is
// the rounding's, 1.7e-8, for both).
//
// Bound: the per-ROI series were bound by the FP64 pipe (about 60 terms, each
// with an FP64 division, at 1/64 of the FP32 rate); with the table the launch is
// its build (about 200 FP64 instructions per warp of nodes) and memory.  ROI cut,
// fit and p-values of 200 000 9x9 ROIs (df 76): 1176 us with the series for every
// ROI, 476 us with the table.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "gmle_internal.h"

namespace {

__device__ double gamma_p(double a, double x)
{
    if (isnan(x)) return x;
    if (x <= 0.0) return 0.0;  // Distributions clamps x at 0: P(a, 0) = 0
    if (isinf(x)) return 1.0;
    const double log_pre = a * log(x) - x - lgamma(a);  // log(x^a e^-x / Gamma(a))
    if (x < a + 1.0) {
        double ap = a, term = 1.0 / a, sum = term;
        for (int n = 0; n < 1000; n++) {
            ap += 1.0;
            term *= x / ap;
            sum += term;
            if (fabs(term) < fabs(sum) * 1e-16) break;
        }
        return sum * exp(log_pre);
    }
    const double tiny = 1e-300;
    double b = x + 1.0 - a, c = 1.0 / tiny, d = 1.0 / b, h = d;
    for (int i = 1; i < 1000; i++) {
        const double an = -i * (i - a);
        b += 2.0;
        d = an * d + b;
        if (fabs(d) < tiny) d = tiny;
        c = b + an / c;
        if (fabs(c) < tiny) c = tiny;
        d = 1.0 / d;
        const double del = d * c;
        h *= del;
        if (fabs(del - 1.0) < 1e-16) break;
    }
    return 1.0 - exp(log_pre) * h;
}

__global__ void pvalue_kernel(const float *__restrict__ llr, int64_t n, double a,
                              float *__restrict__ pvalues)
{
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const float chi2 = -2.0f * llr[k];
        pvalues[k] = 1.0f - (float)gamma_p(a, 0.5 * (double)chi2);
    }
}

// ---- P(a, .) from a table ------------------------------------------------------

constexpr int kPvThreads = 512;
constexpr int kPvNodes = 160;      // at most 129 are used (a = 15.5)
constexpr int kPvTerms = 10;       // polynomial of degree 10 in (x - node) / D
constexpr double kMinTableA = 8.0;

struct PvTable {
    double a, lgamma_a;
    double D;   // node spacing, a power of two: sigma/4..sigma/2 (sigma^2 = a), half that below a = 16
    int k0, nodes;  // nodes (k0 .. k0 + nodes - 1) D; P < 1e-12 before them, 1 - P < 1e-12 after
};

// Node range by the Wilson-Hilferty cube-root normal approximation at +-7.2
// standard deviations.
PvTable make_pv_table(int32_t df)
{
    PvTable t;
    t.a = 0.5 * (double)df;
    int sign;
    t.lgamma_a = ::lgamma_r(t.a, &sign);  // (lgamma writes a global)
    const double sigma = std::sqrt(t.a);
    t.D = std::exp2(std::floor(std::log2(sigma / (t.a >= 16.0 ? 2.0 : 4.0))));
    auto wh = [&](double z) {
        const double r = std::max(0.0, 1.0 - 1.0 / (9.0 * t.a) + z / (3.0 * sigma));
        return t.a * r * r * r;
    };
    t.k0 = (int)std::floor(wh(-7.2) / t.D);
    t.nodes = std::min(kPvNodes, (int)std::ceil(wh(7.2) / t.D) + 2 - t.k0);
    return t;
}

__global__ void __launch_bounds__(kPvThreads)
    pvalue_table_kernel(const float *__restrict__ llr, int64_t n, const PvTable t,
                        float *__restrict__ pvalues)
{
    // P(node) and the first coefficient as pairs of floats, then coefficients 1..9
    __shared__ float s_ph[kPvNodes], s_pl[kPvNodes], s_cl[kPvNodes], s_c[kPvTerms][kPvNodes];
    __shared__ double s_inc[kPvNodes];  // integral of the density over a node's cell
    const int k = threadIdx.x;
    double left = 0.0;                   // and over its lower half
    if (k < kPvNodes) {
        double inc = 0.0;
        if (k < t.nodes) {
            // the density f at the node and its Taylor coefficients G_n D^-n:
            // x f' = (a - 1 - x) f gives G_{n+1} from G_n and G_{n-1}
            const double x = (t.k0 + k) * t.D, am = t.a - 1.0;
            const double fD = x > 0.0 ? exp(am * log(x) - x - t.lgamma_a) * t.D : 0.0;
            const double r = x > 0.0 ? t.D / x : 0.0;
            double g = 1.0, prev = 0.0, half = 0.5;
#pragma unroll
            for (int m = 0; m <= 14; m++) {
                const double c = fD * g * (1.0 / (m + 1));
                if (m < kPvTerms) s_c[m][k] = (float)c;
                if (m == 0) s_cl[k] = (float)(c - (double)(float)c);
                if (m & 1) {
                    left -= c * half;
                } else {
                    left += c * half;
                    inc += 2.0 * c * half;
                }
                half *= 0.5;
                const double next = ((am - x - m) * g - t.D * prev) * r * (1.0 / (m + 1));
                prev = g;
                g = next;
            }
        }
        s_inc[k] = inc;
    }
    __syncthreads();
    if (k < 32) {  // exclusive sums of the cells' integrals
        constexpr int kPer = kPvNodes / 32;
        double v[kPer], sum = 0.0;
#pragma unroll
        for (int i = 0; i < kPer; i++) {
            v[i] = sum;
            sum += s_inc[kPer * k + i];
        }
        double before = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double o = __shfl_up_sync(0xffffffffu, before, off);
            if (k >= off) before += o;
        }
        before -= sum;
#pragma unroll
        for (int i = 0; i < kPer; i++) s_inc[kPer * k + i] = before + v[i];
    }
    __syncthreads();
    if (k < t.nodes) {
        const double p = s_inc[k] + left;
        s_ph[k] = (float)p;
        s_pl[k] = (float)(p - (double)(float)p);
    }
    __syncthreads();
    const float rD = (float)(1.0 / t.D);
    for (int64_t i = (int64_t)blockIdx.x * kPvThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kPvThreads) {
        const float chi2 = -2.0f * llr[i];
        const float y = (0.5f * chi2) * rD;  // x / D, exact
        float P;
        if (!(y == y)) {
            P = y;  // NaN
        } else {
            // rint(y) - k0, saturated by the conversion; x <= 0 is before the nodes
            const float kf = rintf(y);
            const int q = y <= 0.f ? -1 : kf < 2e9f ? (int)kf - t.k0 : t.nodes;
            if (q < 0) {
                P = 0.0f;
            } else if (q >= t.nodes) {
                P = 1.0f;
            } else {
                const float h = y - kf;
                float c = s_c[kPvTerms - 1][q];
#pragma unroll
                for (int m = kPvTerms - 2; m >= 1; m--) c = fmaf(c, h, s_c[m][q]);
                const float c0 = s_c[0][q];
                const float hi = __fmul_rn(c0, h);          // c0 h = hi + lo exactly
                const float lo = fmaf(c0, h, -hi);
                const float ph = s_ph[q];
                const float s = __fadd_rn(ph, hi);           // ph + hi = s + e exactly
                const float b = __fadd_rn(s, -ph);
                const float e = __fadd_rn(__fadd_rn(ph, -__fadd_rn(s, -b)), __fadd_rn(hi, -b));
                P = s + (e + (lo + (s_pl[q] + fmaf(s_cl[q], h, c * h * h))));
            }
        }
        pvalues[i] = 1.0f - P;
    }
}

gmle_status launch_pvalues(gmle_ctx *ctx, const float *d_llr, int64_t n, int32_t df,
                           float *d_pvalues, cudaStream_t s)
{
    if (n <= 0) return GMLE_OK;
    ctx->launches++;
    if (0.5 * (double)df >= kMinTableA) {
        // one block per SM: every block builds the table
        const int64_t blocks = std::min<int64_t>((n + kPvThreads - 1) / kPvThreads, ctx->num_sms);
        pvalue_table_kernel<<<(unsigned)blocks, kPvThreads, 0, s>>>(d_llr, n, make_pv_table(df),
                                                                    d_pvalues);
    } else {
        const int threads = 256;
        const int64_t blocks = std::min<int64_t>((n + threads - 1) / threads,
                                                 (int64_t)ctx->num_sms * 8);
        pvalue_kernel<<<(unsigned)blocks, threads, 0, s>>>(d_llr, n, 0.5 * (double)df, d_pvalues);
    }
    GMLE_CK(cudaGetLastError(), "p-value kernel launch");
    return GMLE_OK;
}

gmle_status check_pvalue_args(gmle_ctx *ctx, const float *llr, int64_t n, int32_t df,
                              const float *pvalues)
{
    if (n < 0) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "n < 0");
    if (n > 0 && (!llr || !pvalues))
        return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "llr and pvalues are required");
    if (df <= 0) return gmle_rt::fail(ctx, GMLE_INVALID_ARG, "degrees of freedom must be > 0");
    return GMLE_OK;
}

}  // namespace

extern "C" gmle_status gmle_pvalues_device(gmle_ctx *ctx, const float *d_llr, int64_t n,
                                           int32_t df, float *d_pvalues, void *stream)
{
    if (!ctx) return GMLE_INVALID_ARG;
    std::lock_guard<std::mutex> lk(ctx->mu);
    gmle_status st = check_pvalue_args(ctx, d_llr, n, df, d_pvalues);
    if (st != GMLE_OK) return st;
    cudaSetDevice(ctx->device);
    return launch_pvalues(ctx, d_llr, n, df, d_pvalues, static_cast<cudaStream_t>(stream));
}

extern "C" gmle_status gmle_pvalues(gmle_ctx *ctx, const float *llr, int64_t n, int32_t df,
                                    float *pvalues)
{
    if (!ctx) return GMLE_INVALID_ARG;
    std::lock_guard<std::mutex> lk(ctx->mu);
    gmle_status st = check_pvalue_args(ctx, llr, n, df, pvalues);
    if (st != GMLE_OK || n == 0) return st;
    cudaSetDevice(ctx->device);
    if (ctx->pv_cap < n) {
        cudaFree(ctx->d_pv);
        ctx->d_pv = nullptr;
        ctx->pv_cap = 0;
        GMLE_CK(cudaMalloc(&ctx->d_pv, 2 * sizeof(float) * (size_t)n), "cudaMalloc(p-values)");
        ctx->pv_cap = n;
    }
    float *d_in = ctx->d_pv, *d_out = ctx->d_pv + n;
    cudaStream_t s = ctx->s_fit;
    GMLE_CK(cudaMemcpyAsync(d_in, llr, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, s),
            "H2D llr");
    st = launch_pvalues(ctx, d_in, n, df, d_out, s);
    if (st != GMLE_OK) return st;
    GMLE_CK(cudaMemcpyAsync(pvalues, d_out, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, s),
            "D2H p-values");
    GMLE_CK(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    return GMLE_OK;
}
