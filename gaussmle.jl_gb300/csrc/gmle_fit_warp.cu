// gmle_fit_warp.cu - the fit with one warp per ROI (the iteration of
// fit_kernel_r1, src/unified_kernel.jl:285-434, with the box a run-time value).
// Compiled once per (model, camera family) with -DGMLE_MODEL=0..3
// -DGMLE_SCMOS=0|1.
//
// It fits the ROIs beyond 16 pixels (17..64), whose pixels and tables exceed
// what one thread can hold, and small batches of the smaller boxes, whose time is
// the latency of a fit's dependent passes (default_tuning draws the line).
//
// A warp's lanes are a grid of 8 column by 4 row classes: lane (rx, ry) owns
// the pixels of columns rx, rx + 8, ... and rows ry, ry + 4, ..., at most
// RMAX rows.  Up to 32 pixels per lane (boxes to 32) stay in its registers for
// the whole fit; larger boxes read them from shared memory.  Per pass:
//  * lanes 0-15 set up the x axis, lanes 16-31 the y axis;
//  * every lane evaluates one pixel edge (one erf, one exp; up to 15 pixels both
//    axes at once); table entries are differences with the neighbouring lane's,
//    written to shared memory;
//  * every lane sums its pixels and applies the column and row terms, which
//    are linear in those sums, to its partial sums;
//  * the P (gradient, Hessian) pairs are summed and scattered over the lanes,
//    so that one lane per parameter divides and clamps, and the new parameters
//    are handed back by shuffles.
// The Fisher matrix (double-float) is summed and scattered the same way, and
// one thread per ROI of the block inverts it in FP64: a warp's FP64
// instruction takes as long for one lane as for all, so the block's ROIs
// share them.
//
// Bound: instruction issue and, at 16 resident warps per SM (128 registers for
// 21x21 sCMOS), the latency of a pass (no contraction, operands in registers).
// 12 000 astigmatic 21x21 sCMOS ADU ROIs: 2281 us with one thread per ROI and
// the pixels and tables in shared memory (one block of 32 threads per SM),
// 270 us so.  200 XYNB 11x11 ROIs: 45 us with four lanes per ROI, 20.5 us so.
#if !defined(GMLE_MODEL) || !defined(GMLE_SCMOS)
#error "compile with -DGMLE_MODEL=<0..3> -DGMLE_SCMOS=<0|1>"
#endif

#include <cuda_runtime.h>

#include "gmle_fit_kernel.cuh"
#include "gmle_warp.h"

namespace gmle {

namespace {

constexpr int kCols = 8, kRows = 4;  // the lane grid

// Rows per lane, RMAX = ceil(box / 4), of the compiled kernels; the row slots
// from RFULL on may lie outside the smallest box of their range.
template <int RMAX> struct WarpShape {
    static constexpr int TS = 4 * RMAX;                   // floats between two tables
    static constexpr bool REG = RMAX <= 8;                // pixels in registers
    static constexpr int CMAX = REG ? (RMAX + 1) / 2 : 1;  // columns per lane, in registers
    static constexpr int RFULL = RMAX == 2 ? 0 : RMAX == 12 ? 8 : RMAX == 16 ? 12 : RMAX - 1;
    // columns that lie inside every box of the range (registers only)
    __host__ __device__ static constexpr int cfull()
    {
        return RMAX == 2 ? 0 : (4 * (RMAX - 1) + 1) / kCols;
    }
};
template <int P> struct RoiResult {  // what the inversion needs, per ROI of a block
    double F[P * (P + 1) / 2];
    float th[P];
    float llr;
    int ok;
};

// The sums over the warp's lanes of M units of K values, scattered: on return
// v[0] holds the sum of unit `unit`, or of padding (lane_of_unit names a lane that
// holds a given unit).
template <int M, int BIT, int U, int K>
__device__ __forceinline__ void scatter_sum(float (&v)[U][K], int lane, int &unit)
{
    if constexpr (BIT > 0) {
        constexpr int H = (M + 1) / 2;
        if constexpr (M == 1) {
#pragma unroll
            for (int k = 0; k < K; k++) v[0][k] += __shfl_xor_sync(0xffffffffu, v[0][k], BIT);
        } else {
            const bool up = lane & BIT;
#pragma unroll
            for (int i = 0; i < H; i++)
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const float hi = H + i < M ? v[H + i][k] : 0.f;
                    const float keep = up ? hi : v[i][k], send = up ? v[i][k] : hi;
                    v[i][k] = keep + __shfl_xor_sync(0xffffffffu, send, BIT);
                }
            unit += up ? H : 0;
        }
        scatter_sum<H, BIT / 2, U, K>(v, lane, unit);
    }
}
// The same for double-float values; `left` (M on entry) counts the values that
// the lane still holds, padding excluded: <= 0 on return means it holds none.
template <int M, int BIT, int U>
__device__ __forceinline__ void scatter_sum_dd(float (&hi)[U], float (&lo)[U], int lane, int &unit,
                                               int &left)
{
    if constexpr (BIT > 0) {
        constexpr int H = (M + 1) / 2;
        const bool up = M > 1 && (lane & BIT);
#pragma unroll
        for (int i = 0; i < H; i++) {
            const bool has = H + i < M;
            const float h2 = M == 1 ? hi[i] : has ? hi[H + i] : 0.f;
            const float l2 = M == 1 ? lo[i] : has ? lo[H + i] : 0.f;
            const float oh = __shfl_xor_sync(0xffffffffu, up ? hi[i] : h2, BIT);
            const float ol = __shfl_xor_sync(0xffffffffu, up ? lo[i] : l2, BIT);
            const float kh = up ? h2 : hi[i], kl = up ? l2 : lo[i];
            float s, e;
            two_sum(kh, oh, s, e);
            e = __fadd_rn(e, __fadd_rn(kl, ol));
            two_sum(s, e, hi[i], lo[i]);
        }
        if (M > 1) {
            unit += up ? H : 0;
            left = up ? left - H : min(left, H);
        }
        scatter_sum_dd<H, BIT / 2, U>(hi, lo, lane, unit, left);
    }
}
// A lane on which scatter_sum leaves unit k of M.
__host__ __device__ constexpr int lane_of_unit(int k, int m)
{
    int lane = 0;
    for (int bit = 16; bit > 0 && m > 1; bit /= 2) {
        const int h = (m + 1) / 2;
        if (k >= h) { k -= h; lane += bit; }
        m = h;
    }
    return lane;
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Table entries of the pixels whose lower edge is e (0-based pixel e, from the
// lanes' edges e and e + 1): walk_entry's values, at tab + k TS for k = 0..4.
// `width` lanes share an axis, edge index = lane within them.
template <int MODEL, int TS>
__device__ __forceinline__ void warp_entry(int e, const Axis &a, int width, bool keep, float *tab)
{
    constexpr bool SIG = ModelInfo<MODEL>::SIG;
    EdgeWalk w;
    w.pos = (float)e + 0.5f;
    w.g3 = 0.f;
    walk_edge<SIG>(a, w);
    auto diff = [&](float v) { return __shfl_down_sync(0xffffffffu, v, 1, width) - v; };
    const float dh = diff(w.h), df = diff(w.f), dg = diff(w.g);
    const float dg3 = SIG ? diff(w.g3) : 0.f;
    if (keep) {
        tab[e] = fmaxf(dh, 0.0f);
        tab[TS + e] = a.cst * df;
        tab[2 * TS + e] = a.cst2 * dg;
        if (SIG) {
            tab[3 * TS + e] = a.kz * dg;
            tab[4 * TS + e] = fmaf(a.kq3, dg3, a.kq * dg);
        }
    }
}

// The start point's parameters from its sums (total, and weighted by column and
// row; mxx, myy: the astigmatic second moments).
template <int MODEL>
__device__ __forceinline__ void warp_start_xy(const int box, float total, float xw, float yw, float &x,
                                              float &y)
{
    const float centre = (float)((box + 1) / 2.0);
    x = jl_clamp(total > 10.f ? __fdiv_rn(xw, total) : centre, 1.5f, (float)(box - 0.5));
    y = jl_clamp(total > 10.f ? __fdiv_rn(yw, total) : centre, 1.5f, (float)(box - 0.5));
}
template <int MODEL>
__device__ __forceinline__ void warp_start(float x, float y, float total, float bg, float mxx,
                                           float myy, const float *psf,
                                           float (&th)[ModelInfo<MODEL>::P])
{
    using S = Slots<MODEL>;
    th[S::IX] = x;
    th[S::IY] = y;
    th[S::IN] = jl_maxf(total, 100.f);
    th[S::IB] = bg;
    if (MODEL == 1 || MODEL == 2) th[4] = 1.3f;
    if (MODEL == 2) th[ModelInfo<MODEL>::P - 1] = 1.3f;
    if (MODEL == 3) {
        float z = 0.f;
        if (total > 10.f) {
            const float rx = __fdiv_rn(sqrtf(jl_maxf(0.5f, __fdiv_rn(mxx, total))), psf[0]);
            const float ry = __fdiv_rn(sqrtf(jl_maxf(0.5f, __fdiv_rn(myy, total))), psf[1]);
            const float da = __fadd_rn(__fmul_rn(rx, rx), -__fmul_rn(ry, ry));
            z = jl_clamp(__fdiv_rn(__fmul_rn(-da, __fmul_rn(psf[7], psf[7])), __fmul_rn(4.0f, psf[6])),
                         -600.f, 600.f);
        }
        th[2] = z;
    }
}

// The ROI's start point (src/unified_kernel.jl:158-255) with every sum in the
// reference's order (initialize_box), bit for bit.  The lanes write the terms of
// the sums in that order into `scr` (three arrays of warp_scratch(box) floats, 16-byte
// aligned, zeros behind the last term), then add them: every lane the edge pixels,
// lane 0, 1 and 2 the plain, column- and row-weighted sums.
__device__ __forceinline__ float ordered_sum(const float *v, int n4)
{
    float acc = 0.f;
#pragma unroll 4
    for (int q = 0; q < n4; q++) {
        const float4 t = reinterpret_cast<const float4 *>(v)[q];
        acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t.x), t.y), t.z), t.w);
    }
    return acc;
}
template <int MODEL, typename Each>
__device__ __forceinline__ void warp_initialize_exact(const int box, Each each, float *scr, int lane,
                                                      const float *psf,
                                                      float (&th)[ModelInfo<MODEL>::P])
{
    const int B2 = box * box, BP = warp_scratch(box);
    each([&](int j, int i, float d) {  // 4 box - 4 edge pixels, column by column
        const int e = j == 0 ? i : j == box - 1 ? 3 * box - 4 + i : box + 2 * (j - 1) + (i ? 1 : 0);
        if (j == 0 || j == box - 1 || i == 0 || i == box - 1) scr[e] = d;
    });
    __syncwarp();
    const float bg = __fdiv_rn(ordered_sum(scr, box - 1), (float)(4 * box - 4));
    __syncwarp();
    each([&](int j, int i, float d) {
        const float sig = jl_max0(__fadd_rn(d, -bg));
        float *t = scr + i + box * j;
        t[0] = sig;
        t[BP] = __fmul_rn(sig, (float)(j + 1));
        t[2 * BP] = __fmul_rn(sig, (float)(i + 1));
    });
    const int own = min(lane, 2) * BP;
    if (lane < 3)
        for (int p = B2; p < BP; p++) scr[own + p] = 0.f;
    __syncwarp();
    const float acc = ordered_sum(scr + own, BP / 4);
    const float total = __shfl_sync(0xffffffffu, acc, 0);
    float x, y, mxx = 0.f, myy = 0.f;
    warp_start_xy<MODEL>(box, total, __shfl_sync(0xffffffffu, acc, 1),
                         __shfl_sync(0xffffffffu, acc, 2), x, y);
    if (MODEL == 3) {  // lane 0: about x, lane 1: about y
        __syncwarp();
        each([&](int j, int i, float d) {
            const float sig = jl_max0(__fadd_rn(d, -bg));
            const float dx = __fadd_rn((float)(j + 1), -x), dy = __fadd_rn((float)(i + 1), -y);
            float *t = scr + i + box * j;
            t[0] = __fmul_rn(__fmul_rn(sig, dx), dx);
            t[BP] = __fmul_rn(__fmul_rn(sig, dy), dy);
        });
        __syncwarp();
        const float m = ordered_sum(scr + min(lane, 1) * BP, BP / 4);
        mxx = __shfl_sync(0xffffffffu, m, 0);
        myy = __shfl_sync(0xffffffffu, m, 1);
    }
    warp_start<MODEL>(x, y, total, bg, mxx, myy, psf, th);
}

// The ROI's start point from the lanes' pixels, summed over the lanes.
// each(fn) calls fn(column, row, value) (0-based) for each of the lane's pixels.
template <int MODEL, typename Each>
__device__ __forceinline__ void warp_initialize(const int box, Each each, const float *psf,
                                                float (&th)[ModelInfo<MODEL>::P])
{
    float edge = 0.f;
    each([&](int j, int i, float d) {
        if (i == 0 || i == box - 1 || j == 0 || j == box - 1) edge += d;
    });
    const float bg = __fdiv_rn(warp_sum(edge), (float)(4 * box - 4));
    float total = 0.f, xw = 0.f, yw = 0.f;
    each([&](int j, int i, float d) {
        const float sig = jl_max0(d - bg);
        total += sig;
        xw = fmaf(sig, (float)(j + 1), xw);
        yw = fmaf(sig, (float)(i + 1), yw);
    });
    total = warp_sum(total);
    xw = warp_sum(xw);
    yw = warp_sum(yw);
    float x, y, mxx = 0.f, myy = 0.f;
    warp_start_xy<MODEL>(box, total, xw, yw, x, y);
    if (MODEL == 3) {
        each([&](int j, int i, float d) {
            const float sig = jl_max0(d - bg);
            const float dx = (float)(j + 1) - x, dy = (float)(i + 1) - y;
            mxx = fmaf(sig * dx, dx, mxx);
            myy = fmaf(sig * dy, dy, myy);
        });
        mxx = warp_sum(mxx);
        myy = warp_sum(myy);
    }
    warp_start<MODEL>(x, y, total, bg, mxx, myy, psf, th);
}

// Fit ROI `roi` of `a` with the calling warp; its shared memory is at `tab`.
template <int MODEL, bool SCMOS, int RMAX>
__device__ __forceinline__ void fit_roi_warp(const KernelArgs &a, const int box, const int64_t roi,
                                             float *tab, RoiResult<ModelInfo<MODEL>::P> &res)
{
    using W = WarpShape<RMAX>;
    using S = Slots<MODEL>;
    constexpr int P = ModelInfo<MODEL>::P, NF = P * (P + 1) / 2;
    constexpr bool SIG = ModelInfo<MODEL>::SIG;
    constexpr bool CROSS = (MODEL == 1 || MODEL == 3);
    constexpr int NB = SIG ? 4 : 3;
    constexpr int CM = W::CMAX, RM = RMAX, NPR = RM / 2;
    constexpr bool ODD = (RM & 1) != 0;
    constexpr int VN = SCMOS ? CM : 1, VR = SCMOS ? RM : 1;
    const int lane = threadIdx.x & 31;
    const int ry = lane & (kRows - 1), rx = lane / kRows;
    const int B2 = box * box;
    constexpr int TS = W::TS;
    float *const spix = tab + 10 * TS, *const svar = spix + warp_scratch(box);  // (warp_floats)
    for (int e = lane; e < 10 * TS; e += 32) tab[e] = 0.f;  // entries past the box
    bool ok = true;
    long long base = 0;
    if (SCMOS) {
        const int32_t x0 = a.xc[roi], y0 = a.yc[roi];
        ok = corner_inside(x0, y0, box, a.ny, a.nx);
        if (!ok && lane == 0) atomicAdd(a.bad_corners, 1ull);
        base = ok ? (long long)(y0 - 1) + (long long)a.ny * (x0 - 1) : 0;
    }
    // pixel p = i + box j, in electrons ((ADU - offset) * gain,
    // src/camera_models.jl:110-113), and its variance
    const float *src = a.data + roi * B2;
    auto fetch = [&](int j, int i, float &d, float &v) {
        d = __ldg(src + i + box * j);
        v = 0.f;
        if (SCMOS && ok) {
            const long long m = base + i + (long long)a.ny * j;
            v = __ldg(a.var + m);
            if (a.adu) d = __fmul_rn(__fadd_rn(d, -__ldg(a.offset + m)), __ldg(a.gain + m));
        }
    };
    float dp[CM][RM], vp[VN][VR];
    if constexpr (W::REG) {
#pragma unroll
        for (int c = 0; c < CM; c++)
#pragma unroll
            for (int r = 0; r < RM; r++) {
                const int j = rx + kCols * c, i = ry + kRows * r;
                // a slot outside the box: with an infinite variance its
                // likelihood terms are 0
                float d = 0.f, v = INFINITY;
                if (j < box && i < box) fetch(j, i, d, v);
                dp[c][r] = d;
                if (SCMOS) vp[c][r] = v;
            }
    } else {
        for (int p = lane; p < B2; p += 32) {
            const int j = p / box;
            float v;
            fetch(j, p - box * j, spix[p], v);
            if (SCMOS) svar[p] = v;
        }
        __syncwarp();
    }
    auto each = [&](auto fn) {
        if constexpr (W::REG) {
#pragma unroll
            for (int c = 0; c < CM; c++)
#pragma unroll
                for (int r = 0; r < RM; r++) {
                    const int j = rx + kCols * c, i = ry + kRows * r;
                    if (j < box && i < box) fn(j, i, dp[c][r]);
                }
        } else {
            for (int j = rx; j < box; j += kCols)
                for (int i = ry; i < box; i += kRows) fn(j, i, spix[i + box * j]);
        }
    };
    // column j of the lane's pixels
    auto load_column = [&](int j) {
#pragma unroll
        for (int r = 0; r < RM; r++) {
            const int i = ry + kRows * r;
            const bool in = r < W::RFULL || i < box;
            dp[0][r] = in ? spix[i + box * j] : 0.f;
            if (SCMOS) vp[0][r] = in ? svar[i + box * j] : INFINITY;
        }
    };

    float th[P];
    if constexpr (RMAX <= 4) {
        warp_initialize_exact<MODEL>(box, each, spix, lane, a.psf, th);
    } else {
        warp_initialize<MODEL>(box, each, a.psf, th);
    }
    float dmax = 0.f;  // Poisson: the largest pixel (NaN if any is), for uncapped()
    if (!SCMOS) {
        dmax = -INFINITY;
        each([&](int, int, float d) { dmax = (d > dmax || d != d) ? d : dmax; });
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, dmax, off);
            dmax = (o > dmax || o != o) ? o : dmax;
        }
    }
    // the parameter this lane updates
    int unit = 0;
    {
        float none[P][1] = {};
        scatter_sum<P, 16, P, 1>(none, lane, unit);
    }
    const int mine = min(unit, P - 1);
    const float lo = a.lower[mine], hi = a.upper[mine], most = a.max_step[mine];
    const int half = lane >> 4;  // 0: x axis, 1: y axis
    const float nk = -__fdiv_rn(1.0f, a.sqrt2pi);
    float *const ytab = tab + 5 * TS;

    for (int it = 0; it <= a.iterations; ++it) {
        const float N = th[S::IN], bg = th[S::IB];
        // this lane's axis: centre, 1/sigma, -N / (sqrt(2 pi) sigma) and, for the
        // astigmatic model, the width's derivatives by z
        const float centre = half ? th[1] : th[0];
        float sigma, ds = 0.f, d2s = 0.f;
        if (MODEL == 0) sigma = a.psf[0];
        else if (MODEL == 1) sigma = th[4];
        else if (MODEL == 2) sigma = half ? th[P - 1] : th[4];
        else
            astig_width(th[2], half ? a.psf[6] : -a.psf[6], half ? a.psf[1] : a.psf[0],
                        half ? a.psf[3] : a.psf[2], half ? a.psf[5] : a.psf[4], a.psf[7], sigma,
                        ds, d2s);
        const float is = __fdiv_rn(1.0f, sigma), cst = N * nk * is;
        __syncwarp();  // the previous pass has read the tables
        if (RMAX <= 4 && box <= 15) {  // both axes at once, at most 16 edges each
            const int e = lane & 15;
            warp_entry<MODEL, TS>(e, make_axis<MODEL>(centre, is, cst, ds, d2s), 16, e < box,
                                  half ? ytab : tab);
        } else {
#pragma unroll
            for (int axis = 0; axis < 2; axis++) {
                auto of = [&](float v) { return __shfl_sync(0xffffffffu, v, 16 * axis); };
                const Axis u = make_axis<MODEL>(of(centre), of(is), of(cst), MODEL == 3 ? of(ds) : 0.f,
                                                MODEL == 3 ? of(d2s) : 0.f);
                for (int e0 = 0; e0 < box; e0 += 31) {
                    const int e = e0 + lane;
                    warp_entry<MODEL, TS>(e, u, 32, lane < 31 && e < box, axis ? ytab : tab);
                }
            }
        }
        __syncwarp();

        // the lane's rows of psf_y (0 outside the box)
        float2 py[NPR];
        float pyl = 0.f;
        auto row = [&](int k, int r) { return ytab[k * TS + ry + kRows * r]; };  // (0 past the box)
#pragma unroll
        for (int k = 0; k < NPR; k++) py[k] = make_float2(row(0, 2 * k), row(0, 2 * k + 1));
        if (ODD) pyl = row(0, RM - 1);

        if (it < a.iterations) {
            float2 py2[NPR], aG[CROSS ? NPR : 1], C[NPR], D[NPR];
            const float py2l = pyl * pyl;
            float aGl = 0.f, Cl = 0.f, Dl = 0.f;
#pragma unroll
            for (int k = 0; k < NPR; k++) {
                py2[k] = __fmul2_rn(py[k], py[k]);
                if (CROSS) aG[k] = __fmul2_rn(py[k], make_float2(row(3, 2 * k), row(3, 2 * k + 1)));
                C[k] = D[k] = f2(0.f);
            }
            if (CROSS && ODD) aGl = pyl * row(3, RM - 1);
            float gh[P][2];
#pragma unroll
            for (int k = 0; k < P; k++) gh[k][0] = gh[k][1] = 0.f;

            auto column = [&](auto uncapped_tag, int j, const float *d, const float *v) {
                constexpr bool UNCAPPED = decltype(uncapped_tag)::value;
                const float xp = tab[j], xd1 = tab[TS + j], xd2 = tab[2 * TS + j];
                const float z1 = SIG ? tab[3 * TS + j] : 0.f, zq = SIG ? tab[4 * TS + j] : 0.f;
                const float2 npx = f2(N * xp), xpv = f2(xp), xp2 = f2(xp * xp), bgv = f2(bg);
                float2 A = f2(0.f), B = f2(0.f), E = f2(0.f), F = f2(0.f), Gc = f2(0.f);
#pragma unroll
                for (int k = 0; k < NPR; k++) {
                    const int r = 2 * k;
                    const float2 mu = __ffma2_rn(npx, py[k], bgv);
                    float2 cf, df;
                    likelihood_terms2<SCMOS, UNCAPPED>(
                        make_float2(d[r], d[r + 1]),
                        SCMOS ? make_float2(v[r], v[r + 1]) : f2(0.f), mu, cf, df);
                    if (!SCMOS && r + 1 >= W::RFULL) {  // slots that may lie outside the box
                        const bool i0 = r < W::RFULL || ry + kRows * r < box;
                        const bool i1 = ry + kRows * (r + 1) < box;
                        cf = make_float2(i0 ? cf.x : 0.f, i1 ? cf.y : 0.f);
                        df = make_float2(i0 ? df.x : 0.f, i1 ? df.y : 0.f);
                    }
                    A = __ffma2_rn(py[k], cf, A);
                    B = __ffma2_rn(py2[k], df, B);
                    E = __fadd2_rn(E, cf);
                    F = __fadd2_rn(F, df);
                    C[k] = __ffma2_rn(xpv, cf, C[k]);
                    D[k] = __ffma2_rn(xp2, df, D[k]);
                    if (CROSS) Gc = __ffma2_rn(aG[k], df, Gc);
                }
                if constexpr (ODD) {
                    const bool in = SCMOS || RM - 1 < W::RFULL || ry + kRows * (RM - 1) < box;
                    const float mu = fmaf(npx.x, pyl, bg);
                    float cf, df;
                    if constexpr (UNCAPPED) likelihood_terms_uncapped(d[RM - 1], mu, cf, df);
                    else likelihood_terms<SCMOS>(d[RM - 1], SCMOS ? v[RM - 1] : 0.f, mu, cf, df);
                    cf = in ? cf : 0.f;
                    df = in ? df : 0.f;
                    A.x = fmaf(pyl, cf, A.x);
                    B.x = fmaf(py2l, df, B.x);
                    E.x += cf;
                    F.x += df;
                    Cl = fmaf(xp, cf, Cl);
                    Dl = fmaf(xp2.x, df, Dl);
                    if (CROSS) Gc.x = fmaf(aGl, df, Gc.x);
                }
                // col_terms with the width's entries already per parameter
                const float As = A.x + A.y, Bs = B.x + B.y;
                gh[S::IX][0] = fmaf(xd1, As, gh[S::IX][0]);
                gh[S::IX][1] = fmaf(xd2, As, fmaf(-(xd1 * xd1), Bs, gh[S::IX][1]));
                gh[S::IN][0] = fmaf(xp, As, gh[S::IN][0]);
                gh[S::IN][1] = fmaf(-xp2.x, Bs, gh[S::IN][1]);
                gh[S::IB][0] += E.x + E.y;
                gh[S::IB][1] -= F.x + F.y;
                if (SIG) {
                    constexpr int K = MODEL == 3 ? 2 : 4;
                    gh[K][0] = fmaf(z1, As, gh[K][0]);
                    gh[K][1] = fmaf(zq, As, fmaf(-(z1 * z1), Bs, gh[K][1]));
                    if (CROSS) gh[K][1] = fmaf(-2.0f * z1 * xp, Gc.x + Gc.y, gh[K][1]);
                }
            };
            auto columns = [&](auto tag) {
                if constexpr (W::REG) {
#pragma unroll
                    for (int c = 0; c < CM; c++) {
                        const int j = rx + kCols * c;
                        if (c < W::cfull() || j < box) column(tag, j, dp[c], vp[SCMOS ? c : 0]);
                    }
                } else {
                    for (int j = rx; j < box; j += kCols) {
                        load_column(j);
                        column(tag, j, dp[0], vp[0]);
                    }
                }
            };
            if (!SCMOS && uncapped(N, bg, dmax)) columns(std::true_type{});
            else columns(std::false_type{});

#pragma unroll
            for (int r = 0; r < RM; r++) {  // row_terms
                const float Ct = r < 2 * NPR ? ((r & 1) ? C[r / 2].y : C[r / 2].x) : Cl;
                const float Dt = r < 2 * NPR ? ((r & 1) ? D[r / 2].y : D[r / 2].x) : Dl;
                const float yd1 = row(1, r), yd2 = row(2, r);
                gh[1][0] = fmaf(yd1, Ct, gh[1][0]);
                gh[1][1] = fmaf(yd2, Ct, fmaf(-(yd1 * yd1), Dt, gh[1][1]));
                if (SIG) {
                    constexpr int K = MODEL == 3 ? 2 : MODEL == 2 ? P - 1 : 4;
                    const float z1 = row(3, r), zq = row(4, r);
                    gh[K][0] = fmaf(z1, Ct, gh[K][0]);
                    gh[K][1] = fmaf(zq, Ct, fmaf(-(z1 * z1), Dt, gh[K][1]));
                }
            }

            // Newton step of this lane's parameter (newton_step)
            int u0 = 0;
            scatter_sum<P, 16, P, 2>(gh, lane, u0);
            float tu = th[0];
#pragma unroll
            for (int k = 1; k < P; k++) tu = mine == k ? th[k] : tu;
            const float g = gh[0][0], h = gh[0][1];
            const float delta = fabsf(h) > 1e-10f ? __fdiv_rn(g, h) : 0.f;
            tu = jl_clamp(__fadd_rn(tu, -jl_clamp(delta, -most, most)), lo, hi);
#pragma unroll
            for (int k = 0; k < P; k++)
                th[k] = __shfl_sync(0xffffffffu, tu, lane_of_unit(k, P));
        } else {
            float llr = 0.f;
            float Fh[P][P], Fl[P][P];
#pragma unroll
            for (int k = 0; k < P; k++)
#pragma unroll
                for (int l = 0; l < P; l++) { Fh[k][l] = 0.f; Fl[k][l] = 0.f; }
            auto column = [&](int j, const float *d, const float *v) {
                const float xp = tab[j], xd1 = tab[TS + j], z1 = SIG ? tab[3 * TS + j] : 0.f;
                const float npx = N * xp;
                float Q[NB][NB];
#pragma unroll
                for (int p = 0; p < NB; p++)
#pragma unroll
                    for (int q = 0; q < NB; q++) Q[p][q] = 0.f;
#pragma unroll
                for (int r = 0; r < RM; r++) {
                    const int i = ry + kRows * r;
                    if (r < W::RFULL || i < box) {
                        const float p = ytab[i];
                        final_pixel<SCMOS, SIG, NB>(d[r], SCMOS ? v[r] : 0.f, fmaf(npx, p, bg),
                                                    p, ytab[TS + i],
                                                    SIG ? ytab[3 * TS + i] : 0.f, llr, Q);
                    }
                }
                fisher_column<MODEL, P, NB>(Fh, Fl, Q, xp, xd1, z1);
            };
            if constexpr (W::REG) {
#pragma unroll
                for (int c = 0; c < CM; c++) {
                    const int j = rx + kCols * c;
                    if (c < W::cfull() || j < box) column(j, dp[c], vp[SCMOS ? c : 0]);
                }
            } else {
                for (int j = rx; j < box; j += kCols) {
                    load_column(j);
                    column(j, dp[0], vp[0]);
                }
            }
            llr = warp_sum(llr);
            float fh[NF], fl[NF];
            int q = 0;
#pragma unroll
            for (int k = 0; k < P; k++)
#pragma unroll
                for (int l = k; l < P; l++, q++) { fh[q] = Fh[k][l]; fl[q] = Fl[k][l]; }
            int f = 0, held = NF;
            scatter_sum_dd<NF, 16, NF>(fh, fl, lane, f, held);
            if (held > 0) res.F[f] = dd_to_double(fh[0], fl[0]);
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < P; k++) res.th[k] = th[k];
                res.llr = llr;
                res.ok = ok;
            }
        }
    }
}

// Fit the ROIs [roi0, roi0 + nroi) of `a`, one per warp of the block.
template <int MODEL, bool SCMOS, int RMAX>
__device__ __forceinline__ void fit_block_warp(const KernelArgs &a, const int box,
                                               const int64_t roi0, const int nroi, float *smem)
{
    constexpr int P = ModelInfo<MODEL>::P;
    __shared__ RoiResult<P> s_res[kWarpMaxRois];
    const int wid = threadIdx.x >> 5;
    if (wid < nroi)  // one decision per warp
        fit_roi_warp<MODEL, SCMOS, RMAX>(a, box, roi0 + wid,
                                         smem + (size_t)wid * warp_floats(box, SCMOS), s_res[wid]);
    __syncthreads();
    if (threadIdx.x < nroi) {
        const RoiResult<P> &res = s_res[threadIdx.x];
        double Fm[P][P];
        float th[P];
        int q = 0;
#pragma unroll
        for (int k = 0; k < P; k++) {
            th[k] = res.th[k];
#pragma unroll
            for (int l = k; l < P; l++, q++) Fm[k][l] = Fm[l][k] = res.F[q];
        }
        write_result<P>(a, roi0 + threadIdx.x, res.ok, th, Fm, res.llr);
    }
}

// TABLE as for fit_kernel_r1, with tiles of one ROI per warp (boxes up to 16).
//
// Resident blocks: registers are what bounds the warps per SM, and with two or
// three warps per scheduler the kernel waits more than it issues (54 % of the
// slots).  Asking for 20 warps (boxes to 16), 16 (to 24) and 12 (beyond) gives
// 96, 128 and 168 registers without spills: 12 000 astigmatic 21x21 sCMOS ROIs
// 320 -> 278 us (148 -> 128 registers).
template <int MODEL, bool SCMOS, int RMAX, bool TABLE>
__global__ void __launch_bounds__(32 * kWarpMaxRois, RMAX <= 4 ? 5 : RMAX <= 6 ? 4 : 3)
    fit_kernel_warp(const KernelArgs a, const TileTable t, const int box)
{
    extern __shared__ __align__(16) float smem[];
    const int nw = blockDim.x >> 5;
    if (!TABLE) {
        const int64_t roi0 = (int64_t)blockIdx.x * nw, left = a.n - roi0;
        fit_block_warp<MODEL, SCMOS, RMAX>(a, box, roi0, left < nw ? (int)left : nw, smem);
    } else {
        TableSlot *ts = table_slot(smem, sizeof(float) * (size_t)warp_floats(box, SCMOS) * nw);
        table_slot_init(ts);
        int64_t roi0;
        int nroi;
        for (int k = 0; table_next(t, nw, ts, k, roi0, nroi); k++) {
            fit_block_warp<MODEL, SCMOS, RMAX>(ts->a, box, roi0, nroi, smem);
            __syncthreads();  // the tile's shared memory and slot are free again
        }
    }
}

using WarpKernel = void (*)(const KernelArgs, const TileTable, const int);

template <int MODEL, bool SCMOS> WarpKernel warp_kernel(int box, bool table)
{
    switch (rows_per_lane(box)) {
        case 2: return table ? fit_kernel_warp<MODEL, SCMOS, 2, true> : fit_kernel_warp<MODEL, SCMOS, 2, false>;
        case 3: return table ? fit_kernel_warp<MODEL, SCMOS, 3, true> : fit_kernel_warp<MODEL, SCMOS, 3, false>;
        case 4: return table ? fit_kernel_warp<MODEL, SCMOS, 4, true> : fit_kernel_warp<MODEL, SCMOS, 4, false>;
        case 5: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 5, false>;
        case 6: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 6, false>;
        case 7: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 7, false>;
        case 8: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 8, false>;
        case 12: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 12, false>;
        case 16: return table ? nullptr : fit_kernel_warp<MODEL, SCMOS, 16, false>;
        default: return nullptr;
    }
}

}  // namespace

template <int MODEL, bool SCMOS>
cudaError_t launch_warp_family(int box, const KernelArgs &a, const TileTable &t,
                               int rois_per_block, int64_t grid, cudaStream_t s)
{
    const bool table = t.header != nullptr;
    if (box < 3 || box > kLargeMaxBox || a.tpr != 32) return cudaErrorInvalidValue;
    WarpKernel k = warp_kernel<MODEL, SCMOS>(box, table);
    if (!k || rois_per_block < 1 || rois_per_block > kWarpMaxRois)
        return cudaErrorInvalidValue;
    size_t smem = sizeof(float) * (size_t)warp_floats(box, SCMOS) * rois_per_block;
    if (table) smem = table_smem_bytes(smem);
    if (smem > 48 * 1024 - 4096) {  // (the kernel's static shared memory counts as well)
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    const int64_t blocks = table ? grid : (a.n + rois_per_block - 1) / rois_per_block;
    if (blocks <= 0) return cudaSuccess;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    k<<<(unsigned)blocks, 32 * rois_per_block, smem, s>>>(a, t, box);
    return cudaGetLastError();
}

template <int MODEL, bool SCMOS> int warp_table_blocks(int box, int rois_per_block)
{
    WarpKernel k = warp_kernel<MODEL, SCMOS>(box, true);
    if (!k) return 0;
    int nb = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &nb, k, 32 * rois_per_block,
        table_smem_bytes(sizeof(float) * (size_t)warp_floats(box, SCMOS) * rois_per_block));
    return e == cudaSuccess ? nb : -(int)e;
}

template cudaError_t launch_warp_family<GMLE_MODEL, (GMLE_SCMOS != 0)>(int, const KernelArgs &,
                                                                      const TileTable &, int,
                                                                      int64_t, cudaStream_t);
template int warp_table_blocks<GMLE_MODEL, (GMLE_SCMOS != 0)>(int, int);

}  // namespace gmle
