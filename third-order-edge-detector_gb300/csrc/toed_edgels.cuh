// toed_edgels.cuh -- the edgel kernel: a CTA takes the segments of one strip
// column over p.ed_rows image rows, stages the pixels that their edgels'
// windows cover in shared memory once, and runs a thread per edgel:
//   QAD false   the third-order orientation at the edgel's 2x-grid point
//               (toed_edgels.cu);
//   QAD true    the same of the nine derivatives cubic-interpolated at its
//               subpixel point (toed_qad.cu).
// The x taps depend on the parity of a 2x column alone -- the edgel's own, or
// its subpixel cell's -- so a chunk's edgels are ordered by it and every warp
// runs one fully unrolled row of compile-time operands.
#pragma once
#include "toed_common.cuh"
#include "toed_edgel.cuh"
#include "toed_internal.h"

namespace toed {

constexpr int kEdThreads = 256;
constexpr int kEdChunk = kEdThreads - 32;  // edgels at a time: ordered by parity, each kind from a warp's start
constexpr int kRefineMost = 8;             // edgels a warp forms again in FP64 before their orientations
static_assert(kEdRowsMax <= kEdThreads && kEdThreads % 32 == 0, "two segments a thread");

template <int R, bool QAD>
struct EdCfg {
    static constexpr int NT = 2 * R + 3;            // window side at a grid point
    // a tile's pixels reach HALO past its own: the window's half, and for a
    // subpixel point up to one pixel of offset and one of interpolation more
    static constexpr int HALO = QAD ? R + 3 : R + 1;
    static constexpr int TW = kInner + 2 * HALO;    // columns of a tile's pixels
    static constexpr int TP = staged_width(R);      // their pitch in shared memory: a box of the detection's row map
    static_assert(TW + 3 <= TP, "a box aligned down to 16 bytes holds them");
    static __host__ __device__ constexpr int boxes(int rows) { return (rows + 2 * HALO + kStepRows - 1) / kStepRows; }
    static constexpr size_t smem(int rows) { return sizeof(float) * TP * boxes(rows) * kStepRows; }
};

// Sums of nine values over the warp into out[0..8], by halving exchanges: an
// SM's FP64 pipe takes about 15 cycles for a warp's instruction, so they take
// 12 additions instead of a butterfly's 45.
__device__ __forceinline__ void warp_sum9(double (&d)[9], int lane, double* __restrict__ out)
{
#define TOED_HALVE(BIT, N, KEEP)                                                            \
    {                                                                                       \
        const bool hi = lane & BIT;                                                         \
        _Pragma("unroll") for (int f = 0; f < KEEP; ++f)                                    \
        {                                                                                   \
            const double up = f + KEEP < N ? d[f + KEEP] : 0.0;                             \
            const double got = __shfl_xor_sync(0xffffffffu, hi ? d[f] : up, BIT);           \
            d[f] = (hi ? up : d[f]) + got;                                                  \
        }                                                                                   \
    }
    TOED_HALVE(16, 9, 5)
    TOED_HALVE(8, 5, 3)
    TOED_HALVE(4, 3, 2)
    TOED_HALVE(2, 2, 1)
#undef TOED_HALVE
    d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1);
    // the lanes past each half's values (5..8 of 9, 3..4 of 5, ...) hold zeros' sums
    const int h16 = (lane & 16) ? 4 : 5, at16 = (lane & 16) ? 5 : 0;
    const int h8 = (lane & 8) ? h16 - 3 : 3, at8 = (lane & 8) ? 3 : 0;
    const int h4 = (lane & 4) ? h8 - 2 : min(h8, 2), at4 = (lane & 4) ? 2 : 0;
    const int h2 = (lane & 2) ? h4 - 1 : min(h4, 1);
    if (h2 > 0 && !(lane & 1)) out[at16 + at8 + at4 + ((lane & 2) ? 1 : 0)] = d[0];
}

// One edgel, one warp: the nine derivatives at 2x-grid point (Gr, Gc) =
// (2i + a, 2j + b) from the staged pixels (win: the corner of its (2r+3)^2
// window, rows `pitch` apart) with FP64 taps -- the (2r+1)^2 window of
// unshifted taps on sub-grid (0, 0) (cpu_toed.cpp:205-221), the (2r+3)^2
// window with the half-pixel shifted taps along the odd axes elsewhere
// (cpu_toed.cpp:246-344) -- into out[0..8].  Lane t forms the four
// column-filtered sums of one window row; the row filters then weight them and
// the warp sums them.  Out of line: it is rare, and inlined its registers
// would crowd the FP32 contraction.
static __device__ __noinline__ void refine_edgel(const BatchParams& p, const float* __restrict__ win, int pitch, int a, int b,
                                          int lane, double* __restrict__ out)
{
    const int r = p.radius;
    const int h = (a | b) ? r + 1 : r;
    const double* X = &p.taps64.v[b ? 4 : 0][0];  // filter f, tap k: X[f * kMaxTaps + k]
    const double* Y = &p.taps64.v[a ? 4 : 0][0];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0, y0 = 0.0, y1 = 0.0, y2 = 0.0, y3 = 0.0;
    if (lane <= 2 * h) {  // row offset lane - h: out = sum in(i - p) Y(p)
        const float* row = win + (r + 1 + h - lane) * pitch + r + 1 + h;
        const int k0 = r + 1 - h;  // tap of column offset q = -h
#pragma unroll 4
        for (int t = 0; t <= 2 * h; ++t) {
            const double x = row[-t];
            s0 = fma(x, X[k0 + t], s0);
            s1 = fma(x, X[kMaxTaps + k0 + t], s1);
            s2 = fma(x, X[2 * kMaxTaps + k0 + t], s2);
            s3 = fma(x, X[3 * kMaxTaps + k0 + t], s3);
        }
        const int kp = lane - h + r + 1;
        y0 = Y[kp];
        y1 = Y[kMaxTaps + kp];
        y2 = Y[2 * kMaxTaps + kp];
        y3 = Y[3 * kMaxTaps + kp];
    }
    // fx fy fxx fxy fyy fxxy fxyy fxxx fyyy
    double d[9] = {y0 * s1, y1 * s0, y0 * s2, y1 * s1, y2 * s0, y1 * s2, y2 * s1, y0 * s3, y3 * s0};
    warp_sum9(d, lane, out);
}

// The third-order orientation (cpu_toed.cpp:227-232) in FP64 of nine derivatives.
__device__ __forceinline__ float orientation64(const double* __restrict__ d)
{
    const double fx = d[0], fy = d[1], fxx = d[2], fxy = d[3], fyy = d[4], fxxy = d[5], fxyy = d[6], fxxx = d[7],
                 fyyy = d[8];
    const double tix = fx * (2 * fxx * fxx + 2 * fxy * fxy) + fy * (2 * fxx * fxy + 2 * fyy * fxy) +
                       2 * fx * fy * fxxy + fy * fy * fxyy + fx * fx * fxxx;
    const double tiy = fx * (2 * fxx * fxy + 2 * fyy * fxy) + fy * (2 * fyy * fyy + 2 * fxy * fxy) +
                       2 * fx * fy * fxyy + fx * fx * fxxy + fy * fy * fyyy;
    return (tix == 0.0 && tiy == 0.0) ? __int_as_float(0x7fc00000) : (float)atan2(tix, -tiy);
}

// The seven higher derivatives (fxx, fxy, fyy, fxxy, fxyy, fxxx, fyyy) of a
// point on 2x column parity B from the staged pixels, `win` its window's
// corner: each window row's responses G, Gx, Gxx, Gxxx -- truncated to 2r+1
// taps (T) on sub-grid (0, 0), full (F) at odd 2x rows a, half-pixel shifted
// (S) at odd columns -- and their products with the row's y taps (G, Gy, Gyy,
// Gyyy), yt[k] that of tap k.  The sums are those of the detection kernel's
// row pass and of the corrected-normal mode's gather_hi, in the same order.
template <int R, int B>
__device__ __forceinline__ void window7(const float* __restrict__ win, int a, const float4* __restrict__ yt,
                                        const TapBlock& tp, float (&d)[7])
{
    constexpr int NT = 2 * R + 3, c = R + 1;  // out = sum_q in(x - q) X(q), in(x - q) = v[c - q]
#pragma unroll
    for (int f = 0; f < 7; ++f) d[f] = 0.f;
#pragma unroll 1
    for (int kk = 0; kk < NT; ++kk) {
        float v[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) v[t] = win[kk * staged_width(R) + t];
        const float4 t = yt[NT - 1 - kk];
        float hG = 0.f, hGx = 0.f, hGxx = 0.f, hGxxx = 0.f;
        if (B == 0) {
#pragma unroll
            for (int q = -R; q <= R; ++q) {
                hG = fmaf(v[c - q], tp.v[0][q + R + 1], hG);
                hGxx = fmaf(v[c - q], tp.v[2][q + R + 1], hGxx);
            }
#pragma unroll
            for (int q = 1; q <= R; ++q) {
                const float df = v[c - q] - v[c + q];
                hGx = fmaf(df, tp.v[1][q + R + 1], hGx);
                hGxxx = fmaf(df, tp.v[3][q + R + 1], hGxxx);
            }
            if (a) {
                hG = fmaf(v[c + R + 1], tp.v[0][0], fmaf(v[c - R - 1], tp.v[0][2 * R + 2], hG));
                hGxx = fmaf(v[c + R + 1], tp.v[2][0], fmaf(v[c - R - 1], tp.v[2][2 * R + 2], hGxx));
                const float df = v[c - R - 1] - v[c + R + 1];
                hGx = fmaf(df, tp.v[1][2 * R + 2], hGx);
                hGxxx = fmaf(df, tp.v[3][2 * R + 2], hGxxx);
            }
        } else {
#pragma unroll
            for (int q = -(R + 1); q <= R + 1; ++q) {
                hG = fmaf(v[c - q], tp.v[4][q + R + 1], hG);
                hGxx = fmaf(v[c - q], tp.v[6][q + R + 1], hGxx);
            }
            hGx = v[c - R - 1] * tp.v[5][2 * R + 2];
            hGxxx = v[c - R - 1] * tp.v[7][2 * R + 2];
#pragma unroll
            for (int q = 0; q <= R; ++q) {
                const float df = v[c - q] - v[c + 1 + q];
                hGx = fmaf(df, tp.v[5][q + R + 1], hGx);
                hGxxx = fmaf(df, tp.v[7][q + R + 1], hGxxx);
            }
        }
        d[1] = fmaf(hGx, t.y, d[1]);
        d[2] = fmaf(hG, t.z, d[2]);
        d[4] = fmaf(hGx, t.z, d[4]);
        d[6] = fmaf(hG, t.w, d[6]);
        d[0] = fmaf(hGxx, t.x, d[0]);
        d[3] = fmaf(hGxx, t.y, d[3]);
        d[5] = fmaf(hGxxx, t.x, d[5]);
    }
}

// ---------------------------------------------------------------------------
// Quick-and-dirty mode: the nine derivatives interpolated at a subpixel point
// ---------------------------------------------------------------------------
// Keys cubic convolution kernel, a = -1/2 (subpix_to_correction.cpp:57-67).
template <typename T>
__device__ __forceinline__ T keys(T s)
{
    const T a = T(-0.5), x = fabs(s);
    if (x <= T(1)) return ((a + T(2)) * x - (a + T(3))) * x * x + T(1);
    if (x < T(2)) return ((a * x - T(5) * a) * x + T(8) * a) * x - T(4) * a;
    return T(0);
}

__device__ __forceinline__ float4 fma4(float a, float4 x, float4 y)
{
    return make_float4(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y), fmaf(a, x.z, y.z), fmaf(a, x.w, y.w));
}

// One window row's responses (G, Gx, Gxx, Gxxx) at the column C of v: T
// (truncated) and F (full), or S (half-pixel shifted).
template <int R, int C>
__device__ __forceinline__ void row_tf(const float* v, const TapBlock& tp, float4& t, float4& f)
{
    t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = -R; q <= R; ++q) {
        t.x = fmaf(v[C - q], tp.v[0][q + R + 1], t.x);
        t.z = fmaf(v[C - q], tp.v[2][q + R + 1], t.z);
    }
#pragma unroll
    for (int q = 1; q <= R; ++q) {
        const float df = v[C - q] - v[C + q];
        t.y = fmaf(df, tp.v[1][q + R + 1], t.y);
        t.w = fmaf(df, tp.v[3][q + R + 1], t.w);
    }
    f.x = fmaf(v[C + R + 1], tp.v[0][0], fmaf(v[C - R - 1], tp.v[0][2 * R + 2], t.x));
    f.z = fmaf(v[C + R + 1], tp.v[2][0], fmaf(v[C - R - 1], tp.v[2][2 * R + 2], t.z));
    const float df = v[C - R - 1] - v[C + R + 1];
    f.y = fmaf(df, tp.v[1][2 * R + 2], t.y);
    f.w = fmaf(df, tp.v[3][2 * R + 2], t.w);
}
template <int R, int C>
__device__ __forceinline__ float4 row_s(const float* v, const TapBlock& tp)
{
    float4 s = make_float4(0.f, v[C - R - 1] * tp.v[5][2 * R + 2], 0.f, v[C - R - 1] * tp.v[7][2 * R + 2]);
#pragma unroll
    for (int q = -(R + 1); q <= R + 1; ++q) {
        s.x = fmaf(v[C - q], tp.v[4][q + R + 1], s.x);
        s.z = fmaf(v[C - q], tp.v[6][q + R + 1], s.z);
    }
#pragma unroll
    for (int q = 0; q <= R; ++q) {
        const float df = v[C - q] - v[C + 1 + q];
        s.y = fmaf(df, tp.v[5][q + R + 1], s.y);
        s.w = fmaf(df, tp.v[7][q + R + 1], s.w);
    }
    return s;
}

// x = (G, Gx, Gxx, Gxxx) responses, y = (G, Gy, Gyy, Gyyy) taps, added to
// fx fy fxx fxy fyy fxxy fxyy fxxx fyyy.
__device__ __forceinline__ void pair9(float4 x, float4 y, float (&d)[9])
{
    d[0] = fmaf(x.y, y.x, d[0]);
    d[1] = fmaf(x.x, y.y, d[1]);
    d[2] = fmaf(x.z, y.x, d[2]);
    d[3] = fmaf(x.y, y.y, d[3]);
    d[4] = fmaf(x.x, y.z, d[4]);
    d[5] = fmaf(x.z, y.y, d[5]);
    d[6] = fmaf(x.y, y.z, d[6]);
    d[7] = fmaf(x.w, y.x, d[7]);
    d[8] = fmaf(x.x, y.w, d[8]);
}

// The nine derivatives interpolated at (X1 + tx, Y1 + ty) of the 2x grid,
// X1 = 2 j + (1 - E), from the window of pixels j - r - 2 .. j + r + 2 and
// rows i - r - 2 .., i = Y1 >> 1, whose corner is `win`.  The 4 x 4 block's
// columns X1 - 1 .. X1 + 2 alternate in parity: two on whole columns (pixels j
// and j + 1), which take T responses in rows on whole rows and F in the
// others, and two shifted (j - 1 and j for X1 even, j and j + 1 for X1 odd).
// Interpolation is linear, so their responses fold into three weighted
// sums xT, xF, xS per window row, the block rows' taps into yT, yF (two whole
// rows) and yS (two shifted): D = yT xT + yF xS + yS (xF + xS).
// sTab: per variant T, F, S the taps k - 2 with two zero entries each side.
template <int R, int E>
__device__ __forceinline__ void subpixel9(const float* __restrict__ win, int Y1, float tx, float ty,
                                          const float4* __restrict__ sTab, const TapBlock& tp, float (&d)[9])
{
    constexpr int NT = 2 * R + 3, NTP = NT + 4, NU = NT + 2, C = R + 2;  // pixel j is window column C
    float wx[4], wy[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        wx[s] = keys(tx + 1.f - (float)s);
        wy[s] = keys(ty + 1.f - (float)s);
    }
    // block row s: 2x row Y1 - 1 + s, pixel row offset from i; whole rows first
    const int od = Y1 & 1, s0 = od ? 0 : 1;  // whole rows are s0 and s0 + 2, shifted ones 1 - s0 and 3 - s0
    const int i = Y1 >> 1;
    const float w0 = od ? wy[0] : wy[1], w1 = od ? wy[2] : wy[3], v0 = od ? wy[1] : wy[0], v1 = od ? wy[3] : wy[2];
    // tap of window row u for a point at row offset o: entry NT + 2 + o - u
    const float4* tw0 = sTab + NT + 2 + ((Y1 - 1 + s0) >> 1) - i;
    const float4* tw1 = sTab + NT + 2 + ((Y1 + 1 + s0) >> 1) - i;
    const float4* ts0 = sTab + 2 * NTP + NT + 2 + ((Y1 - s0) >> 1) - i;
    const float4* ts1 = sTab + 2 * NTP + NT + 2 + ((Y1 + 2 - s0) >> 1) - i;
#pragma unroll
    for (int f = 0; f < 9; ++f) d[f] = 0.f;
#pragma unroll 1
    for (int u = 0; u < NU; ++u) {
        float v[NU];
#pragma unroll
        for (int t = 0; t < NU; ++t) v[t] = win[u * staged_width(R) + t];
        float4 xT, xF, xS;
        {
            float4 t0, f0, t1, f1;
            row_tf<R, C>(v, tp, t0, f0);
            row_tf<R, C + 1>(v, tp, t1, f1);
            const float a = E ? wx[1] : wx[0], b = E ? wx[3] : wx[2];
            xT = fma4(b, t1, make_float4(a * t0.x, a * t0.y, a * t0.z, a * t0.w));
            xF = fma4(b, f1, make_float4(a * f0.x, a * f0.y, a * f0.z, a * f0.w));
        }
        {
            const float4 a = row_s<R, E ? C - 1 : C>(v, tp), b = row_s<R, E ? C : C + 1>(v, tp);
            const float wa = E ? wx[0] : wx[1], wb = E ? wx[2] : wx[3];
            xS = fma4(wb, b, make_float4(wa * a.x, wa * a.y, wa * a.z, wa * a.w));
        }
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        pair9(xT, fma4(w1, tw1[-u], fma4(w0, tw0[-u], zero)), d);
        pair9(xS, fma4(w1, tw1[NTP - u], fma4(w0, tw0[NTP - u], zero)), d);
        const float4 yS = fma4(v1, ts1[-u], fma4(v0, ts0[-u], zero));
        pair9(make_float4(xF.x + xS.x, xF.y + xS.y, xF.z + xS.z, xF.w + xS.w), yS, d);
    }
}

// The same in FP64 for one record, the whole warp: lane c takes window column
// c, contracts it with the folded y taps and weights the sums with its folded
// x taps; the lanes' products are summed into out[0..8].  Out of line: rare.
static __device__ __noinline__ void refine_subpixel(const BatchParams& p, const float* __restrict__ win, int pitch, int X1, int Y1,
                                             double tx, double ty, int lane, double* __restrict__ out)
{
    const int R = p.radius, NT = 2 * R + 3, NU = NT + 2;
    const int j = X1 >> 1, i = Y1 >> 1;
    double d[9];
#pragma unroll
    for (int f = 0; f < 9; ++f) d[f] = 0.0;
    if (lane < NU) {
        // this column's x taps, folded: variant 0 T, 1 F (whole columns), 2 S
        double x[3][4] = {};
        for (int s = 0; s < 4; ++s) {
            const int X = X1 - 1 + s, k = NT + ((X >> 1) - j) - lane;  // tap of column `lane`
            const double w = keys(tx + 1.0 - (double)s);
            if (k < 0 || k >= NT) continue;
            for (int f = 0; f < 4; ++f) {
                if (X & 1) {
                    x[2][f] += w * p.taps64.v[4 + f][k];
                } else {
                    if (k > 0 && k < NT - 1) x[0][f] += w * p.taps64.v[f][k];
                    x[1][f] += w * p.taps64.v[f][k];
                }
            }
        }
        // the column contracted with each block row's taps (F on whole rows, S on shifted ones) ...
        double cs[4][4] = {};
        for (int u = 0; u < NU; ++u) {
            const double v = win[u * pitch + lane];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int Y = Y1 - 1 + s, k = NT + ((Y >> 1) - i) - u;
                if (k < 0 || k >= NT) continue;
                const double(*tap)[kMaxTaps] = p.taps64.v + ((Y & 1) ? 4 : 0);
#pragma unroll
                for (int f = 0; f < 4; ++f) cs[s][f] = fma(v, tap[f][k], cs[s][f]);
            }
        }
        // ... and folded: yT (F less its two end taps), yF, yS
        double c[3][4] = {};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int Y = Y1 - 1 + s, o = (Y >> 1) - i;
            const double w = keys(ty + 1.0 - (double)s);
            const double va = win[(NT + o) * pitch + lane], vb = win[(o + 1) * pitch + lane];  // of taps 0 and NT - 1
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                if (Y & 1) {
                    c[2][f] = fma(w, cs[s][f], c[2][f]);
                } else {
                    c[1][f] = fma(w, cs[s][f], c[1][f]);
                    c[0][f] = fma(w, fma(-vb, p.taps64.v[f][NT - 1], fma(-va, p.taps64.v[f][0], cs[s][f])), c[0][f]);
                }
            }
        }
        for (int g = 0; g < 3; ++g) {
            const double* y = c[g];
            const double xs[4] = {g == 0 ? x[0][0] : (g == 1 ? x[2][0] : x[1][0] + x[2][0]),
                                  g == 0 ? x[0][1] : (g == 1 ? x[2][1] : x[1][1] + x[2][1]),
                                  g == 0 ? x[0][2] : (g == 1 ? x[2][2] : x[1][2] + x[2][2]),
                                  g == 0 ? x[0][3] : (g == 1 ? x[2][3] : x[1][3] + x[2][3])};
            d[0] += xs[1] * y[0];
            d[1] += xs[0] * y[1];
            d[2] += xs[2] * y[0];
            d[3] += xs[1] * y[1];
            d[4] += xs[0] * y[2];
            d[5] += xs[2] * y[1];
            d[6] += xs[1] * y[2];
            d[7] += xs[3] * y[0];
            d[8] += xs[0] * y[3];
        }
    }
    warp_sum9(d, lane, out);
}

// The cell of the 2x grid that an edgel's subpixel point lies in, pos = 2 x_out + 1 (FP64, cpu_toed.cpp:516).
struct Subpixel {
    double tx, ty;
    int X1, Y1;
};
__device__ __forceinline__ Subpixel subpixel_of(const Staged& e, int W2, bool hyb)
{
    const int Gr = e.idx / W2, Gc = e.idx - Gr * W2;
    const Fitted ft = fit_edgel(e, e.gx, e.gy, false, hyb, Gr, Gc);
    const double px = 2.0 * ft.x + 1.0, py = 2.0 * ft.y + 1.0, fx = floor(px), fy = floor(py);
    // the offset is at most sqrt(2), so the cell lies within these; the staged pixels reach no further
    return {px - fx, py - fy, min(max((int)fx, Gc - 2), Gc + 1), min(max((int)fy, Gr - 2), Gr + 1)};
}

// A tile of band `ty` is done: the CTA that completes the band -- tiles of all
// strip columns over the same rows, whose edgels are consecutive in the list --
// copies its part of the list to the host, in whole lines.  So the lists cross
// the link while later bands are worked on.  (The tiles' own stores, single
// records at scattered places, took 0.45 ms more per 40 MB over the link; a copy
// kernel afterwards 0.2 ms.)
static __device__ __noinline__ void band_done(const BatchParams& p, const DetImage& im, int ty, int* s_last)
{
    __syncthreads();
    if (!TOED_IN_BOUNDS(im.band_base + ty < p.n_bands, p.sc.words)) return;
    if (threadIdx.x == 0) {
        __threadfence();
        *s_last = atomicAdd(&p.sc.band[im.band_base + ty], 1) == im.nsc - 1;
        __threadfence();
    }
    __syncthreads();
    if (!*s_last) return;
    const long long row = 2LL * p.ed_rows * im.nsc;  // segments a band
    const long long q0 = ty * row, q1 = q0 + row;
    if (!TOED_IN_BOUNDS(q0 < im.nseg && im.seg_base + im.nseg <= p.sc.seg_cap, p.sc.words)) return;
    const int lo = min(p.sc.seg_dst[im.seg_base + q0], im.cap);
    const int hi = min(q1 < im.nseg ? p.sc.seg_dst[im.seg_base + q1] : *im.count, im.cap);
    if (!TOED_IN_BOUNDS(lo >= 0, p.sc.words)) return;
    const int per = p.out_f64 ? 2 : 1;  // 16-byte parts of a record
    const uint4* src = static_cast<const uint4*>(im.out);
    uint4* dst = static_cast<uint4*>(im.host_out);
    for (long long i = (long long)lo * per + threadIdx.x; i < (long long)hi * per; i += blockDim.x) dst[i] = __ldcg(src + i);
    if (im.host_index)
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) im.host_index[i] = __ldcg(im.index + i);
}

template <int R, bool QAD>
__global__ void __launch_bounds__(kEdThreads, R <= 8 && !QAD ? 3 : 2) fin_edgels(const __grid_constant__ BatchParams p)
{
    using E = EdCfg<R, QAD>;
    constexpr int NT = E::NT, TP = E::TP;
    constexpr int PAD = QAD ? 2 : 0, NTP = NT + 2 * PAD;  // zero taps each side (subpixel9)
    extern __shared__ __align__(128) float sPix[];
    __shared__ int s_warp[33];
    __shared__ float4 sTab[3 * NTP];     // y taps per variant T, F, S: (G, Gy, Gyy, Gyyy) of tap k - PAD
    __shared__ int2 sList[kEdChunk];     // a chunk's edgels: staging slot, list position
    __shared__ Staged sRec[kEdThreads];  // their records, ordered
    __shared__ int sPos[kEdThreads];     // and list positions, -1: none; -2 - position: FP64 orientation wanted
    __shared__ Subpixel sAt[QAD ? kEdThreads : 1];
    __shared__ unsigned char sFlag[kEdThreads];  // the slots of those
    __shared__ int sFlags;
    __shared__ double sD64[kEdThreads / 32][kRefineMost][9];
    __shared__ __align__(8) unsigned long long sBar;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int t = blockIdx.x;
    const int k = find_image(p.n_img, t, [&](int i) { return p.img[i].ed_base; });
    const DetImage& im = p.img[k];
    const int H = im.H, W = im.W, W2 = 2 * W;
    const int lt = t - im.ed_base, ty = lt / im.nsc, sc = lt - ty * im.nsc;
    const int rows = p.ed_rows, y0 = ty * rows, nrow = min(rows, H - y0);
    for (int i = tid; i < 3 * NTP; i += kEdThreads) {
        const int v = i / NTP, q = i - v * NTP - PAD;
        const int f = (v == 2) ? 4 : 0;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q >= 0 && q < NT && !(v == 0 && (q == 0 || q == NT - 1)))
            w = make_float4(p.taps.v[f][q], p.taps.v[f + 1][q], p.taps.v[f + 2][q], p.taps.v[f + 3][q]);
        sTab[i] = w;
    }
    grid_wait();
    // the tile's segments: 2x rows 2 y0 .., strip column sc; at most two of them a thread
    int2 seg[2];
    int dst[2], sum = 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int r2 = 2 * tid + u;
        seg[u] = make_int2(0, 0);
        dst[u] = 0;
        if (r2 < 2 * nrow) {
            const long long q = im.seg_base + (long long)(2 * y0 + r2) * im.nsc + sc;
            if (TOED_IN_BOUNDS(q < im.seg_base + im.nseg && q < p.sc.seg_cap, p.sc.words)) {
                seg[u] = p.sc.seg[q];
                dst[u] = p.sc.seg_dst[q];
            }
        }
        sum += seg[u].y;
    }
    int total;
    int run = block_excl_scan<kEdThreads>(sum, s_warp, &total);
    if (total == 0) {
        if (im.host_out) band_done(p, im, ty, s_warp);
        return;
    }
    // pixels x0 - HALO .. x0 + 29 + HALO, rows y0 - HALO .., zero outside the image, by TMA where the detection kernel's rows came so
    const int px = sc * kInner - E::HALO, py = y0 - E::HALO;
    const int x_al = floor4(px), shift = px - x_al;
    const uint32_t bar = smem_addr(&sBar);
    // the staged pixels' floats, and whether a window of `side` rows and floats at `win` lies in them
    [[maybe_unused]] const int n_pix = E::boxes(nrow) * kStepRows * TP;
    [[maybe_unused]] auto staged = [&](const float* win, int side) {
        return win >= sPix && (win - sPix) + (side - 1) * TP + side <= n_pix;
    };
    if (im.tma) {
        if (tid == 0) {
            mbar_init(bar);
            const int nb = E::boxes(nrow);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                         "r"((uint32_t)(nb * kStepRows * TP * sizeof(float)))
                         : "memory");
            for (int q = 0; q < nb; ++q)
                tma_copy_rows(&p.tmap[k], smem_addr(sPix + q * kStepRows * TP), bar, x_al, py + q * kStepRows);
        }
    } else {
        const int nr = nrow + 2 * E::HALO;
        if (im.dtype == TOED_U8) {  // a word a lane, two rows a warp
            static_assert(E::TW + 3 <= 64, "sixteen words a row");
#pragma unroll 4
            for (int r0 = 2 * wid; r0 < nr; r0 += 2 * (kEdThreads / 32)) {
                const int r = r0 + (lane >> 4);
                const Bytes4 b = fetch_bytes(im.src, im.pitch, H, W, py + r, px, lane & 15, E::TW);
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (r < nr && (unsigned)(b.c + e) < (unsigned)E::TW &&
                        TOED_IN_BOUNDS(r * TP + shift + b.c + e < n_pix, p.sc.words))
                        sPix[r * TP + shift + b.c + e] = (float)((b.w >> (8 * e)) & 255u);
            }
        } else {
            const float* src = static_cast<const float*>(im.src);
#pragma unroll 4
            for (int r = wid; r < nr; r += kEdThreads / 32) {
#pragma unroll
                for (int c = 0; c < (E::TW + 31) / 32; ++c) {
                    const int col = lane + 32 * c, y = py + r, x = px + col;
                    if (col < E::TW && TOED_IN_BOUNDS(r * TP + shift + col < n_pix, p.sc.words))
                        sPix[r * TP + shift + col] = (unsigned)y < (unsigned)H && (unsigned)x < (unsigned)W
                                                         ? __ldg(src + (long long)y * im.pitch + x)
                                                         : 0.f;
                }
            }
        }
    }
    const long long cap = im.cap;
    for (int c0 = 0; c0 < total; c0 += kEdChunk) {
        // the chunk's edgels, then their records ordered by 2x column parity
        for (int u = 0, at = run - c0; u < 2; ++u)
            for (int e = 0; e < seg[u].y; ++e, ++at)
                if (at >= 0 && at < kEdChunk) sList[at] = make_int2(seg[u].x + e, dst[u] + e);
        sPos[tid] = -1;
        if (tid == 0) sFlags = 0;
        __syncthreads();
        if (im.tma && c0 == 0 && !mbar_wait(bar, 0) && tid == 0) {
            atomicOr(&p.sc.words[2], TOED_FLAG_TIMEOUT);
            mbar_wait(bar, 0);  // once more: nothing may be in flight towards an exited CTA's memory
        }
        const int n = min(kEdChunk, total - c0);
        Staged e = {};
        int pos = -1;
        if (tid < n) {
            const int2 l = sList[tid];
            if (l.y < cap && l.x < p.sc.staging_cap && TOED_IN_BOUNDS(l.x >= 0 && l.y >= 0, p.sc.words)) {
                pos = l.y;
                e = load_staged(p.sc, l.x);
            }
        }
        bool odd = (e.idx - e.idx / W2 * W2) & 1;
        Subpixel at = {};
        if (QAD) {
            if (pos >= 0) at = subpixel_of(e, W2, p.hyb != 0);
            odd = at.X1 & 1;
        }
        const unsigned b0 = __ballot_sync(0xffffffffu, pos >= 0 && !odd), b1 = __ballot_sync(0xffffffffu, pos >= 0 && odd);
        if (lane == 0) s_warp[wid] = __popc(b0) << 16 | __popc(b1);
        __syncthreads();
        int n0 = 0, before = 0;
#pragma unroll
        for (int w = 0; w < kEdThreads / 32; ++w) {
            n0 += s_warp[w] >> 16;
            if (w < wid) before += s_warp[w];
        }
        n0 = (n0 + 31) & ~31;  // where the odd ones start
        if (pos >= 0) {
            const unsigned lt_ = (1u << lane) - 1u;
            const int to = odd ? n0 + (before & 0xffff) + __popc(b1 & lt_) : (before >> 16) + __popc(b0 & lt_);
            if (TOED_IN_BOUNDS(to < kEdThreads, p.sc.words)) {
                sRec[to] = e;
                sPos[to] = pos;
                if (QAD) sAt[to] = at;
            }
        }
        __syncthreads();
        pos = sPos[tid];
        if (__any_sync(0xffffffffu, pos >= 0)) {
            e = sRec[pos >= 0 ? tid : (wid * 32)];  // a warp's first slot is used if any is
            const int Gr = e.idx / W2, Gc = e.idx - Gr * W2;
            [[maybe_unused]] const int a = Gr & 1, b = Gc & 1;
            float d7[7], gx = e.gx, gy = e.gy;
            if constexpr (QAD) {
                const Subpixel q = sAt[pos >= 0 ? tid : (wid * 32)];
                const float* win = sPix + ((q.Y1 >> 1) - y0 + 1) * TP + (q.X1 >> 1) - sc * kInner + 1 + shift;
                if (!TOED_IN_BOUNDS(staged(win, NT + 2), p.sc.words)) win = sPix;
                float d9[9];
                if (32 * wid < n0)
                    subpixel9<R, 1>(win, q.Y1, (float)q.tx, (float)q.ty, sTab, p.taps, d9);
                else
                    subpixel9<R, 0>(win, q.Y1, (float)q.tx, (float)q.ty, sTab, p.taps, d9);
                gx = d9[0];
                gy = d9[1];
#pragma unroll
                for (int f = 0; f < 7; ++f) d7[f] = d9[f + 2];
            } else {
                const float* win = sPix + ((Gr >> 1) - y0) * TP + (Gc >> 1) - sc * kInner + shift;
                if (!TOED_IN_BOUNDS(staged(win, NT), p.sc.words)) win = sPix;
                if (32 * wid < n0)
                    window7<R, 0>(win, a, sTab + (a ? 2 : b) * NT, p.taps, d7);
                else
                    window7<R, 1>(win, a, sTab + (a ? 2 : b) * NT, p.taps, d7);
            }
            float tix, tiy, ori;
            to_vec32(gx, gy, d7, &tix, &tiy);
            const Fitted ft =
                fit_edgel(e, p.nms_to ? tix : e.gx, p.nms_to ? tiy : e.gy, p.nms_to != 0, p.hyb != 0, Gr, Gc);
            if (p.hyb) {
                ori = (tix == 0.f && tiy == 0.f) ? __int_as_float(0x7fc00000) : atan2f(tix, -tiy);
                if (pos >= 0 && cancels(gx, gy, d7, tix, tiy)) {
                    sPos[tid] = -2 - pos;
                    const int f = atomicAdd(&sFlags, 1);
                    if (TOED_IN_BOUNDS(f < kEdThreads, p.sc.words)) sFlag[f] = (unsigned char)tid;
                }
            } else {
                const float fxx = d7[0], fxy = d7[1], fyy = d7[2], fxxy = d7[3], fxyy = d7[4], fxxx = d7[5], fyyy = d7[6];
                tix = gx * (2.f * fxx * fxx + 2.f * fxy * fxy) + gy * (2.f * fxx * fxy + 2.f * fyy * fxy) +
                      2.f * gx * gy * fxxy + gy * gy * fxyy + gx * gx * fxxx;
                tiy = gx * (2.f * fxx * fxy + 2.f * fyy * fxy) + gy * (2.f * fyy * fyy + 2.f * fxy * fxy) +
                      2.f * gx * gy * fxyy + gx * gx * fxxy + gy * gy * fyyy;
                ori = (tix == 0.f && tiy == 0.f) ? __int_as_float(0x7fc00000) : atan2f(tix, -tiy);
            }
            if (pos >= 0) write_edgel(p, im, pos, ft.x, ft.y, ori, ft.str, e.idx);
        }
        __syncthreads();
        // the orientations to be formed again in FP64, all warps' alike: each
        // takes up to kRefineMost, then their orientations at once
        const int nf = sFlags;
        for (int f0 = wid; f0 < nf; f0 += kRefineMost * (kEdThreads / 32)) {
            int m = 0;
            for (int f = f0; f < nf && m < kRefineMost; f += kEdThreads / 32, ++m) {
                if constexpr (QAD) {
                    const Subpixel q = sAt[sFlag[f]];
                    const float* win = sPix + ((q.Y1 >> 1) - y0 + 1) * TP + (q.X1 >> 1) - sc * kInner + 1 + shift;
                    if (TOED_IN_BOUNDS(staged(win, NT + 2), p.sc.words))
                        refine_subpixel(p, win, TP, q.X1, q.Y1, q.tx, q.ty, lane, sD64[wid][m]);
                } else {
                    const int idx = sRec[sFlag[f]].idx;
                    const int Gr = idx / W2, Gc = idx - Gr * W2;
                    const float* win = sPix + ((Gr >> 1) - y0) * TP + (Gc >> 1) - sc * kInner + shift;
                    if (TOED_IN_BOUNDS(staged(win, NT), p.sc.words))
                        refine_edgel(p, win, TP, Gr & 1, Gc & 1, lane, sD64[wid][m]);
                }
            }
            __syncwarp();
            if (lane < m) {
                const int pos = -2 - sPos[sFlag[f0 + lane * (kEdThreads / 32)]];
                const float ori = orientation64(sD64[wid][lane]);
                if (TOED_IN_BOUNDS(pos >= 0 && pos < cap, p.sc.words)) {
                    if (p.out_f64)
                        static_cast<double*>(im.out)[4LL * pos + 2] = (double)ori;
                    else
                        static_cast<float*>(im.out)[4LL * pos + 2] = ori;
                }
            }
            __syncwarp();
        }
        __syncthreads();  // the next chunk overwrites the lists
    }
    if (im.host_out) band_done(p, im, ty, s_warp);
}

struct EdEntry {
    const void* func;
    size_t smem;  // at p.ed_rows
};

template <bool QAD>
static EdEntry edgels_entry(int radius, int rows)
{
    switch (radius) {
#define TOED_ED_CASE(R) \
    case R: return {(const void*)fin_edgels<R, QAD>, EdCfg<R, QAD>::smem(rows)};
        TOED_ED_CASE(1) TOED_ED_CASE(2) TOED_ED_CASE(3) TOED_ED_CASE(4) TOED_ED_CASE(5) TOED_ED_CASE(6)
        TOED_ED_CASE(7) TOED_ED_CASE(8) TOED_ED_CASE(9) TOED_ED_CASE(10) TOED_ED_CASE(11) TOED_ED_CASE(12)
#undef TOED_ED_CASE
    default: return {nullptr, 0};
    }
}

template <bool QAD>
static cudaError_t prepare_edgels_as(int radius)
{
    const EdEntry ent = edgels_entry<QAD>(radius, kEdRowsMax);
    if (!ent.func) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(ent.func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ent.smem);
}

template <bool QAD>
static cudaError_t launch_edgels_as(const BatchParams& p, cudaStream_t stream)
{
    const EdEntry ent = edgels_entry<QAD>(p.radius, p.ed_rows);
    if (!ent.func) return cudaErrorInvalidValue;
    void* args[] = {const_cast<BatchParams*>(&p)};
    return launch_after(ent.func, dim3(p.n_ed), dim3(kEdThreads), args, ent.smem, stream);
}

}  // namespace toed
