// toed_backward.cu -- adjoint of the fused detection with the selection
// frozen: gradients of every edgel's [x, y, orientation, strength] with
// respect to the image pixels and sigma.  The reference has no backward; the
// forward whose adjoint this is follows cpu_toed.cpp:128-545.
//
// One kernel, bw_adjoint<R>.  A CTA owns an equal run of edgels (sized so that
// the launch is one wave), orders a chunk of them by 2x column parity and gives
// its warps rounds of up to 32:
//   1. a thread per edgel evaluates, from the image, the nine derivatives at
//      the edgel's 2x-grid point P and Ix, Iy at the eight points around it,
//      each with its d/dsigma, in one pass over the window's rows: the warp
//      copies row after row of the 32 windows to shared memory (asynchronous
//      copies of aligned groups of four pixels, a row ahead), each thread
//      filters its row at the three columns with compile-time taps and weights
//      the responses with the y taps of the three rows;
//   2. it runs the chain rule through the peak fit and the third-order
//      orientation of its (frozen) sector (the peak fit's sums and the vector
//      in FP64) and accumulates dL/dsigma;
//   3. a warp per edgel adds the separable cotangent windows
//      sum_f X_f(q) V_f(p) of its five points onto the pixel gradient with
//      float reductions in global memory (cleared first by bw_clear, one
//      launch for the whole batch).
// What bounds it: instruction issue (65 % of the slots while an SM is busy, 16
// warps of 128 registers each; DRAM under 2 %), about 110 of 200 us in the row
// filters, 70 in the scatter.  At r = 8, 134,000 edgels of six 777 x 1001
// images: 1000 warp instructions an edgel and 203 us with the clearing, 2270
// and 384 us when a warp evaluated one edgel at a time, a lane per window
// column with the sums through shared memory.  Tried on the way: single pixels
// copied (4 bytes each: 293 us), borders and interior in one round (260), three
// CTAs an SM with 168 registers (245).  bw_adjoint starts while bw_clear runs
// and waits for it before its first addition (412 edgels of a 64 x 64 image:
// 16.5 us one after the other with a memset of dL/dsigma, 12.3 so).
// Reductions from different edgels land in an unspecified order, so the
// pixel gradient is reproducible to float rounding, not bit for bit.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>

#include "toed_common.cuh"
#include "toed_groups.h"
#include "toed_internal.h"

namespace toed {

constexpr int kBwAdjThreads = 128;

struct BwImage {
    const void* src;
    long long pitch;
    const int* gidx;
    const void* gout;
    float* gpix;
    int H, W, dtype, n;
    int edgel_base;
};

struct BwParams {
    float tap[16][kMaxTaps];  // 0..3 G Gx Gxx Gxxx, 4..7 shifted by 1/2, 8..15 their d/dsigma
    float4 sum_lo[3], sum_hi[3];  // the taps' sums by variant (T, F, S): (G, Gx, dG, dGx), (Gxx, Gxxx, dGxx, dGxxx)
    float ill_curve;  // kIllCurve / sigma^2, the scale of a peak's curvature
    int r;
    int out_f64;
    int first;  // clears dL/dsigma
    int n_img;
    int n_edgels;
    int per_cta;  // edgels per CTA: all CTAs of the launch resident at once
    double* gsig;
    BwImage img[kBatchMax];
};

__device__ __forceinline__ void variants(int rho, int kap, int* xv, int* yv)
{
    const int a = rho & 1, b = kap & 1;
    *xv = (a == 0 && b == 0) ? 0 : (b ? 2 : 1);
    *yv = (a == 0 && b == 0) ? 0 : (a ? 2 : 1);
}

__device__ __forceinline__ float pix(const BwImage& im, int y, int x)
{
    if ((unsigned)y >= (unsigned)im.H || (unsigned)x >= (unsigned)im.W) return 0.f;
    const long long o = (long long)y * im.pitch + x;
    return im.dtype == TOED_U8 ? (float)__ldg((const unsigned char*)im.src + o) : __ldg((const float*)im.src + o);
}

constexpr int kBwWarps = kBwAdjThreads / 32;
constexpr int kBwChunk = 2 * kBwAdjThreads;  // edgels ordered at a time
// Edgels a warp up to which it evaluates one at a time: the pass over the rows
// takes as long for one as for 32 (412 edgels of a 64 x 64 image, sigma 1: 41 us
// a call; 2,108 of 200 x 300, sigma 1.5: 52 us, one at a time 37).
constexpr int kBwFew = 6;

template <int R>
struct BwCfg {
    static constexpr int NT = 2 * R + 3, NTP = NT + 4, NU = NT + 2;  // taps, padded taps, side of the union window
    static constexpr int NUP = (NU + 3) / 4 * 4;
    static constexpr int RECW = 20;                                  // words of an edgel's cotangent record
    static constexpr int kRed = 33, kVals = 34;                      // fallback: column sums of 34 values
    // a window row is staged as the CH aligned groups of four pixels that cover
    // it, wherever it starts; rows lie ROW floats apart (an odd number of
    // groups: a thread per row reads them without bank conflicts)
    static constexpr int CH = (NU + 6) / 4, ROW = 4 * (CH | 1);
    // per warp: two buffers of 32 windows' rows; phase 3's records and
    // y-vectors, or the fallback's sums, over them
    static constexpr size_t rows_b = sizeof(float) * 2 * 32 * ROW;
    static constexpr size_t p3_b = sizeof(float) * 32 * RECW + sizeof(float4) * 3 * NUP;
    static constexpr size_t fb_b = sizeof(float) * (kVals * kRed + kVals + 2);
    static constexpr size_t max3(size_t a, size_t b, size_t c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }
    static constexpr size_t warp_b = (max3(rows_b, p3_b, fb_b) + 15) / 16 * 16;
    static constexpr size_t tab_b = sizeof(float4) * 2 * 3 * NTP;
    static constexpr size_t off_warp = tab_b, off_list = off_warp + kBwWarps * warp_b;
    static constexpr size_t smem = off_list + sizeof(int) * (kBwChunk + 64);
    // above r = 8 the wider rows need more than 128 registers (r = 12, 123,000
    // edgels: 728 us with two CTAs an SM, 382 with three)
    static constexpr int MINB = R <= 8 ? 4 : 3;
};

// Tap tables with two zero entries on each side: entry k + 2 holds tap k, so
// a window offset by -1..+1 pixel (the points around P) indexes them without
// bounds tests.  Per variant T, F, S: lo = (G, Gx, dG, dGx), hi = (Gxx, Gxxx,
// dGxx, dGxxx), d the derivative with respect to sigma.
template <int R>
__device__ __forceinline__ void build_tables(const BwParams& p, float4* lo, float4* hi)
{
    constexpr int NT = BwCfg<R>::NT, NTP = BwCfg<R>::NTP;
    for (int i = threadIdx.x; i < 3 * NTP; i += blockDim.x) {
        const int v = i / NTP, k = i - v * NTP - 2;
        const int f = (v == 2) ? 4 : 0;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), s = a;
        if (k >= 0 && k < NT && !(v == 0 && (k == 0 || k == NT - 1))) {
            a = make_float4(p.tap[f][k], p.tap[f + 1][k], p.tap[8 + f][k], p.tap[9 + f][k]);
            s = make_float4(p.tap[f + 2][k], p.tap[f + 3][k], p.tap[10 + f][k], p.tap[11 + f][k]);
        }
        lo[i] = a;
        hi[i] = s;
    }
}

// One window row's responses (G, Gx) and their d/dsigma -- HI: (Gxx, Gxxx) --
// at window column C: t truncated, e what the two end taps add (whole
// columns), or shifted.  Even filters over mirrored sums, odd ones over
// mirrored differences, which low and high share.
template <int R, int C, bool HI>
__device__ __forceinline__ void resp_whole(const float* v, const float (&tap)[16][kMaxTaps], float4& t, float4& e)
{
    constexpr int f = HI ? 2 : 0;
    t = make_float4(v[C] * tap[f][R + 1], 0.f, v[C] * tap[8 + f][R + 1], 0.f);
#pragma unroll
    for (int q = 1; q <= R; ++q) {
        const float sm = v[C - q] + v[C + q], df = v[C - q] - v[C + q];
        t.x = fmaf(sm, tap[f][q + R + 1], t.x);
        t.y = fmaf(df, tap[f + 1][q + R + 1], t.y);
        t.z = fmaf(sm, tap[8 + f][q + R + 1], t.z);
        t.w = fmaf(df, tap[9 + f][q + R + 1], t.w);
    }
    const float sm = v[C - R - 1] + v[C + R + 1], df = v[C - R - 1] - v[C + R + 1];
    e.x = sm * tap[f][2 * R + 2];
    e.y = df * tap[f + 1][2 * R + 2];
    e.z = sm * tap[8 + f][2 * R + 2];
    e.w = df * tap[9 + f][2 * R + 2];
}
template <int R, int C, bool HI>
__device__ __forceinline__ float4 resp_shift(const float* v, const float (&tap)[16][kMaxTaps])
{
    constexpr int f = HI ? 6 : 4;
    const float vl = v[C - R - 1];  // the tap without a mirror image
    float4 s = make_float4(vl * tap[f][2 * R + 2], vl * tap[f + 1][2 * R + 2], vl * tap[8 + f][2 * R + 2],
                           vl * tap[9 + f][2 * R + 2]);
#pragma unroll
    for (int q = 0; q <= R; ++q) {
        const float sm = v[C - q] + v[C + 1 + q], df = v[C - q] - v[C + 1 + q];
        s.x = fmaf(sm, tap[f][q + R + 1], s.x);
        s.y = fmaf(df, tap[f + 1][q + R + 1], s.y);
        s.z = fmaf(sm, tap[8 + f][q + R + 1], s.z);
        s.w = fmaf(df, tap[9 + f][q + R + 1], s.w);
    }
    return s;
}
__device__ __forceinline__ float4 add_scaled(float4 t, float s, float4 e)
{
    return make_float4(fmaf(s, e.x, t.x), fmaf(s, e.y, t.y), fmaf(s, e.z, t.z), fmaf(s, e.w, t.w));
}

// fx, fy and their d/dsigma of one point: x responses (G, Gx, dG, dGx) of a
// row times its y taps (G, Gy, dG, dGy).
__device__ __forceinline__ void add_point(float4 x, float4 y, float (&n)[4])
{
    n[0] = fmaf(x.y, y.x, n[0]);
    n[1] = fmaf(x.x, y.y, n[1]);
    n[2] = fmaf(x.w, y.x, fmaf(x.y, y.z, n[2]));
    n[3] = fmaf(x.z, y.y, fmaf(x.x, y.w, n[3]));
}

// Per edgel: the nine derivatives at P (fx fy fxx fxy fyy fxxy fxyy fxxx fyyy),
// their d/dsigma, and (fx, fy, d/dsigma) at the points around it, row by row:
// 0..2 row above (columns -1, 0, 1), 3, 4 same row (-1, 1), 5..7 row below.
struct BwValues {
    float d[9], s[9], n[8][4];
    float top;  // the magnitude of the window's pixels
};

// One row's x responses at P (x: low, h: high) times its y taps, onto P's values.
__device__ __forceinline__ void add_center(float4 x, float4 h, float4 y, float4 g, BwValues& o)
{
    o.d[0] = fmaf(x.y, y.x, o.d[0]);  // fx   (Gx, G)
    o.d[1] = fmaf(x.x, y.y, o.d[1]);  // fy   (G, Gy)
    o.d[2] = fmaf(h.x, y.x, o.d[2]);  // fxx  (Gxx, G)
    o.d[3] = fmaf(x.y, y.y, o.d[3]);  // fxy  (Gx, Gy)
    o.d[4] = fmaf(x.x, g.x, o.d[4]);  // fyy  (G, Gyy)
    o.d[5] = fmaf(h.x, y.y, o.d[5]);  // fxxy (Gxx, Gy)
    o.d[6] = fmaf(x.y, g.x, o.d[6]);  // fxyy (Gx, Gyy)
    o.d[7] = fmaf(h.y, y.x, o.d[7]);  // fxxx (Gxxx, G)
    o.d[8] = fmaf(x.x, g.y, o.d[8]);  // fyyy (G, Gyyy)
    o.s[0] = fmaf(x.w, y.x, fmaf(x.y, y.z, o.s[0]));
    o.s[1] = fmaf(x.z, y.y, fmaf(x.x, y.w, o.s[1]));
    o.s[2] = fmaf(h.z, y.x, fmaf(h.x, y.z, o.s[2]));
    o.s[3] = fmaf(x.w, y.y, fmaf(x.y, y.w, o.s[3]));
    o.s[4] = fmaf(x.z, g.x, fmaf(x.x, g.z, o.s[4]));
    o.s[5] = fmaf(h.z, y.y, fmaf(h.x, y.w, o.s[5]));
    o.s[6] = fmaf(x.w, g.x, fmaf(x.y, g.z, o.s[6]));
    o.s[7] = fmaf(h.w, y.x, fmaf(h.y, y.z, o.s[7]));
    o.s[8] = fmaf(x.z, g.y, fmaf(x.x, g.w, o.s[8]));
}

// A window of the constant b onto the values: what evaluating the window less
// b leaves out.
__device__ __forceinline__ void add_constant(const BwParams& p, int a, int b_odd, float b, BwValues& o)
{
    auto scaled = [&](float4 t) { return make_float4(b * t.x, b * t.y, b * t.z, b * t.w); };
    // x and y variants at P, at its row's neighbours, at its column's and at the diagonal ones
    const int T = 0, F = 1, S = 2;
    const int xp = b_odd ? S : a ? F : T, yp = a ? S : b_odd ? F : T;
    const int xs = b_odd ? (a ? F : T) : S, ys = a ? S : b_odd ? T : F;
    const int xc = b_odd ? S : a ? T : F, yc = a ? (b_odd ? F : T) : S;
    const int xd = b_odd ? (a ? T : F) : S, yd = a ? (b_odd ? T : F) : S;
    add_center(scaled(p.sum_lo[xp]), scaled(p.sum_hi[xp]), p.sum_lo[yp], p.sum_hi[yp], o);
    const float4 s = scaled(p.sum_lo[xs]), c = scaled(p.sum_lo[xc]), d = scaled(p.sum_lo[xd]);
    const float4 us = p.sum_lo[ys], uc = p.sum_lo[yc], ud = p.sum_lo[yd];
    add_point(s, us, o.n[3]);
    add_point(s, us, o.n[4]);
    add_point(c, uc, o.n[1]);
    add_point(c, uc, o.n[6]);
    add_point(d, ud, o.n[0]);
    add_point(d, ud, o.n[2]);
    add_point(d, ud, o.n[5]);
    add_point(d, ud, o.n[7]);
}

// One window row, B the parity of P's 2x column; lo/hi: the tap tables, the
// row's entry of the offset-0 taps at [v * NTP + at].
template <int R, int B>
__device__ __forceinline__ void eval_row(const float (&v)[BwCfg<R>::NU], const BwParams& p, int a,
                                         const float4* __restrict__ lo, const float4* __restrict__ hi, BwValues& o)
{
    using C = BwCfg<R>;
    constexpr int NTP = C::NTP, M = R + 2;  // pixel j is window column M
    // x responses: P's column, for its row's parity a (xp) and the other (xq);
    // the columns left and right, likewise (l0, r0 for a; l1, r1)
    float4 xp, xq, xh, l0, l1, r0, r1;
    const float fa = a ? 1.f : 0.f, fb = 1.f - fa;  // whole columns: full filters in odd 2x rows, truncated in even ones
    if (B == 0) {
        float4 t, e;
        resp_whole<R, M, false>(v, p.tap, t, e);
        xp = add_scaled(t, fa, e);
        xq = add_scaled(t, fb, e);
        resp_whole<R, M, true>(v, p.tap, t, e);
        xh = add_scaled(t, fa, e);
        l0 = l1 = resp_shift<R, M - 1, false>(v, p.tap);
        r0 = r1 = resp_shift<R, M, false>(v, p.tap);
    } else {
        xp = xq = resp_shift<R, M, false>(v, p.tap);
        xh = resp_shift<R, M, true>(v, p.tap);
        float4 t, e;
        resp_whole<R, M, false>(v, p.tap, t, e);
        l0 = add_scaled(t, fa, e);
        l1 = add_scaled(t, fb, e);
        resp_whole<R, M + 1, false>(v, p.tap, t, e);
        r0 = add_scaled(t, fa, e);
        r1 = add_scaled(t, fb, e);
    }
    // the rows' scale: their smooth responses and every third pixel
    o.top = fmaxf(o.top, fabsf(xp.x));
#pragma unroll
    for (int t = 0; t < C::NU; t += 3) o.top = fmaxf(o.top, fabsf(v[t]));
    // y taps: P's row on its column and beside it, the rows above and below
    // (pixel row offset -1 or 0, 0 or 1) likewise
    const int vp = a ? 2 : B, vs = a ? 2 : 1 - B;  // variants on even columns T, on odd ones F; shifted in odd rows
    const int up = a ? 0 : -1, dn = a ? 1 : 0, wp = a ? B : 2, ws = a ? 1 - B : 2;
    const float4 yp = lo[vp * NTP], yh = hi[vp * NTP], ys = lo[vs * NTP];
    add_point(l0, ys, o.n[3]);
    add_point(r0, ys, o.n[4]);
    {
        const float4 y = lo[wp * NTP + up], z = lo[ws * NTP + up];
        add_point(l1, z, o.n[0]);
        add_point(xq, y, o.n[1]);
        add_point(r1, z, o.n[2]);
    }
    {
        const float4 y = lo[wp * NTP + dn], z = lo[ws * NTP + dn];
        add_point(l1, z, o.n[5]);
        add_point(xq, y, o.n[6]);
        add_point(r1, z, o.n[7]);
    }
    add_center(xp, xh, yp, yh, o);
}

// Sum over the union columns of one value, in a fixed order.
__device__ __forceinline__ float column_sum(const float* red_k, int n)
{
    float a = 0.f, b = 0.f;
    int t = 0;
    for (; t + 1 < n; t += 2) {
        a += red_k[t];
        b += red_k[t + 1];
    }
    if (t < n) a += red_k[t];
    return a + b;
}

// The values of one ill-conditioned edgel by a whole warp: lane c holds union
// column j-R-2+c, contracts it with each point's y taps, multiplies by its x
// taps, and the columns are summed in a fixed order.  An edgel whose gradient
// lies on a sector's border to within rounding, or whose peak fit or
// third-order vector nearly vanishes, amplifies the rounding of these sums a
// thousandfold, so for these few the order of summation is the definition.
// val[0..17]: the derivatives at P and their d/dsigma; val[18..33]: fx, fy,
// dfx/dsigma, dfy/dsigma at A+, D+, A-, D-; returns the sector (bit 0 |fx| >=
// |fy|, bit 1 fx >= 0, bit 2 fy >= 0).
template <int R>
__device__ __noinline__ int eval_edgel_warp(const BwImage& im, int rho, int kap, int lane, const float4* lo, const float4* hi,
                                            float* buf)
{
    using C = BwCfg<R>;
    constexpr int NT = C::NT, NTP = C::NTP, NU = C::NU;
    float(*red)[C::kRed] = reinterpret_cast<float(*)[C::kRed]>(buf);
    float* val = buf + C::kVals * C::kRed;
    const int i = rho >> 1, j = kap >> 1, x = j - R - 2 + lane;
    const int lc = lane < NU ? lane : NU - 1;  // lanes past the window add nothing
    float v[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) v[u] = lane < NU ? pix(im, i - R - 2 + u, x) : 0.f;
    // A point's y contractions (G, Gy and their d/dsigma) depend on its y taps
    // and row alone: points that share both share the sums (P's is point 4)
    float4 sums[5];
    int keys[5];
    {
        int xv, yv;
        variants(rho, kap, &xv, &yv);
        const float4 *YA = lo + yv * NTP + NT + 2, *YS = hi + yv * NTP + NT + 2;
        float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f, s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        keys[4] = yv * 4 + 1;
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            const float4 a = YA[-u], h = YS[-u];
            c0 = fmaf(v[u], a.x, c0); c1 = fmaf(v[u], a.y, c1);
            s0 = fmaf(v[u], a.z, s0); s1 = fmaf(v[u], a.w, s1);
            c2 = fmaf(v[u], h.x, c2); c3 = fmaf(v[u], h.y, c3);
            s2 = fmaf(v[u], h.z, s2); s3 = fmaf(v[u], h.w, s3);
        }
        sums[4] = make_float4(c0, c1, s0, s1);
        if (lane < NU) {
            const float4 x0 = lo[xv * NTP + NT + 2 - lc], x1 = hi[xv * NTP + NT + 2 - lc];
            const float4 xa = make_float4(x0.x, x0.y, x1.x, x1.y), xs = make_float4(x0.z, x0.w, x1.z, x1.w);
            red[0][lane] = xa.y * c0;  red[9][lane] = fmaf(xs.y, c0, xa.y * s0);    // fx   (Gx, G)
            red[1][lane] = xa.x * c1;  red[10][lane] = fmaf(xs.x, c1, xa.x * s1);   // fy   (G, Gy)
            red[2][lane] = xa.z * c0;  red[11][lane] = fmaf(xs.z, c0, xa.z * s0);   // fxx  (Gxx, G)
            red[3][lane] = xa.y * c1;  red[12][lane] = fmaf(xs.y, c1, xa.y * s1);   // fxy  (Gx, Gy)
            red[4][lane] = xa.x * c2;  red[13][lane] = fmaf(xs.x, c2, xa.x * s2);   // fyy  (G, Gyy)
            red[5][lane] = xa.z * c1;  red[14][lane] = fmaf(xs.z, c1, xa.z * s1);   // fxxy (Gxx, Gy)
            red[6][lane] = xa.y * c2;  red[15][lane] = fmaf(xs.y, c2, xa.y * s2);   // fxyy (Gx, Gyy)
            red[7][lane] = xa.w * c0;  red[16][lane] = fmaf(xs.w, c0, xa.w * s0);   // fxxx (Gxxx, G)
            red[8][lane] = xa.x * c3;  red[17][lane] = fmaf(xs.x, c3, xa.x * s3);   // fyyy (G, Gyyy)
        }
    }
    __syncwarp();
    if (lane < 18) val[lane] = column_sum(red[lane], NU);
    __syncwarp();
    const float fx = val[0], fy = val[1];
    const bool xmaj = fabsf(fx) >= fabsf(fy);
    const int sx = fx >= 0.f ? 1 : -1, sy = fy >= 0.f ? 1 : -1;
    const int ar = xmaj ? 0 : sy, ac = xmaj ? sx : 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int dr = (q & 1) ? sy : ar, dc = (q & 1) ? sx : ac;
        const int pr = q < 2 ? rho + dr : rho - dr, pc = q < 2 ? kap + dc : kap - dc;
        int xv, yv;
        variants(pr, pc, &xv, &yv);
        const int di = (pr >> 1) - i;
        keys[q] = yv * 4 + di + 1;
        bool have = false;  // (warp-uniform)
#pragma unroll
        for (int k = 4; k >= 0; --k)
            if ((k == 4 || k < q) && !have && keys[k] == keys[q]) {
                sums[q] = sums[k];
                have = true;
            }
        if (!have) {
            const float4* Y = lo + yv * NTP + NT + 2 + di;
            float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                const float4 y = Y[-u];
                c.x = fmaf(v[u], y.x, c.x);
                c.y = fmaf(v[u], y.y, c.y);
                c.z = fmaf(v[u], y.z, c.z);
                c.w = fmaf(v[u], y.w, c.w);
            }
            sums[q] = c;
        }
        if (lane < NU) {
            const float4 c = sums[q], xa = lo[xv * NTP + NT + 2 + ((pc >> 1) - j) - lc];
            red[18 + 4 * q][lane] = xa.y * c.x;  // fx (Gx, G)
            red[19 + 4 * q][lane] = xa.x * c.y;  // fy (G, Gy)
            red[20 + 4 * q][lane] = fmaf(xa.w, c.x, xa.y * c.z);
            red[21 + 4 * q][lane] = fmaf(xa.z, c.y, xa.x * c.w);
        }
    }
    __syncwarp();
    if (lane < 16) val[18 + lane] = column_sum(red[18 + lane], NU);
    __syncwarp();
    return (xmaj ? 1 : 0) | (sx > 0 ? 2 : 0) | (sy > 0 ? 4 : 0);
}

// True where rounding in the values decides the result (see eval_edgel_warp):
// a gradient on a sector's border; a neighbour's gradient small against the
// pixels' magnitude top, to which all rounding is relative; a peak flatter than
// kIllFit of that and than kIllCurve m / sigma^2 (a median edge has twice the
// latter); a third-order vector below kIllVector of its terms' magnitudes.  With
// these limits the gradients of 72 noisy images (777 x 1001, sigma 2) differ by
// up to 1e-6 of their norm from those all summed in the fixed order, without
// them by up to 1.4e-4; few edgels pay (6 of 219 us; with every faint edgel's
// cotangents used, 243 us, but 388 without kIllCurve).  An edgel whose cotangents are all zero is
// not used: zero times a finite gradient.
constexpr float kIllStrength = 3e-4f, kIllFit = 1e-3f, kIllCurve = 0.12f, kIllVector = 0.25f;

__device__ __forceinline__ bool ill_conditioned(const BwValues& o, const float (&nv)[4][4], bool xmaj, bool used,
                                                float curve)
{
    const float fx = o.d[0], fy = o.d[1], fxx = o.d[2], fxy = o.d[3], fyy = o.d[4], fxxy = o.d[5], fxyy = o.d[6],
                fxxx = o.d[7], fyyy = o.d[8];
    const float m = sqrtf(fx * fx + fy * fy);
    float M[4], low = m;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        M[q] = sqrtf(nv[q][0] * nv[q][0] + nv[q][1] * nv[q][1]);
        low = fminf(low, M[q]);
    }
    const float t = xmaj ? fabsf(fy / fx) : fabsf(fx / fy);
    const float den = (M[0] + M[2]) * (1.f - t) + (M[1] + M[3]) * t - 2.f * m;
    // the third-order vector against the sum of its terms' magnitudes
    const float ax = fabsf(fx), ay = fabsf(fy), bxx = fabsf(fxx), bxy = fabsf(fxy), byy = fabsf(fyy);
    const float TIx = fx * (2 * fxx * fxx + 2 * fxy * fxy) + fy * (2 * fxx * fxy + 2 * fyy * fxy) + 2 * fx * fy * fxxy +
                      fy * fy * fxyy + fx * fx * fxxx;
    const float TIy = fx * (2 * fxx * fxy + 2 * fyy * fxy) + fy * (2 * fyy * fyy + 2 * fxy * fxy) + 2 * fx * fy * fxyy +
                      fx * fx * fxxy + fy * fy * fyyy;
    const float all = (ax + ay) * (2 * bxx * bxx + 2 * byy * byy + 2 * bxy * bxy + 2 * bxy * (bxx + byy)) +
                      (ax * ax + ay * ay) * (fabsf(fxxx) + fabsf(fyyy) + fabsf(fxxy) + fabsf(fxyy));
    const float tol = 2.6e-6f * o.top;
    // (negated: a value that is not a number counts as ill-conditioned)
    return !(low > kIllStrength * o.top && fabsf(den) > 0.f &&
             (!used || (fabsf(ax - ay) > tol && ax > tol && ay > tol && fabsf(den) > fminf(kIllFit * o.top, curve * m) &&
                        fabsf(TIx) + fabsf(TIy) > kIllVector * all)));
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
          "l"(reinterpret_cast<unsigned long long&>(c)));
    return reinterpret_cast<float2&>(d);
}

// Scatter of one edgel's cotangents onto the pixel gradient, by a whole
// warp: grad I(u) += sum over the five points and their filters of
// X_f(q) V_f(p), V_f = the y taps weighted by the point's cotangents.  All
// five windows lie in the (NT+2) x (NT+2) union window around the edgel's
// pixel.  Lane r stages the 12 y-vectors of union row r in shared memory
// (P's four, two per neighbour); then lane (rg, cg) takes the rows rg + 4 m
// and the columns cg + 8 k, whose x taps it holds -- 4 x 8 pixels an
// instruction keep 32 lanes in work for the 21 x 21 window of r = 8, where a
// lane per column kept 21 -- and adds each pixel with a reduction
// (red.global.add.f32).  The 12 products are six packed ones (f32x2).  The
// grid pixels outside the image are the zero padding and receive nothing.
// g: the cotangent record; its last three words hold the points' table
// entries, a byte each (see tap_entries).
template <int R>
__device__ __forceinline__ void scatter_edgel_warp(const BwImage& im, int rho, int kap, int lane, const float4* lo,
                                                   const float4* hi, const float* g, float4 (*sV)[3])
{
    using C = BwCfg<R>;
    constexpr int NU = C::NU, KC = (NU + 7) / 8, KR = C::NUP / 4;
    float gv[20];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const float4 t = reinterpret_cast<const float4*>(g)[q];
        gv[4 * q] = t.x;
        gv[4 * q + 1] = t.y;
        gv[4 * q + 2] = t.z;
        gv[4 * q + 3] = t.w;
    }
    const unsigned e0 = __float_as_uint(gv[17]), e1 = __float_as_uint(gv[18]), e2 = __float_as_uint(gv[19]);
    const unsigned xe[5] = {e0 & 255u, e0 >> 16 & 255u, e1 & 255u, e1 >> 16 & 255u, e2 & 255u};
    const unsigned ye[5] = {e0 >> 8 & 255u, e0 >> 24, e1 >> 8 & 255u, e1 >> 24, e2 >> 8 & 255u};
    if (lane < C::NUP) {
        const int l = lane < NU ? lane : NU - 1;  // (rows past the window: read, not added)
        const float4 y = lo[ye[0] - l], h = hi[ye[0] - l];
        sV[lane][0] = make_float4(gv[1] * y.y + gv[4] * h.x + gv[8] * h.y,  // G    x (fy, fyy, fyyy)
                                  gv[0] * y.x + gv[3] * y.y + gv[6] * h.x,  // Gx   x (fx, fxy, fxyy)
                                  gv[2] * y.x + gv[5] * y.y,                // Gxx  x (fxx, fxxy)
                                  gv[7] * y.x);                             // Gxxx x fxxx
        float2 n[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // G x fy, Gx x fx at the neighbour
            const float2 t = *reinterpret_cast<const float2*>(lo + (ye[q + 1] - l));
            n[q] = make_float2(gv[10 + 2 * q] * t.y, gv[9 + 2 * q] * t.x);
        }
        sV[lane][1] = make_float4(n[0].x, n[0].y, n[1].x, n[1].y);
        sV[lane][2] = make_float4(n[2].x, n[2].y, n[3].x, n[3].y);
    }
    const int cg = lane & 7, rg = lane >> 3;
    const int x0 = (kap >> 1) - R - 2 + cg, y0 = (rho >> 1) - R - 2 + rg;
    float2 xt[KC][6];
    bool okx[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) {
        const int l = cg + 8 * k;
        okx[k] = l < NU && (unsigned)(x0 + 8 * k) < (unsigned)im.W;
        const int lc = 8 * k + 7 < NU ? l : min(l, NU - 1);
#pragma unroll
        for (int q = 0; q < 5; ++q) xt[k][q == 0 ? 0 : q + 1] = *reinterpret_cast<const float2*>(lo + (xe[q] - lc));
        xt[k][1] = *reinterpret_cast<const float2*>(hi + (xe[0] - lc));
    }
    __syncwarp();
    float* out = im.gpix + ((long long)y0 * im.W + x0);
    const long long step = 4LL * im.W;
#pragma unroll 2
    for (int m = 0; m < KR; ++m) {
        const int r = rg + 4 * m;
        const float4 a = sV[r][0], b = sV[r][1], c = sV[r][2];
        const bool oky = r < NU && (unsigned)(y0 + 4 * m) < (unsigned)im.H;
#pragma unroll
        for (int k = 0; k < KC; ++k) {
            float2 s = make_float2(xt[k][0].x * a.x, xt[k][0].y * a.y);
            s = fma2(xt[k][1], make_float2(a.z, a.w), s);
            s = fma2(xt[k][2], make_float2(b.x, b.y), s);
            s = fma2(xt[k][3], make_float2(b.z, b.w), s);
            s = fma2(xt[k][4], make_float2(c.x, c.y), s);
            s = fma2(xt[k][5], make_float2(c.z, c.w), s);
            if (oky && okx[k]) atomicAdd(out + 8 * k, s.x + s.y);
        }
        out += step;
    }
    __syncwarp();
}

// The table entries of a point's x and y taps at union column and row 0, a
// byte each: variant and pixel offset from P's pixel.
template <int R>
__device__ __forceinline__ unsigned tap_entries(int rho, int kap, int pr, int pc)
{
    constexpr int NT = BwCfg<R>::NT, NTP = BwCfg<R>::NTP;
    static_assert(3 * NTP <= 256, "table entries fit a byte");
    int xv, yv;
    variants(pr, pc, &xv, &yv);
    return (xv * NTP + NT + 2 + (pc >> 1) - (kap >> 1)) | (yv * NTP + NT + 2 + (pr >> 1) - (rho >> 1)) << 8;
}

template <int R>
__global__ void __launch_bounds__(kBwAdjThreads, BwCfg<R>::MINB) bw_adjoint(const __grid_constant__ BwParams p)
{
    using C = BwCfg<R>;
    constexpr int NT = C::NT, NTP = C::NTP, NU = C::NU;
    extern __shared__ __align__(16) unsigned char bw_smem[];
    float4* lo = reinterpret_cast<float4*>(bw_smem);
    float4* hi = lo + 3 * NTP;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* mine = bw_smem + C::off_warp + wid * C::warp_b;
    float* rows = reinterpret_cast<float*>(mine);                         // [2][32][ROW]
    float* rec = reinterpret_cast<float*>(mine);                          // [32][RECW], phase 3
    float4(*sV)[3] = reinterpret_cast<float4(*)[3]>(mine + sizeof(float) * 32 * C::RECW);  // [NUP], phase 3
    int* list = reinterpret_cast<int*>(bw_smem + C::off_list);                           // [kBwChunk]: a chunk's edgels
    unsigned long long* cnt = reinterpret_cast<unsigned long long*>(list + kBwChunk);    // [2 * warps]
    build_tables<R>(p, lo, hi);
    double gsig = 0.0;
    const long long first = (long long)blockIdx.x * p.per_cta;
    const int cend = (int)min((long long)p.n_edgels, first + p.per_cta);
    for (int c0 = (int)min(first, (long long)p.n_edgels); c0 < cend;) {
        // a chunk: up to kBwChunk edgels of one image
        const int k = find_image(p.n_img, c0, [&](int i) { return p.img[i].edgel_base; });
        const BwImage& im = p.img[k];
        const int n = min(min(kBwChunk, cend - c0), im.edgel_base + im.n - c0), W2 = 2 * im.W;
        __syncthreads();  // the tables are built, the last chunk's list has been read
        int n0 = n;  // edgels on even columns
        const bool few = n <= kBwFew * kBwWarps;
        if (!few) {
        // order: even 2x columns with their windows inside the image, even and
        // at its border, odd and at its border, odd and inside
        int kind[2];
        unsigned pos[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int e = threadIdx.x + u * kBwAdjThreads;
            kind[u] = 4;
            if (e < n) {
                const int gi = im.gidx[c0 - im.edgel_base + e], rho = gi / W2, kap = gi - rho * W2;
                const int y = (rho >> 1) - R - 2, x = (kap >> 1) - R - 2;
                const bool in = y >= 0 && y + NU <= im.H && x >= 0 && x + NU <= im.W;
                kind[u] = (kap & 1) ? (in ? 3 : 2) : (in ? 0 : 1);
            }
            unsigned long long c = 0;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const unsigned same = __ballot_sync(0xffffffffu, kind[u] == v);
                if (kind[u] == v) pos[u] = __popc(same & ((1u << lane) - 1u));
                c |= (unsigned long long)__popc(same) << 16 * v;
            }
            if (lane == 0) cnt[u * kBwWarps + wid] = c;
        }
        __syncthreads();
        unsigned long long sum = 0, before[2] = {0, 0};  // four counts of 16 bits
#pragma unroll
        for (int w = 0; w < 2 * kBwWarps; ++w) {
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (w == u * kBwWarps + wid) before[u] = sum;
            sum += cnt[w];
        }
        const unsigned long long start = sum * 0x0001000100010000ull;  // the kinds' first places
        n0 = (int)(start >> 32 & 0xffff);
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (kind[u] < 4)
                list[((unsigned)((start + before[u]) >> 16 * kind[u]) & 0xffffu) + pos[u]] =
                    c0 - im.edgel_base + threadIdx.x + u * kBwAdjThreads;
        __syncthreads();
        }
        // rounds of at most 32, as many for every warp, shared out between the
        // two columns' parities; where that needs a round more, one round holds
        // both and its warp evaluates both kinds of rows
        int Q = kBwWarps, q0 = kBwWarps, per0 = (n + kBwWarps - 1) / kBwWarps, per1 = per0;
        bool apart = false;
        if (!few) {
            Q = (n + 32 * kBwWarps - 1) / (32 * kBwWarps) * kBwWarps;
            q0 = (n0 * Q + n / 2) / n;
            if (n0 > 32 * q0) ++q0;
            if (n - n0 > 32 * (Q - q0)) --q0;
            apart = n0 <= 32 * q0;
            per0 = apart ? (n0 + q0 - 1) / max(q0, 1) : (n + Q - 1) / Q;
            per1 = apart ? (n - n0 + Q - q0 - 1) / max(Q - q0, 1) : per0;
        }
        for (int q = wid; q < Q; q += kBwWarps) {
            const bool second = apart && q >= q0;
            const int l0 = second ? n0 + (q - q0) * per1 : q * per0;
            const int nw = min(second ? per1 : per0, (apart && !second ? n0 : n) - l0);
            if (nw <= 0) continue;
            const int at = l0 + min(lane, nw - 1);  // (lanes past the round repeat its last edgel)
            const bool B = at >= n0;
            const int local = few ? c0 - im.edgel_base + at : list[at];
            const int gi = im.gidx[local];
            const int rho = gi / W2, kap = gi - rho * W2, a = rho & 1;
            // ---- phase 1 ----
            const int wy = (rho >> 1) - R - 2, wx = (kap >> 1) - R - 2;  // the window's corner
            // Eight lanes copy a window's row, an aligned group of four pixels
            // (16 bytes of a float image, 4 of an 8-bit one) each, a row ahead of
            // its use.  A group is copied if it holds a pixel of the row and lies
            // wholly between the image's first and last pixel (toed_groups.h);
            // where a window reaches outside the image, what is read there is
            // masked to zero.
            const bool u8 = im.dtype == TOED_U8;
            const long long span = (long long)(im.H - 1) * im.pitch + im.W;
            // A round this short is cheaper a warp per edgel (below), which also
            // takes images whose offsets need 64 bits, and those narrower than a group
            const bool by_warp = few || span + 32LL * im.pitch >= (1LL << 30) || im.W < 4;
            const bool inside = __all_sync(0xffffffffu, wy >= 0 && wy + NU <= im.H && wx >= 0 && wx + NU <= im.W);
            const uintptr_t src = reinterpret_cast<uintptr_t>(im.src);
            const int skew = (int)(u8 ? src & 3 : src >> 2 & 3);  // the first pixel's place in its group
            const uintptr_t first_group = src - (u8 ? skew : 4 * skew);
            const unsigned whole = whole_groups(span);
            // the window's first pixel, from first_group
            const int own = by_warp ? 0 : (int)(wy * im.pitch) + wx + skew;
            int off[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) off[t] = __shfl_sync(0xffffffffu, own, 4 * t + (lane >> 3)) + 4 * (lane & 7);
            auto stage = [&](int u, int buf) {  // window row u of all windows
                const int up = u * (int)im.pitch;
                const uint32_t d = smem_addr(rows + buf * 32 * C::ROW);
                auto wanted = [&](int at) { return group_copied<NU, C::CH>(at, lane & 7, skew, whole); };
                if (u8) {
                    const uint32_t dst = d + (lane >> 3) * C::ROW + 4 * (lane & 7);
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (wanted(off[t] + up))
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * t * C::ROW),
                                         "l"(first_group + ((off[t] + up) & ~3))
                                         : "memory");
                } else {
                    const uint32_t dst = d + (lane >> 3) * 4 * C::ROW + 16 * (lane & 7);
#pragma unroll
                    for (int t = 0; t < 8; ++t)
                        if (wanted(off[t] + up))
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * t * C::ROW),
                                         "l"(first_group + 4LL * ((off[t] + up) & ~3))
                                         : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            // The windows are evaluated less their middle pixel, whose constant is
            // added at the end: the sums' rounding is then relative to the
            // window's contrast, not to its brightness
            // (8-bit pixels carry 2^23, the float whose last bits they are)
            // -- not a number where the window needs a group that is not copied, so
            // that all its values are none and count as ill-conditioned
            const float mid = by_warp ? 0.f
                              : window_cut(wy, wx, NU, im.H, im.W, skew, span) ? __int_as_float(0x7fc00000)
                                                                               : pix(im, rho >> 1, kap >> 1);
            const float zero = u8 ? 8388608.f : 0.f, less = zero + mid;
            BwValues o = {};
            __syncwarp();
            if (!by_warp) stage(0, 0);
#pragma unroll 1
            for (int u = by_warp ? NU : 0; u < NU; ++u) {
                if (u + 1 < NU) {
                    stage(u + 1, (u + 1) & 1);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");
                } else {
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                }
                __syncwarp();
                // the row, from where it starts in its first group
                float v[NU];
                {
                    const float* buf = rows + (u & 1) * 32 * C::ROW;
                    float w[4 * C::CH];
                    if (u8) {
                        const unsigned* row = reinterpret_cast<const unsigned*>(buf) + lane * (C::ROW / 4);
#pragma unroll
                        for (int t = 0; t < C::CH; ++t) {
                            const unsigned g = row[t];
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                w[4 * t + k] = __uint_as_float(__byte_perm(g, 0x4b000000u, 0x7440u | k));
                        }
                    } else {
                        const float4* row = reinterpret_cast<const float4*>(buf + lane * C::ROW);
#pragma unroll
                        for (int t = 0; t < C::CH; ++t) {
                            const float4 g = row[t];
                            w[4 * t] = g.x;
                            w[4 * t + 1] = g.y;
                            w[4 * t + 2] = g.z;
                            w[4 * t + 3] = g.w;
                        }
                    }
                    const unsigned s = (unsigned)(own + u * (int)im.pitch);
#pragma unroll
                    for (int t = 0; t < NU + 1; ++t) w[t] = (s & 2u) ? w[t + 2] : w[t];
#pragma unroll
                    for (int t = 0; t < NU; ++t) v[t] = (s & 1u) ? w[t + 1] : w[t];
                    if (!inside) {
                        const unsigned cols = (0xffffffffu >> (32 - min(NU, im.W - wx))) & (0xffffffffu << max(0, -wx));
                        const unsigned in = (unsigned)(wy + u) < (unsigned)im.H ? cols : 0u;
#pragma unroll
                        for (int t = 0; t < NU; ++t) v[t] = (in >> t & 1u) ? v[t] : zero;
                    }
                }
#pragma unroll
                for (int t = 0; t < NU; ++t) v[t] -= less;
                if (B)
                    eval_row<R, 1>(v, p, a, lo + NT + 2 - u, hi + NT + 2 - u, o);
                else
                    eval_row<R, 0>(v, p, a, lo + NT + 2 - u, hi + NT + 2 - u, o);
                __syncwarp();  // the row after next overwrites the buffer
            }
            if (!by_warp) add_constant(p, a, B, mid, o);
            o.top += fabsf(mid);
            // ---- the frozen sector (cpu_toed.cpp:415-462 in closed form) ----
            bool xmaj = fabsf(o.d[0]) >= fabsf(o.d[1]);
            int sx = o.d[0] >= 0.f ? 1 : -1, sy = o.d[1] >= 0.f ? 1 : -1;
            float nv[4][4];  // A+, D+, A-, D-
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const float l = o.n[3][f], r = o.n[4][f], t = o.n[1][f], b = o.n[6][f];
                nv[0][f] = xmaj ? (sx > 0 ? r : l) : (sy > 0 ? b : t);
                nv[2][f] = xmaj ? (sx > 0 ? l : r) : (sy > 0 ? t : b);
                nv[1][f] = sy > 0 ? (sx > 0 ? o.n[7][f] : o.n[5][f]) : (sx > 0 ? o.n[2][f] : o.n[0][f]);
                nv[3][f] = sy > 0 ? (sx > 0 ? o.n[0][f] : o.n[2][f]) : (sx > 0 ? o.n[5][f] : o.n[7][f]);
            }
            __syncwarp();
            float go[4];
            if (p.out_f64) {
                const double* g = (const double*)im.gout + 4LL * local;
#pragma unroll
                for (int q = 0; q < 4; ++q) go[q] = (float)g[q];
            } else {
                const float* g = (const float*)im.gout + 4LL * local;
#pragma unroll
                for (int q = 0; q < 4; ++q) go[q] = g[q];
            }
            const bool used = go[0] != 0.f || go[1] != 0.f || go[2] != 0.f || go[3] != 0.f;
            unsigned ill = __ballot_sync(0xffffffffu,
                                         lane < nw && (by_warp || ill_conditioned(o, nv, xmaj, used, p.ill_curve)));
            for (; ill; ill &= ill - 1) {
                const int w = __ffs(ill) - 1;
                const int bits = eval_edgel_warp<R>(im, __shfl_sync(0xffffffffu, rho, w), __shfl_sync(0xffffffffu, kap, w),
                                                    lane, lo, hi, rows);
                if (lane == w) {
                    const float* val = rows + C::kVals * C::kRed;
#pragma unroll
                    for (int q = 0; q < 9; ++q) {
                        o.d[q] = val[q];
                        o.s[q] = val[9 + q];
                    }
#pragma unroll
                    for (int q = 0; q < 16; ++q) nv[q / 4][q % 4] = val[18 + q];
                    xmaj = bits & 1;
                    sx = (bits & 2) ? 1 : -1;
                    sy = (bits & 4) ? 1 : -1;
                }
                __syncwarp();
            }
            // ---- phase 2: the chain rule ----
            if (lane < nw) {
            const float fx = o.d[0], fy = o.d[1], fxx = o.d[2], fxy = o.d[3], fyy = o.d[4], fxxy = o.d[5],
                        fxyy = o.d[6], fxxx = o.d[7], fyyy = o.d[8];
            float nd[4][2], M[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                nd[q][0] = nv[q][0];
                nd[q][1] = nv[q][1];
                M[q] = sqrtf(nd[q][0] * nd[q][0] + nd[q][1] * nd[q][1]);
            }
            // ---- forward values ----
            const float m = sqrtf(fx * fx + fy * fy);
            const float rm = 1.f / m;
            const float nx = fx * rm, ny = fy * rm;
            const float c = (float)(sx * sy);
            const float t = xmaj ? c * fy / fx : c * fx / fy;  // slope |ny|/|nx| or |nx|/|ny|
            float num, den;
            {
                const double td = t;
                const double fp = (double)M[0] * (1.0 - td) + (double)M[1] * td;
                const double fm = (double)M[2] * (1.0 - td) + (double)M[3] * td;
                num = (float)(fp - fm);
                den = (float)(fm + fp - 2.0 * (double)m);
            }
            const float rden = 1.f / den;
            const float S = sqrtf(1.f + t * t);
            const float sst = -0.5f * num * S * rden;
            // ---- reverse: position, strength ----
            const float g_sst = 0.5f * (go[0] * nx + go[1] * ny);
            const float g_nx = 0.5f * go[0] * sst, g_ny = 0.5f * go[1] * sst;
            const float g_maxf = go[3];  // strength = |max_f| |n| = max_f (max_f > 0 at a maximum)
            const float g_num = -0.5f * S * rden * g_sst - 0.25f * num * rden * g_maxf;
            const float g_den = 0.5f * num * S * rden * rden * g_sst + 0.125f * num * num * rden * rden * g_maxf;
            float g_t = g_sst * (-0.5f * num * rden) * t / S;
            const float g_m = g_maxf - 2.f * g_den;
            const float g_fp = g_num + g_den, g_fm = -g_num + g_den;
            const float gM[4] = {g_fp * (1.f - t), g_fp * t, g_fm * (1.f - t), g_fm * t};
            g_t += g_fp * (M[1] - M[0]) + g_fm * (M[3] - M[2]);
            float gfx = 0.f, gfy = 0.f;
            if (xmaj) {
                gfx += g_t * (-t / fx);
                gfy += g_t * (c / fx);
            } else {
                gfx += g_t * (c / fy);
                gfy += g_t * (-t / fy);
            }
            const float rm3 = rm * rm * rm;
            gfx += g_nx * (rm - fx * fx * rm3) + g_ny * (-fx * fy * rm3) + g_m * fx * rm;
            gfy += g_nx * (-fx * fy * rm3) + g_ny * (rm - fy * fy * rm3) + g_m * fy * rm;
            // ---- reverse: orientation atan2(TIx, -TIy) (cpu_toed.cpp:227-232) ----
            float gP[9];
            gP[2] = gP[3] = gP[4] = gP[5] = gP[6] = gP[7] = gP[8] = 0.f;
            if (go[2] != 0.f) {
                const double dx = fx, dy = fy, dxx = fxx, dxy = fxy, dyy = fyy;
                const double TIx = dx * (2 * dxx * dxx + 2 * dxy * dxy) + dy * (2 * dxx * dxy + 2 * dyy * dxy) +
                                   2 * dx * dy * (double)fxxy + dy * dy * (double)fxyy + dx * dx * (double)fxxx;
                const double TIy = dx * (2 * dxx * dxy + 2 * dyy * dxy) + dy * (2 * dyy * dyy + 2 * dxy * dxy) +
                                   2 * dx * dy * (double)fxyy + dx * dx * (double)fxxy + dy * dy * (double)fyyy;
                const float tix = (float)TIx, tiy = (float)TIy;
                const float q2 = tix * tix + tiy * tiy;
                if (q2 > 0.f) {
                    const float gX = go[2] * (-tiy) / q2, gY = go[2] * tix / q2;
                    gfx += gX * (2 * fxx * fxx + 2 * fxy * fxy + 2 * fy * fxxy + 2 * fx * fxxx) +
                           gY * (2 * fxx * fxy + 2 * fyy * fxy + 2 * fy * fxyy + 2 * fx * fxxy);
                    gfy += gX * (2 * fxx * fxy + 2 * fyy * fxy + 2 * fx * fxxy + 2 * fy * fxyy) +
                           gY * (2 * fyy * fyy + 2 * fxy * fxy + 2 * fx * fxyy + 2 * fy * fyyy);
                    gP[2] = gX * (4 * fx * fxx + 2 * fy * fxy) + gY * (2 * fx * fxy);
                    gP[3] = gX * (4 * fx * fxy + 2 * fy * fxx + 2 * fy * fyy) + gY * (2 * fx * fxx + 2 * fx * fyy + 4 * fy * fxy);
                    gP[4] = gX * (2 * fy * fxy) + gY * (2 * fx * fxy + 4 * fy * fyy);
                    gP[5] = gX * (2 * fx * fy) + gY * (fx * fx);
                    gP[6] = gX * (fy * fy) + gY * (2 * fx * fy);
                    gP[7] = gX * (fx * fx);
                    gP[8] = gY * (fy * fy);
                }
            }
            gP[0] = gfx;
            gP[1] = gfy;
            // the cotangents: [0..8] at P, [9 + 2q, 10 + 2q] = (gx, gy) at
            // neighbour q, [17..19] the table entries of P, A+, D+, A-, D-
            float gs = 0.f;
#pragma unroll
            for (int q = 0; q < 9; ++q) gs = fmaf(gP[q], o.s[q], gs);
            float gN[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float rM = gM[q] / M[q];
                gN[2 * q] = rM * nd[q][0];
                gN[2 * q + 1] = rM * nd[q][1];
                gs = fmaf(gN[2 * q], nv[q][2], fmaf(gN[2 * q + 1], nv[q][3], gs));
            }
            const int ar = xmaj ? 0 : sy, ac = xmaj ? sx : 0;
            float4* out = reinterpret_cast<float4*>(rec + lane * C::RECW);
            out[0] = make_float4(gP[0], gP[1], gP[2], gP[3]);
            out[1] = make_float4(gP[4], gP[5], gP[6], gP[7]);
            out[2] = make_float4(gP[8], gN[0], gN[1], gN[2]);
            out[3] = make_float4(gN[3], gN[4], gN[5], gN[6]);
            out[4] = make_float4(gN[7],
                                 __uint_as_float(tap_entries<R>(rho, kap, rho, kap) |
                                                 tap_entries<R>(rho, kap, rho + ar, kap + ac) << 16),
                                 __uint_as_float(tap_entries<R>(rho, kap, rho + sy, kap + sx) |
                                                 tap_entries<R>(rho, kap, rho - ar, kap - ac) << 16),
                                 __uint_as_float(tap_entries<R>(rho, kap, rho - sy, kap - sx)));
            gsig += gs;
            }
            __syncwarp();
            // ---- phase 3: scatter, a warp per edgel (scatter_edgel_warp) ----
            grid_wait();  // bw_clear's zeros
            for (int w = 0; w < nw; ++w)
                scatter_edgel_warp<R>(im, __shfl_sync(0xffffffffu, rho, w), __shfl_sync(0xffffffffu, kap, w), lane, lo, hi,
                                      rec + w * C::RECW, sV);
            __syncwarp();  // the next round overwrites the records
        }
        c0 += n;
    }
    // dL/dsigma: warp sums in FP64, one FP64 atomic per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) gsig += __shfl_down_sync(0xffffffffu, gsig, o);
    if (lane == 0 && gsig != 0.0) atomicAdd(p.gsig, gsig);
}

// Resident CTAs of bw_adjoint<R> on each device (SMs x CTAs per SM), found once.
constexpr int kBwMaxDevices = 64;

template <int R>
static int bw_resident_ctas()
{
    static std::atomic<int> cache[kBwMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kBwMaxDevices) return 0;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        int sms = 0, bps = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaFuncSetAttribute(bw_adjoint<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BwCfg<R>::smem) !=
                cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, bw_adjoint<R>, kBwAdjThreads, BwCfg<R>::smem) != cudaSuccess ||
            bps <= 0)
            return 0;
        n = sms * bps;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

template <int R>
static cudaError_t launch_bw(BwParams& p, cudaStream_t stream)
{
    if (p.n_edgels == 0) return cudaSuccess;
    // every CTA the same run of edgels, as short as keeps the launch in one wave and its warps busy
    const long long ctas = bw_resident_ctas<R>();
    if (ctas <= 0) return cudaErrorInvalidConfiguration;
    p.per_cta = (int)std::max<long long>(kBwWarps, (p.n_edgels + ctas - 1) / ctas);
    void* args[] = {&p};
    return launch_after((const void*)bw_adjoint<R>, dim3((unsigned)((p.n_edgels + p.per_cta - 1) / p.per_cta)),
                        dim3(kBwAdjThreads), args, BwCfg<R>::smem, stream);
}

// Clears dL/dI of image blockIdx.y (rows of width W, contiguous): 16-byte
// stores from the first 16-byte boundary, scalar stores around them.
__global__ void __launch_bounds__(256) bw_clear(const __grid_constant__ BwParams p)
{
    launch_dependents();  // bw_adjoint evaluates its edgels meanwhile
    const BwImage& d = p.img[blockIdx.y];
    float* g = d.gpix;
    if (p.first && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *p.gsig = 0.0;
    const long long npx = (long long)d.H * d.W;
    const long long head = min(npx, (long long)(((16u - (reinterpret_cast<uintptr_t>(g) & 15u)) & 15u) / 4u));
    const long long nv = (npx - head) / 4;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
    float4* g4 = reinterpret_cast<float4*>(g + head);
    for (long long i = t0; i < nv; i += st) g4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t0 < head) g[t0] = 0.f;
    const long long tail = head + 4 * nv;
    if (t0 < npx - tail) g[tail + t0] = 0.f;
}

cudaError_t backward_launch(const toed_grad_image* items, int n, const toed_params* prm, int r, double* gsig,
                            bool first, cudaStream_t stream)
{
    std::unique_ptr<BwParams> pp(new BwParams());
    BwParams& p = *pp;
    std::memset(&p, 0, sizeof(p));
    const double s = prm->sigma, nrm = std::sqrt(2.0 * 3.14159265358979323846);
    for (int sh = 0; sh < 2; ++sh)
        for (int k = 0; k < 2 * r + 3; ++k) {
            const double x = (double)(k - (r + 1)) + (sh ? 0.5 : 0.0);
            const double e = std::exp(-(x * x) / (2.0 * s * s));
            const double G = e / (nrm * s), Gx = (-x * e) / (nrm * s * s * s);
            const double Gxx = ((x * x - s * s) * e) / (nrm * s * s * s * s * s);
            const double Gxxx = ((x * (3.0 * s * s - x * x)) * e) / (nrm * s * s * s * s * s * s * s);
            const double q = x * x / (s * s * s);  // d e / d sigma = e * x^2 / sigma^3
            const double v[8] = {G, Gx, Gxx, Gxxx, G * (q - 1.0 / s), Gx * (q - 3.0 / s),
                                 -2.0 * s * e / (nrm * s * s * s * s * s) + Gxx * (q - 5.0 / s),
                                 6.0 * s * x * e / (nrm * s * s * s * s * s * s * s) + Gxxx * (q - 7.0 / s)};
            for (int f = 0; f < 4; ++f) {
                p.tap[4 * sh + f][k] = (float)v[f];
                p.tap[8 + 4 * sh + f][k] = (float)v[4 + f];
            }
        }
    for (int v = 0; v < 3; ++v) {
        // sums as the kernel forms them: over mirrored sums and differences, and
        // the shifted filters' last tap, which has no mirror image
        const int f0 = v == 2 ? 4 : 0;
        float c[8];
        for (int f = 0; f < 8; ++f) {
            const float* t = p.tap[(f < 4 ? f : f + 4) + f0];
            double sum = v == 2 ? t[2 * r + 2] : (f & 1) ? 0.f : t[r + 1];
            if (!(f & 1))
                for (int q = v == 2 ? 0 : 1; q <= r + (v == 1 ? 1 : 0); ++q) sum += 2.0 * t[q + r + 1];
            c[f] = (float)sum;
        }
        p.sum_lo[v] = make_float4(c[0], c[1], c[4], c[5]);
        p.sum_hi[v] = make_float4(c[2], c[3], c[6], c[7]);
    }
    p.ill_curve = (float)(kIllCurve / (s * s));
    p.r = r;
    p.out_f64 = prm->out_dtype == TOED_F64;
    p.n_img = n;
    p.gsig = gsig;
    p.first = first;
    int edg = 0;
    for (int i = 0; i < n; ++i) {
        BwImage& d = p.img[i];
        d.src = items[i].pixels;
        d.pitch = items[i].pitch;
        d.gidx = items[i].grid_index;
        d.gout = items[i].grad_edgels;
        d.gpix = items[i].grad_pixels;
        d.H = items[i].height;
        d.W = items[i].width;
        d.dtype = items[i].dtype;
        d.n = items[i].n_edgels;
        d.edgel_base = edg;
        edg += d.n;
    }
    p.n_edgels = edg;
    {
        // dL/dI of every image cleared by one launch (the scatter adds into it)
        void* args[] = {&p};
        const cudaError_t e = cudaLaunchKernel((const void*)bw_clear, dim3(64, n), dim3(256), args, 0, stream);
        if (e != cudaSuccess) return e;
    }
    switch (r) {
    case 1: return launch_bw<1>(p, stream);
    case 2: return launch_bw<2>(p, stream);
    case 3: return launch_bw<3>(p, stream);
    case 4: return launch_bw<4>(p, stream);
    case 5: return launch_bw<5>(p, stream);
    case 6: return launch_bw<6>(p, stream);
    case 7: return launch_bw<7>(p, stream);
    case 8: return launch_bw<8>(p, stream);
    case 9: return launch_bw<9>(p, stream);
    case 10: return launch_bw<10>(p, stream);
    case 11: return launch_bw<11>(p, stream);
    case 12: return launch_bw<12>(p, stream);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace toed
