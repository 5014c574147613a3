// toed_detect.cuh -- fused single-pass TOED detection kernel (sm_103a).
//
// One persistent CTA (256 threads) repeatedly takes a work unit from an
// atomic queue.  A unit is a vertical strip of one image: 30 output columns
// (32 with a one-pixel ring) by S output rows.  The CTA slides down the strip
// in steps of B = 16 rows, keeping everything on chip:
//
//   1. B new input rows (+ halo) arrive in shared memory by TMA, or by loads
//      prefetched in registers (8-bit images, unaligned rows);
//   2. row pass: six horizontal responses -- G and Gx, each truncated to
//      2r+1 taps (T), full 2r+3 taps (F) and half-pixel shifted (S) -- into a
//      ring of row-pass rows (the corrected-normal mode adds Gxx and Gxxx);
//   3. column pass: Ix and Iy at the four half-pixel sub-grids (the 2x grid
//      of the reference, cpu_toed.cpp:204-355) for the B new rows, and the
//      threshold test on |grad I|^2 as one ballot mask per (2x row, column
//      parity);
//   4. each warp lists the points above the threshold of four 2x rows in
//      row-major order and decides them: subpixel NMS along the gradient with
//      the reference's 8-sector interpolation, max test and parabola fit
//      (cpu_toed.cpp:399-495), in FP32; the survivors' gradient and neighbour
//      magnitudes go to a staging area, each row's {offset, count} to the
//      row-segment table.
//
// The edgel kernel (toed_edgels.cu) turns these into the reference's row-major
// edgel list: the fit's result, the seven higher derivatives -- contracted
// from the image at the edgels alone -- and the third-order orientation.
//
// The row-pass ring holds a multiple of 8 rows (the live window rounded up)
// and is indexed by absolute row, so sliding the window moves no data.
//
// What bounds it: instruction issue (75 % of the slots), about 790 warp
// instructions a warp and step at r = 6, of which 340 are the two dense passes.
// 78.8 Mpixel at r = 6: 1.28 ms, three CTAs per SM with two barriers a step;
// it was 2.17 ms (61 % issue) when the kernel also held the Gxx / Gxxx responses
// for the edgels' sums (two CTAs per SM), converted its rows and listed the
// points for the whole CTA (six barriers a step).
//
// Compared with the reference kernel (direct 17x17 and 19x19 sums of nine
// derivatives at every point, gpu_convolve.cu:114-131) this evaluates the
// separable form, keeps the nine-derivative stack off HBM entirely and
// leaves seven of the nine derivatives to the edgel kernel.
#pragma once
#include "toed_common.cuh"

namespace toed {

__host__ __device__ constexpr size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// NMS-window rows are kFxyStride float2 apart (FW = 2 kExt used): the two
// spare entries shift each row by four banks, so that the NMS stage's reads
// at scattered (row, column) points collide less.
constexpr int kFxyStride = 2 * kExt + 2;

// NMSTO: the corrected-normal mode holds the Gxx / Gxxx row responses too.
template <int R, bool NMSTO = false>
struct Cfg {
    static constexpr int NP = NMSTO ? 6 : 3;        // row-pass planes held
    static constexpr int NWARP = kThreads / 32;
    static constexpr int B = kStepRows;
    static constexpr int NT = 2 * R + 3;            // taps of a full / shifted filter
    static constexpr int NIN = kExt + 2 * R + 2;    // input columns of a row's window
    static constexpr int HS = B + 2 * R + 3;        // live rows of the row-pass window
    // ring rows: HS rounded up to a multiple of 8, so that the ring row of
    // slot 0 (advancing by B) stays a multiple of 8 and the column pass knows
    // where its window can wrap (col_pass)
    static constexpr int RING = (HS + 7) / 8 * 8;
    static constexpr int MS = 2 * B + 2;            // 2x-grid rows held for NMS
    static constexpr int NMS_ROWS = 2 * B;          // 2x-grid rows decided per step
    // each warp decides WROWS consecutive 2x-grid rows; its list holds them whole
    static constexpr int WROWS = NMS_ROWS / NWARP;
    static constexpr int MAXC = WROWS * 2 * kExt;
    static constexpr int FW = 2 * kExt;             // 2x-grid columns held per row
    // staged input rows: boxes of B rows, BW floats apart; the first step's
    // window is Q0 boxes, all of them in flight at once
    static constexpr int BW = staged_width(R);
    static constexpr int OFF = R & 1;               // parity of the window's first column in a staged row
    static constexpr int Q0 = (HS + B - 1) / B;
    static constexpr int NBUF = 3;
    static_assert(Q0 <= NBUF, "the first step's boxes fit the buffers");
    static constexpr size_t box_bytes = sizeof(float) * B * BW;
    static_assert(box_bytes % 128 == 0, "TMA destinations");
    static constexpr size_t off_raw = 0;
    static constexpr size_t off_mbar = off_raw + NBUF * box_bytes;
    static constexpr size_t off_P = align_up(off_mbar + 8 * NBUF, 16);
    // row-pass ring rows are PS float2 apart: two spare entries per row shift
    // each row by four banks, so that scattered reads (one point's column per
    // lane) collide less
    static constexpr int PS = kExt + 2;
    static constexpr size_t off_fxy = off_P + sizeof(float2) * NP * RING * PS;
    static constexpr size_t off_mask = off_fxy + sizeof(float2) * MS * kFxyStride;
    static constexpr size_t off_list = align_up(off_mask + sizeof(unsigned) * MS * 2, 16);
    static constexpr size_t off_tab = align_up(off_list + sizeof(unsigned short) * NWARP * MAXC, 16);
    static constexpr size_t off_misc = off_tab + (NMSTO ? sizeof(float4) * 3 * NT : 0);
    static constexpr size_t smem = off_misc + sizeof(int) * 4;
    // three CTAs per SM where their shared memory fits (r <= 8), two beyond
    static constexpr int MINB = smem <= 74 * 1024 ? 3 : 2;
};

// Image pixel with zero padding outside the image (cpu_toed.cpp:207-208).
__device__ __forceinline__ float fetch_px(const float* src, long long pitch, int H, int W, int y, int x)
{
    if ((unsigned)y >= (unsigned)H || (unsigned)x >= (unsigned)W) return 0.f;
    return __ldg(src + (long long)y * pitch + x);
}

// Ring row of x for 0 <= x < 2 * N (every ring index the kernel forms).
template <int N>
__device__ __forceinline__ int ring_wrap(int x) { return x >= N ? x - N : x; }

// ---------------------------------------------------------------------------
// Row pass of one staged input row at columns 2k, 2k+1: window float 0 is the
// row's float at image column x0 - R - 2 + 2k, `src` the even-aligned address
// at or before it (Cfg::OFF floats before it); the responses go to ring row ph.
// Planes: 0 PT=(T_G,T_Gx) 1 PF=(F_G,F_Gx) 2 PS=(S_G,S_Gx), each [RING][PS]
// float2 (32 used per row); NMSTO adds 3 QT=(T_Gxx,T_Gxxx) 4 QF 5 QS.
// Convolution direction as the reference: out(x) = sum_q in(x-q) X(q).
// ---------------------------------------------------------------------------
template <int R, bool NMSTO>
__device__ __forceinline__ void row_pass(const float* __restrict__ src, int k, int ph, float2* __restrict__ sP,
                                         const TapBlock& tp, int* dbg)
{
    using C = Cfg<R, NMSTO>;
    constexpr int NV = 2 * R + 4, NL = (NV + C::OFF + 1) / 2;
    if (TOED_IN_BOUNDS(ph < C::RING, dbg)) {
        float w[2 * NL];
#pragma unroll
        for (int t = 0; t < NL; ++t) {
            const float2 q = reinterpret_cast<const float2*>(src)[t];
            w[2 * t] = q.x;
            w[2 * t + 1] = q.y;
        }
        const float* v = w + C::OFF;
        float o_[2][2 * C::NP];
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            // The odd filters (Gx, Gxxx) are exactly antisymmetric about 0 (about
            // -1/2 for the shifted set): each mirrored pair of inputs is
            // differenced once -- fewer operations and a smaller rounding
            // error, since neighbouring inputs nearly cancel.  The even filters
            // (G, Gxx) are summed tap by tap: folding them would round the sum
            // of two full-scale inputs and double the error of Gxx.
            const int c = o + R + 1;  // centre: out(x) = sum_q in(x-q) X(q), in(x-q) = v[c-q]
            float tG = 0.f, tGxx = 0.f, tGx = 0.f, tGxxx = 0.f;
#pragma unroll
            for (int q = -R; q <= R; ++q) {
                tG = fmaf(v[c - q], tp.v[0][q + R + 1], tG);
                if (NMSTO) tGxx = fmaf(v[c - q], tp.v[2][q + R + 1], tGxx);
            }
#pragma unroll
            for (int q = 1; q <= R; ++q) {
                const float df = v[c - q] - v[c + q];
                tGx = fmaf(df, tp.v[1][q + R + 1], tGx);
                if (NMSTO) tGxxx = fmaf(df, tp.v[3][q + R + 1], tGxxx);
            }
            // full 2r+3-tap responses add the taps q = +-(r+1)
            const float fG = fmaf(v[c + R + 1], tp.v[0][0], fmaf(v[c - R - 1], tp.v[0][2 * R + 2], tG));
            const float dfo = v[c - R - 1] - v[c + R + 1];
            const float fGx = fmaf(dfo, tp.v[1][2 * R + 2], tGx);
            // shifted taps X(q + 1/2), q = -(r+1)..r+1: even filters tap by tap,
            // odd ones over the pairs (q, -1-q) for q = 0..r plus q = r+1 alone
            float sG = 0.f, sGxx = 0.f;
#pragma unroll
            for (int q = -(R + 1); q <= R + 1; ++q) {
                sG = fmaf(v[c - q], tp.v[4][q + R + 1], sG);
                if (NMSTO) sGxx = fmaf(v[c - q], tp.v[6][q + R + 1], sGxx);
            }
            const float vl = v[c - R - 1];
            float sGx = vl * tp.v[5][2 * R + 2], sGxxx = vl * tp.v[7][2 * R + 2];
#pragma unroll
            for (int q = 0; q <= R; ++q) {
                const float df = v[c - q] - v[c + 1 + q];
                sGx = fmaf(df, tp.v[5][q + R + 1], sGx);
                if (NMSTO) sGxxx = fmaf(df, tp.v[7][q + R + 1], sGxxx);
            }
            o_[o][0] = tG;  o_[o][1] = tGx;  o_[o][2] = fG;  o_[o][3] = fGx;
            o_[o][4] = sG;  o_[o][5] = sGx;
            if constexpr (NMSTO) {
                const float fGxx = fmaf(v[c + R + 1], tp.v[2][0], fmaf(v[c - R - 1], tp.v[2][2 * R + 2], tGxx));
                const float fGxxx = fmaf(dfo, tp.v[3][2 * R + 2], tGxxx);
                o_[o][6] = tGxx; o_[o][7] = tGxxx;
                o_[o][8] = fGxx; o_[o][9] = fGxxx; o_[o][10] = sGxx; o_[o][11] = sGxxx;
            }
        }
#pragma unroll
        for (int a = 0; a < C::NP; ++a) {
            float4* dst = reinterpret_cast<float4*>(sP + (a * C::RING + ph) * C::PS + 2 * k);
            *dst = make_float4(o_[0][2 * a], o_[0][2 * a + 1], o_[1][2 * a], o_[1][2 * a + 1]);
        }
    }
}

// ---------------------------------------------------------------------------
// Column pass for one (column, sub-grid, 8-row group): Ix and Iy.  Window
// rows are read from the row-pass ring: logical slot h <-> ring row
// (rb + h) mod RING, rb the ring row of slot 0 at this step.
// V = 0: unshifted y taps truncated to 2r+1 (sub-grid (0,0), cpu_toed.cpp:205-221)
// V = 1: unshifted y taps, full 2r+3 (sub-grid (0,1/2), :246-262)
// V = 2: shifted y taps (sub-grids (1/2, .), :287-344)
// ---------------------------------------------------------------------------
// (Ix, Iy) of a row is one packed FP32 pair: a window row's (G, Gx) responses
// are one 8-byte load, the taps (Gy, G) one 8-byte constant, and fma.rn.f32x2
// rounds each half as fmaf does (the pass issues half the FMAs: 184 -> 177 us
// on 8.2 Mpixel at r = 6).
template <int R, int V>
__device__ __forceinline__ void col_pass(const float2* __restrict__ P, int rb, int g, int col, const float2 (&yt)[2][kMaxTaps],
                                         float2 (&f)[kColRows])
{
    using C = Cfg<R>;
    constexpr int YF = (V == 2) ? 1 : 0;
    constexpr int NW = kColRows + 2 * R + 2;  // window rows
    // Window row t is ring row (r0 + t) mod RING.  RING, rb and 8g are
    // multiples of 8, so r0 = 1 (mod 8) and the wrap, if any, falls at
    // t = 7 (mod 8): every block of window rows t in [8b - 1, 8b + 7) reads
    // from one base pointer, chosen once, plus a constant offset.
    static_assert(C::RING % 8 == 0 && kStepRows % 8 == 0 && kColRows == 8, "column-pass wrap blocks");
    constexpr int NBLK = (NW + 8) / 8;
    unsigned long long acc[kColRows];  // (Iy, Ix)
#pragma unroll
    for (int o = 0; o < kColRows; ++o) acc[o] = 0ull;
    const int r0 = ring_wrap<C::RING>(rb + g * kColRows + 1);
    const int tw = C::RING - r0;  // first window row past the ring's end
    const float2* base[NBLK];
#pragma unroll
    for (int b = 0; b < NBLK; ++b)
        base[b] = P + (r0 - ((8 * b - 1 >= tw) ? C::RING : 0)) * C::PS + col;
#pragma unroll
    for (int t = 0; t < NW; ++t) {
        const unsigned long long h = *reinterpret_cast<const unsigned long long*>(&base[(t + 1) / 8][t * C::PS]);
#pragma unroll
        for (int o = 0; o < kColRows; ++o) {
            const int p = o + R + 1 - t;
            const bool in = (V == 0) ? (p >= -R && p <= R) : (p >= -(R + 1) && p <= R + 1);
            if (in) {
                const unsigned long long tap = *reinterpret_cast<const unsigned long long*>(&yt[YF][p + R + 1]);
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[o]) : "l"(h), "l"(tap));
            }
        }
    }
#pragma unroll
    for (int o = 0; o < kColRows; ++o)
        f[o] = make_float2(__uint_as_float((unsigned)(acc[o] >> 32)), __uint_as_float((unsigned)acc[o]));
}

// The NMS decision at 2x-grid slot (m, c) of the step window, without
// branches: every value is formed unconditionally (the neighbour offsets are
// within one row and column whatever the direction) and the tests are combined
// at the end, so a warp runs it as one straight sequence.  The values that the
// fit needs are left in `e`.
// TOD (the corrected-normal mode, an extension beyond the reference): the
// sector and the neighbours are taken along the third-order vector (tx, ty)
// instead of along (Ix, Iy); the candidate tests (threshold, gradient epsilon)
// stay those of the reference.
struct NmsPoint {
    float gx, gy, Map, Mdp, Mam, Mdm;
};

template <bool TOD = false>
__device__ __forceinline__ bool nms_decide(const float2* __restrict__ sFxy, int m, int c, float thr, NmsPoint& e,
                                           float tx = 0.f, float ty = 0.f, int* dbg = nullptr)
{
    constexpr int FS = kFxyStride;
#ifdef TOED_DEBUG_BOUNDS
    if (!TOED_IN_BOUNDS(m >= 1 && m + 1 < 2 * kStepRows + 2 && c >= 1 && c + 1 < 2 * kExt, dbg)) return false;
#endif
    const float2* at = sFxy + m * FS + c;
    const float2 g = *at;
    const float mv = grad_mag(g);
    const float dx = TOD ? tx : g.x, dy = TOD ? ty : g.y;
    // Eight sectors of cpu_toed.cpp:415-462 in closed form: x-major when
    // |Ix| >= |Iy|; the axis neighbour steps along the major axis towards
    // the gradient, the diagonal one along both; fm mirrors fp.  The slope
    // (minor over major component of the unit normal) is the ratio of the
    // direction's own components, the normalisation cancelling.
    const float ax = fabsf(dx), ay = fabsf(dy);
    const int sx = (dx >= 0.f) ? 1 : -1, sy = (dy >= 0.f) ? FS : -FS;
    const float slope = __fdividef(fminf(ax, ay), fmaxf(ax, ay));
    const int oa = ax >= ay ? sx : sy, od = sx + sy;
    e.gx = g.x;
    e.gy = g.y;
    e.Map = grad_mag(at[oa]);
    e.Mdp = grad_mag(at[od]);
    e.Mam = grad_mag(at[-oa]);
    e.Mdm = grad_mag(at[-od]);
    const float fp = e.Map * (1.f - slope) + e.Mdp * slope;
    const float fm = e.Mam * (1.f - slope) + e.Mdm * slope;
    const bool maxt = (mv > fm && mv >= fp) || (mv >= fm && mv > fp);  // :466-468
    // s* = -B/(2A) with A = (fm+fp-2f)/(2s^2), B = (fp-fm)/(2s), s = sqrt(1 +
    // slope^2) (:471-476), kept when |s*| <= sqrt(2) (:478), tested as
    // |fp - fm| s <= 2 sqrt(2) |fm + fp - 2f| without the division.  The max
    // test gives fm + fp <= 2f, so the denominator is negative unless it is
    // zero, where s* is inf or 0/0 and the point is rejected as before.
    const float num = fp - fm, den = fm + fp - 2.f * mv;
    bool dir = true;
    if (TOD) {  // a direction to go along
        const float tm = sqrtf(fmaf(tx, tx, ty * ty));
        dir = tm > 0.f && isfinite(tm);
    }
    // mv > thr: cpu_toed.cpp:403 (also rejects NaN); the gradient epsilon: :407
    return (mv > thr) && !(fabsf(g.x) < 10e-6f && fabsf(g.y) < 10e-6f) && dir && maxt && den < 0.f &&
           fabsf(num) * sqrt_approx(fmaf(slope, slope, 1.f)) <= -2.82842712f * den;
}

// The seven higher derivatives at 2x-grid slot (m, c) of the step window
// from the row-pass ring (the Q planes hold the Gxx / Gxxx row responses):
// fxx, fxy, fyy, fxxy, fxyy, fxxx, fyyy, contracted with the y taps of the
// point's sub-grid.  Used by the per-edgel stage and, in the corrected-normal
// mode, by the NMS decision, so that both see identical numbers.
template <int R>
__device__ __forceinline__ void gather_hi(const float2* __restrict__ sP, const float4* __restrict__ sTab, int rb, int m,
                                          int c, float (&d)[7], int* dbg = nullptr)
{
    using C = Cfg<R, true>;
    constexpr int NT = C::NT;
    const int a = m & 1, xe = c >> 1, b = c & 1;
    const int xv = b ? 2 : (a ? 1 : 0);
    const int yv = a ? 2 : (b ? 1 : 0);
    const float2* Pp = sP + xv * C::RING * C::PS + xe;
    const float2* Qp = sP + (3 + xv) * C::RING * C::PS + xe;
    const float4* tab = sTab + yv * NT;
    float fxy = 0.f, fyy = 0.f, fxyy = 0.f, fyyy = 0.f, fxx = 0.f, fxxy = 0.f, fxxx = 0.f;
    const int h0 = rb + (m >> 1);
#ifdef TOED_DEBUG_BOUNDS
    if (!TOED_IN_BOUNDS(xe >= 0 && xe < kExt && h0 >= 0 && h0 + NT - 1 < 2 * C::RING, dbg)) {
        for (int f = 0; f < 7; ++f) d[f] = 0.f;
        return;
    }
#endif
    // window row kk is ring row hw + kk, less RING from kk = tw on
    const int hw = ring_wrap<C::RING>(h0), tw = C::RING - hw;
    const float2* Pb = Pp + hw * C::PS;
    const float2* Qb = Qp + hw * C::PS;
#pragma unroll
    for (int kk = 0; kk < NT; ++kk) {
        const int ph = kk * C::PS - ((kk >= tw) ? C::RING * C::PS : 0);
        const float2 hp = Pb[ph];
        const float2 hq = Qb[ph];
        const float4 t = tab[NT - 1 - kk];
        fxy = fmaf(hp.y, t.y, fxy);
        fyy = fmaf(hp.x, t.z, fyy);
        fxyy = fmaf(hp.y, t.z, fxyy);
        fyyy = fmaf(hp.x, t.w, fyyy);
        fxx = fmaf(hq.x, t.x, fxx);
        fxxy = fmaf(hq.x, t.y, fxxy);
        fxxx = fmaf(hq.y, t.x, fxxx);
    }
    d[0] = fxx; d[1] = fxy; d[2] = fyy; d[3] = fxxy; d[4] = fxyy; d[5] = fxxx; d[6] = fyyy;
}

// Bounded wait (one thread) until a copy group's ready flag reads `epoch`:
// the copy engine writes the flag after the group's pixels, in stream order.
// Returns false -- the unit is skipped -- once `spins` polls have gone by, or
// while the flag is not yet set and some CTA's wait has already given up
// (TOED_FLAG_TIMEOUT in words[2], checked after the first poll and every 256
// polls): a lost copy costs one bounded wait per resident CTA, not one per
// work unit, and units whose group did arrive are still detected.
static __device__ __noinline__ bool wait_ready(const int* flag, int epoch, int spins, int* words)
{
    for (int it = 0; it < spins; ++it) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v == epoch) {
            asm volatile("fence.proxy.async;" ::: "memory");  // the pixels are read by TMA
            return true;
        }
        if ((it & 255) == 0) {
            int f;
            asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(f) : "l"(words + 2) : "memory");
            if (f & TOED_FLAG_TIMEOUT) return false;
        }
        __nanosleep(256);
    }
    atomicOr(&words[2], TOED_FLAG_TIMEOUT);
    return false;
}

// Input rows: by TMA (DetImage::tma; float32 with 16-byte aligned rows), boxes
// of 16 rows up to three ahead in a ring of three buffers that the row pass
// reads in place; otherwise every warp loads the two rows of a box that it
// alone reads, one box ahead in registers (8-bit rows a word a lane), and
// converts them.  Either way the
// rows need no barrier of their own: two per step are left, row pass -> column
// pass and column pass -> NMS (six when rows were converted into a ring and
// the points listed for the whole CTA).
// NMSTO: NMS and peak fit along the corrected normal (TOED_NMS_TO_NORMAL).
template <int R, bool NMSTO = false>
__global__ void __launch_bounds__(kThreads, Cfg<R, NMSTO>::MINB)
    toed_detect_kernel(const __grid_constant__ BatchParams p)
{
    using C = Cfg<R, NMSTO>;
    constexpr int B = C::B;
    static_assert(kThreads / 32 == 8 && kExt == 32, "column pass: one warp per (sub-grid, 8-row group)");
    static_assert(kThreads == B * (kExt / 2), "row pass: a thread per (row, column pair), a warp per two rows");
    static_assert(C::WROWS == 4, "NMS: four 2x-grid rows per warp");
    static_assert(C::NIN + 3 <= 64, "a row's window: two floats a lane, or four bytes a half-warp's lane");
    extern __shared__ __align__(128) unsigned char smem[];
    float* sRaw = reinterpret_cast<float*>(smem + C::off_raw);
    float2* sP = reinterpret_cast<float2*>(smem + C::off_P);
    float2* sFxy = reinterpret_cast<float2*>(smem + C::off_fxy);
    unsigned* sMask = reinterpret_cast<unsigned*>(smem + C::off_mask);  // [MS][2] threshold ballots
    float4* sTab = reinterpret_cast<float4*>(smem + C::off_tab);        // NMSTO only
    int* sScal = reinterpret_cast<int*>(smem + C::off_misc);            // [0..1] next unit [2] pixels are in
    const uint32_t bar = smem_addr(smem + C::off_mbar);

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const TapBlock& tp = p.taps;
    unsigned short* wlist = reinterpret_cast<unsigned short*>(smem + C::off_list) + wid * C::MAXC;  // this warp's points
    const int brow = tid / (kExt / 2), bk = tid % (kExt / 2);  // row pass: row of a box, column pair
    const int sg = wid & 3, g = wid >> 2;  // column pass: sub-grid (a, b), 8-row group
    const int a = sg >> 1, b = sg & 1;

    if (NMSTO) {
        // y-direction tap table for the higher derivatives: [variant][k] = (G, Gy, Gyy, Gyyy)
        constexpr int NT = C::NT;
        for (int i = tid; i < 3 * NT; i += kThreads) {
            const int v = i / NT, k = i % NT;
            const int f = (v == 2) ? 4 : 0;
            float4 t = make_float4(tp.v[f][k], tp.v[f + 1][k], tp.v[f + 2][k], tp.v[f + 3][k]);
            if (v == 0 && (k == 0 || k == NT - 1)) t = make_float4(0.f, 0.f, 0.f, 0.f);
            sTab[i] = t;
        }
    }
    launch_dependents();
    // the scan, which runs after this kernel, takes tiles by a ticket and
    // publishes tile states: both start at zero
    for (int i = blockIdx.x * kThreads + tid; i < p.n_tiles; i += gridDim.x * kThreads) p.sc.tile_state[i] = 0ull;
    for (int i = blockIdx.x * kThreads + tid; i < p.n_bands; i += gridDim.x * kThreads) p.sc.band[i] = 0;
    if (blockIdx.x == 0 && tid == 0) p.sc.words[3] = 0;
    int stg_next = 0, stg_end = 0;  // this warp's reserved staging range [next, end) (uniform)
    if (tid == 0) {
        for (int q = 0; q < C::NBUF; ++q) mbar_init(bar + 8 * q);
        sScal[0] = atomicAdd(&p.sc.words[0], 1);
    }
    __syncthreads();
    int bi = 0;             // buffer of the next box to arrive by TMA
    uint32_t phase = 0;     // its mbarrier's phase
    bool dead = false;      // a wait for a box gave up
    int slot = 0;           // of sScal that holds the unit

    for (;;) {
        const int u = sScal[slot];
        if (u >= p.n_units) break;
        // the next unit's number is fetched while this one is worked on; it is
        // read after this unit's last barrier, and its slot written again only
        // past the next unit's first
        slot ^= 1;
        if (tid == 0) sScal[slot] = atomicAdd(&p.sc.words[0], 1);
        const int k = find_image(p.n_img, u, [&](int i) { return p.img[i].unit_base; });
        const DetImage& im = p.img[k];
        const void* src = im.src;
        const long long pitch = im.pitch;
        const int H = im.H, W = im.W, dtype = im.dtype;
        const int local = u - im.unit_base;
        const int sr = local / im.nsc, sc = local - sr * im.nsc;
        const int ys = sr * im.S, x0 = sc * kInner;
        const int S_act = min(im.S, H - ys);
        if (im.wait_slot > 0) {  // pixels still arriving: wait for the group (uniform across the CTA)
            if (tid == 0)
                sScal[2] = wait_ready(p.ready + (im.wait_slot - 1), p.ready_epoch, p.ready_spins, p.sc.words) ? 1 : 0;
            __syncthreads();
            const int in = sScal[2];
            __syncthreads();
            if (!in) {
                // the copy never arrived: the unit finds no edgels (its row
                // segments are written empty, so the scan reads no
                // stale entries) and the call reports TOED_ERR_TIMEOUT
                for (int i = tid; i < 2 * S_act; i += kThreads)
                    if (TOED_IN_BOUNDS(im.seg_base + (long long)(2 * ys + i) * im.nsc + sc < p.sc.seg_cap, p.sc.words))
                        p.sc.seg[im.seg_base + (long long)(2 * ys + i) * im.nsc + sc] = make_int2(0, 0);
                continue;
            }
        }
        const int nsteps = (2 * S_act + 3 + 2 * B - 1) / (2 * B);
        const int nbox = C::Q0 + nsteps - 1;
        const int W2 = 2 * W;
        const int row_lo = max(p.border, 2 * ys), row_n = min(2 * H - p.border, 2 * ys + 2 * S_act) - row_lo;
        const int gc_base = 2 * (x0 - 1);
        // the strip's output columns inside the image's border: bit L <-> 2x column 2 L + parity
        unsigned colmask[2];
#pragma unroll
        for (int par = 0; par < 2; ++par) {
            const int Gc = gc_base + 2 * lane + par;
            colmask[par] = __ballot_sync(0xffffffffu, lane >= 1 && lane <= kInner && Gc >= p.border && Gc < W2 - p.border);
        }
        // Box q holds image rows row0(q) + 0..15: boxes 0 .. Q0 - 1 the first
        // step's window, box Q0 - 1 + s the new rows of step s >= 1.
        auto row0 = [&](int q) { return q < C::Q0 ? ys - R - 3 + q * B : ys + (q - C::Q0 + 1) * B + R; };
        const int xin = x0 - R - 2;  // image column of the window's first float
        const bool tma = im.tma != 0;
        const int x_al = floor4(xin);
        const int shift = tma ? xin - x_al : C::OFF;               // where the window starts in a staged row
        int issued = 0, ib = bi;  // thread 0: boxes requested, the next one's buffer
        auto issue = [&](int upto) {
            for (; issued < min(nbox, upto) && !dead; ++issued) {
                tma_load_rows(&p.tmap[k], smem_addr(sRaw + ib * (B * C::BW)), bar + 8 * ib, x_al, row0(issued),
                              (uint32_t)C::box_bytes);
                ib = ib + 1 == C::NBUF ? 0 : ib + 1;
            }
        };
        // this warp's two rows of box q, zero outside the image: float32, columns
        // lane and lane + 32 of both; 8 bits, four columns of one a lane
        const bool u8 = dtype == TOED_U8;
        float pre[4];
        Bytes4 pre8;
        auto fetch = [&](int q) {
            if (u8) {
                pre8 = fetch_bytes(src, pitch, H, W, row0(q) + 2 * wid + (lane >> 4), xin, lane & 15, C::NIN);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c = lane + 32 * (e & 1);
                    pre[e] = c < C::NIN ? fetch_px(static_cast<const float*>(src), pitch, H, W,
                                                   row0(q) + 2 * wid + (e >> 1), xin + c)
                                        : 0.f;
                }
            }
        };
        if (tma) {
            if (tid == 0) issue(C::NBUF);
        } else {
            fetch(0);
        }
        // the 2x-grid rows 0 and 1 of a step's NMS window are rows 2B, 2B + 1
        // of the step before: kept by the threads that formed them
        float2 fcarry = make_float2(0.f, 0.f);
        unsigned mcarry = 0u;
        // segment of the lane's 2x row (lanes 0..3), advancing by 2B rows a step
        int2* seg = p.sc.seg + im.seg_base + (long long)(2 * ys - 4 + 1 + C::WROWS * wid + lane) * im.nsc + sc;
        int rb = 0;
        for (int s = 0; s < nsteps; ++s) {
            // logical slot h <-> ring row (rb + h) mod RING <-> ext row
            // s*B - R - 2 + h <-> image row ys - 1 + ext row
            // ---- 1, 2. input rows, row pass ---------------------------------
            const int qa = s == 0 ? 0 : C::Q0 - 1 + s, qb = s == 0 ? C::Q0 : qa + 1;
            for (int q = qa; q < qb; ++q) {
                const int h0 = s == 0 ? q * B : 2 * R + 3;  // slot of the box's row 0
                float* box = sRaw + bi * (B * C::BW);
                if (tma) {
                    if (!dead && !mbar_wait(bar + 8 * bi, phase)) {
                        dead = true;
                        atomicOr(&p.sc.words[2], TOED_FLAG_TIMEOUT);
                        // once more for what is in flight, nothing of which may outlive
                        // the CTA's memory (thread 0 requests no more boxes)
                        if (tid == 0)
                            for (int k = q, b = bi, ph = phase; k < issued; ++k) {
                                mbar_wait(bar + 8 * b, ph);
                                if (++b == C::NBUF) {
                                    b = 0;
                                    ph ^= 1;
                                }
                            }
                    }
                } else {
                    __syncwarp();
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int c = u8 ? pre8.c + e : lane + 32 * (e & 1);
                        const int row = 2 * wid + (u8 ? lane >> 4 : e >> 1);
                        if ((unsigned)c < (unsigned)C::NIN && TOED_IN_BOUNDS(shift + c < C::BW, p.sc.words))
                            box[row * C::BW + shift + c] = u8 ? (float)((pre8.w >> (8 * e)) & 255u) : pre[e];
                    }
                    __syncwarp();
                    if (q + 1 < nbox) fetch(q + 1);
                }
                if (h0 + brow < C::HS)
                    row_pass<R, NMSTO>(box + brow * C::BW + (shift - C::OFF) + 2 * bk, bk,
                                       ring_wrap<C::RING>(ring_wrap<C::RING>(rb + h0) + brow), sP, tp, p.sc.words);
                if (tma && ++bi == C::NBUF) {  // (a warp's own rows need no second buffer)
                    bi = 0;
                    phase ^= 1u;
                }
            }
            __syncthreads();
            if (tma && tid == 0) issue(qb + C::NBUF);  // the qb boxes read so far are free again
            // ---- 3. column pass: Ix, Iy for 2x rows m = 2..2B+1, and the
            // threshold test as ballots over the strip's columns
            const int gr_base = 2 * ys - 4 + 2 * s * B;  // global 2x row of NMS row m: gr_base + m
            {
                float2* out = sFxy + (2 * g * kColRows + a + 2) * kFxyStride + 2 * lane + b;
                unsigned* mout = sMask + (2 * g * kColRows + a + 2) * 2 + b;
                if (g == 1) {
                    sFxy[a * kFxyStride + 2 * lane + b] = fcarry;
                    if (lane == 0) sMask[a * 2 + b] = mcarry;
                }
                float2 f[kColRows];
                // sub-grid (a, b): x taps T / F / S for (0,0) / (1,0) / (.,1),
                // y taps truncated for (0,0), full for (0,1), shifted for (1,.)
                const float2* P = sP + (sg == 0 ? 0 : (sg == 2 ? 1 : 2)) * C::RING * C::PS;
                if (sg == 0)
                    col_pass<R, 0>(P, rb, g, lane, p.ytap, f);
                else if (sg == 1)
                    col_pass<R, 1>(P, rb, g, lane, p.ytap, f);
                else
                    col_pass<R, 2>(P, rb, g, lane, p.ytap, f);
#pragma unroll
                for (int o = 0; o < kColRows; ++o) {
                    out[2 * o * kFxyStride] = f[o];
                    // cpu_toed.cpp:403 as a prefilter on the squared magnitude (thr2 a
                    // little below thr^2, so the list holds every point nms_decide's exact
                    // test `|grad I| > thr` keeps; no square root per point)
                    const unsigned bal = __ballot_sync(0xffffffffu, fmaf(f[o].x, f[o].x, f[o].y * f[o].y) > p.thr2);
                    if (lane == 0) mout[4 * o] = bal;
                    if (o == kColRows - 1) mcarry = bal;
                }
                fcarry = f[kColRows - 1];
            }
            __syncthreads();
            // ---- 4. each warp decides the points above the threshold of its
            // own four 2x-grid rows, m = m0 .. m0 + 3, and stages the edgels:
            // no barrier from here to the next step's row pass
            {
                const int m0 = 1 + C::WROWS * wid;
                // mask (m, parity): bit L <-> 2x column 2 L + parity; the points listed row-major
                int LA = 0, first = 0;  // points; where the lane's row starts (lanes 0..3)
#pragma unroll
                for (int q = 0; q < C::WROWS; ++q) {
                    uint2 mk = *reinterpret_cast<const uint2*>(sMask + (m0 + q) * 2);
                    const bool in = (unsigned)(gr_base + m0 + q - row_lo) < (unsigned)max(row_n, 0);
                    mk.x = in ? mk.x & colmask[0] : 0u;
                    mk.y = in ? mk.y & colmask[1] : 0u;
                    if (lane == q) first = LA;
                    const unsigned k0 = (mk.x >> lane) & 1u, k1 = (mk.y >> lane) & 1u;
                    const int pos = LA + __popc(mk.x & lt) + __popc(mk.y & lt);
                    const unsigned short e = (unsigned short)(((m0 + q) << 6) | (2 * lane));
                    if (k0 && TOED_IN_BOUNDS(pos < C::MAXC, p.sc.words)) wlist[pos] = e;
                    if (k1 && TOED_IN_BOUNDS(pos + (int)k0 < C::MAXC, p.sc.words)) wlist[pos + k0] = e + 1;
                    LA += __popc(mk.x) + __popc(mk.y);
                }
                int last = __shfl_down_sync(0xffffffffu, first, 1);  // where it ends
                if (lane == C::WROWS - 1) last = LA;
                __syncwarp();
                auto decide = [&](int rec, NmsPoint& e) {
                    const int m = rec >> 6, c = rec & 63;
                    if (NMSTO) {
                        float d7[7], tx, ty;
                        gather_hi<R>(sP, sTab, rb, m, c, d7, p.sc.words);
                        const float2 g = sFxy[m * kFxyStride + c];
                        to_vec32(g.x, g.y, d7, &tx, &ty);
                        return nms_decide<true>(sFxy, m, c, p.thr, e, tx, ty, p.sc.words);
                    }
                    return nms_decide(sFxy, m, c, p.thr, e, 0.f, 0.f, p.sc.words);
                };
                // staging slots for n edgels: carved from the warp's reserved
                // range, refilled from the global cursor; more than an eighth
                // of a reservation block at once is reserved by itself, so that
                // less than an eighth of a block is left behind when it is
                // (the staging area has room for that: staging_records)
                auto reserve = [&](int n) {
                    int base = stg_next;
                    if (stg_next + n <= stg_end) {
                        stg_next += n;
                    } else {
                        const bool whole = n * 8 > p.stage_blk;
                        int got = 0;
                        if (lane == 0) got = atomicAdd(&p.sc.words[1], whole ? n : p.stage_blk);
                        base = __shfl_sync(0xffffffffu, got, 0);
                        if (!whole) {
                            stg_next = base + n;
                            stg_end = base + p.stage_blk;
                        }
                    }
                    return base;
                };
                auto stage = [&](int dst, int rec, const NmsPoint& e) {
                    const int m = rec >> 6, c = rec & 63;
                    if (dst >= p.sc.staging_cap) {
                        atomicOr(&p.sc.words[2], TOED_FLAG_STAGING_FULL);
                        return;
                    }
                    float4* r = det_stage(p.sc) + 2 * (long long)dst;
                    r[0] = make_float4(e.gx, e.gy, e.Map, e.Mdp);
                    r[1] = make_float4(e.Mam, e.Mdm, __int_as_float((gr_base + m) * W2 + gc_base + c), 0.f);
                };
                int base = 0, off = 0, cnt = 0;  // staging; the lane's row (lanes 0..3): edgels before it, its edgels
                if (LA <= 32) {
                    // one round: the values stay in registers
                    const int rec = lane < LA ? wlist[lane] : 0;
                    NmsPoint e;
                    bool acc = false;
                    if (lane < LA) acc = decide(rec, e);
                    const unsigned bal = __ballot_sync(0xffffffffu, acc);
                    if (lane < C::WROWS) {
                        off = __popc(bal & (unsigned)((1ull << first) - 1));
                        cnt = __popc(bal & (unsigned)((1ull << last) - 1)) - off;
                    }
                    if (bal) {
                        base = reserve(__popc(bal));
                        if (acc) stage(base + __popc(bal & lt), rec, e);
                    }
                } else {
                    // survivors compacted in place, order kept (their rank never
                    // exceeds their list position); their values formed again
                    int nacc = 0;
                    for (int e0 = 0; e0 < LA; e0 += 32) {
                        const int rec = e0 + lane < LA ? wlist[e0 + lane] : 0;
                        NmsPoint e;
                        bool acc = false;
                        if (e0 + lane < LA) acc = decide(rec, e);
                        const unsigned bal = __ballot_sync(0xffffffffu, acc);
                        if (lane < C::WROWS) {
                            const int f0 = min(32, max(0, first - e0)), f1 = min(32, max(0, last - e0));
                            const int before = __popc(bal & (unsigned)((1ull << f0) - 1));
                            off += before;
                            cnt += __popc(bal & (unsigned)((1ull << f1) - 1)) - before;
                        }
                        if (acc) wlist[nacc + __popc(bal & lt)] = (unsigned short)rec;
                        nacc += __popc(bal);
                        __syncwarp();
                    }
                    if (nacc > 0) {
                        base = reserve(nacc);
                        for (int e0 = lane; e0 < nacc; e0 += 32) {
                            const int rec = wlist[e0];
                            NmsPoint e;
                            decide(rec, e);
                            stage(base + e0, rec, e);
                        }
                    }
                }
                // the row-segment table: {staging offset, count} per 2x row
                const int Gr = gr_base + m0 + lane;
                if (lane < C::WROWS && Gr >= 2 * ys && Gr < 2 * ys + 2 * S_act &&
                    TOED_IN_BOUNDS(seg - p.sc.seg < p.sc.seg_cap, p.sc.words))
                    *seg = make_int2(base + off, cnt);
                seg += 2 * B * (long long)im.nsc;
            }
            if (NMSTO) __syncthreads();  // the next row pass overwrites rows that the points' sums read
            rb = ring_wrap<C::RING>(rb + B);
        }
    }
}

}  // namespace toed
