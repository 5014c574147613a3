// toed_edgels.cu -- from the detection's staged records and row-segment table
// to each image's edgel list in the reference's order (row-major over the 2x
// grid, cpu_toed.cpp:510-538), in two launches:
//
//   fin_scan     every segment's place in its image's list.  A tile is
//                p.seg_tile consecutive segments -- (2x-grid row, strip column)
//                pairs, row-major per image -- and one CTA's work: it scans
//                its counts and adds the sum of the image's earlier tiles,
//                which every tile publishes as soon as it has its own (a
//                chained scan with look-back: tiles are taken in order by a
//                ticket, so every earlier tile is running or done, and the
//                bounded wait ends);
//   fin_edgels   the edgels themselves.  A CTA takes the segments of one strip
//                column over p.ed_rows image rows and stages the pixels that
//                their windows cover in shared memory once; then a thread per
//                edgel runs the peak fit and contracts the seven higher
//                derivatives from its (2r+3)^2 window -- each row's four
//                x responses, then their products with the row's y taps --
//                forms the third-order orientation (cpu_toed.cpp:227-232) and
//                writes the edgel.  In HYBRID precision the orientations of
//                edgels whose vector nearly cancels are formed again in FP64,
//                a warp each, and written over.
//
// The x taps depend on the parity of the edgel's 2x column alone, so a chunk's
// edgels are ordered by it and every warp runs one fully unrolled row of
// compile-time operands.  It is bound by latency and issue: 94 warp
// instructions an edgel at half the issue slots, 390 us for the 2.5 M edgels of
// 78.8 Mpixel at r = 6 (scan 35 us), against 0.6 ms of the detection kernel's
// former time and 80 us of three ordering kernels.  The lists come out bit for
// bit as they did.  (Eight lanes an edgel, a lane per window column straight
// from global memory, takes the same 394 us but sums in another order; 96 rows
// a tile instead of up to 192 leave warps a third empty.)
#include "toed_common.cuh"
#include "toed_edgel.cuh"
#include "toed_internal.h"

namespace toed {

namespace {

constexpr int kScanThreads = 256;
constexpr int kEdThreads = 256;
constexpr int kEdChunk = kEdThreads - 32;  // edgels at a time: ordered by parity, each kind from a warp's start
constexpr int kRefineMost = 8;           // edgels a warp forms again in FP64 before their orientations
constexpr int kLookBackSpins = 1 << 22;  // polls before the wait for an earlier tile gives up (seconds)

__device__ __forceinline__ unsigned long long ld_state(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_state(unsigned long long* p, unsigned flag, int count)
{
    const unsigned long long v = ((unsigned long long)flag << 32) | (unsigned)count;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Edgels in the image's tiles before t (t0 its first), by one warp; publishes
// the sum up to and with t.
__device__ __forceinline__ int look_back(const BatchParams& p, int t, int t0, int total, int lane)
{
    unsigned long long* st = p.sc.tile_state;
    int excl = 0;
    if (t > t0) {
        if (lane == 0) st_state(st + t, 1, total);
        int spins = 0;
        for (int j = t - 1;;) {
            const int i = j - lane;
            const unsigned long long s = i >= t0 ? ld_state(st + i) : 2ull << 32;
            const unsigned f = (unsigned)(s >> 32);
            const unsigned done = __ballot_sync(0xffffffffu, f == 2), none = __ballot_sync(0xffffffffu, f == 0);
            const int last = done ? __ffs(done) - 1 : 31;  // the nearest tile whose sum is known, or all 32
            if (none & (0xffffffffu >> (31 - last))) {
                if (++spins > kLookBackSpins) {
                    if (lane == 0) atomicOr(&p.sc.words[2], TOED_FLAG_TIMEOUT);
                    break;
                }
                continue;
            }
            excl += __reduce_add_sync(0xffffffffu, lane <= last ? (int)(unsigned)s : 0);
            if (done) break;
            j -= 32;
        }
    }
    if (lane == 0) st_state(st + t, 2, excl + total);
    return excl;
}

// PER: segments a thread.
template <int PER>
__global__ void __launch_bounds__(kScanThreads) fin_scan(const __grid_constant__ BatchParams p)
{
    constexpr int kTile = PER * kScanThreads;
    __shared__ int s_warp[33];
    __shared__ int s_scal[2];  // tile, its place in the list
    const int tid = threadIdx.x;
    launch_dependents();
    grid_wait();
    if (tid == 0) s_scal[0] = atomicAdd(&p.sc.words[3], 1);
    __syncthreads();
    const int t = s_scal[0];
    const int k = find_image(p.n_img, t, [&](int i) { return p.img[i].tile_base; });
    const DetImage& im = p.img[k];
    // (an image's segments are padded to whole tiles, so whole groups are read and written)
    const long long q0 = (long long)(t - im.tile_base) * kTile + tid * PER, left = im.nseg - q0;
    const int4* seg = reinterpret_cast<const int4*>(p.sc.seg + im.seg_base + q0);
    int cnt[PER], sum = 0;
#pragma unroll
    for (int u = 0; u < PER; u += 2) {
        const int4 sg = u < left ? seg[u / 2] : make_int4(0, 0, 0, 0);
        cnt[u] = sg.y;
        cnt[u + 1] = u + 1 < left ? sg.w : 0;
        sum += cnt[u] + cnt[u + 1];
    }
    int total;
    int run = block_excl_scan<kScanThreads>(sum, s_warp, &total);
    if (tid < 32) {
        const int excl = look_back(p, t, im.tile_base, total, tid);
        if (tid == 0) {
            s_scal[1] = excl;
            if (t + 1 == (k + 1 < p.n_img ? p.img[k + 1].tile_base : p.n_tiles)) {  // the image's last tile
                *im.count = excl + total;
                if (excl + total > im.cap) atomicOr(&p.sc.words[2], TOED_FLAG_OVER_CAPACITY);
            }
        }
    }
    __syncthreads();
    run += s_scal[1];
    int4* dst = reinterpret_cast<int4*>(p.sc.seg_dst + im.seg_base + q0);
#pragma unroll
    for (int u = 0; u < PER; u += 4) {
        int4 d;
        d.x = run;
        d.y = d.x + cnt[u];
        d.z = d.y + cnt[u + 1];
        d.w = d.z + cnt[u + 2];
        run = d.w + cnt[u + 3];
        if (u < left) dst[u / 4] = d;
    }
}

// One edgel, one warp: the nine derivatives at 2x-grid point (Gr, Gc) =
// (2i + a, 2j + b) from the staged pixels (win: the corner of its (2r+3)^2
// window, rows `pitch` apart) with FP64 taps -- the (2r+1)^2 window of
// unshifted taps on sub-grid (0, 0) (cpu_toed.cpp:205-221), the (2r+3)^2
// window with the half-pixel shifted taps along the odd axes elsewhere
// (cpu_toed.cpp:246-344) -- into out[0..8].  Lane t forms the four
// column-filtered sums of one window row; the row filters then weight them and
// the warp sums them by halving exchanges: an SM's FP64 pipe takes about 15
// cycles for a warp's instruction, so the sums take 12 additions instead of a
// butterfly's 45.  Out of line: it is rare, and inlined its registers would
// crowd the FP32 contraction.
__device__ __noinline__ void refine_edgel(const BatchParams& p, const float* __restrict__ win, int pitch, int a, int b,
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

}  // namespace

template <int R>
struct EdCfg {
    static constexpr int NT = 2 * R + 3;            // window side
    static constexpr int TW = kInner + 2 * R + 2;   // columns of a tile's pixels
    static constexpr int TP = staged_width(R);      // their pitch in shared memory: a box of the detection's row map
    static __host__ __device__ constexpr int boxes(int rows) { return (rows + 2 * R + 2 + kStepRows - 1) / kStepRows; }
    static constexpr size_t smem(int rows) { return sizeof(float) * TP * boxes(rows) * kStepRows; }
};

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
        for (int t = 0; t < NT; ++t) v[t] = win[kk * EdCfg<R>::TP + t];
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

template <int R>
__global__ void __launch_bounds__(kEdThreads, R <= 8 ? 3 : 2) fin_edgels(const __grid_constant__ BatchParams p)
{
    using E = EdCfg<R>;
    constexpr int NT = E::NT, TP = E::TP;
    extern __shared__ __align__(128) float sPix[];
    __shared__ int s_warp[33];
    __shared__ float4 sTab[3 * NT];      // y taps per variant T, F, S: (G, Gy, Gyy, Gyyy) of tap k
    __shared__ int2 sList[kEdChunk];     // a chunk's edgels: staging slot, list position
    __shared__ Staged sRec[kEdThreads];  // their records, ordered
    __shared__ int sPos[kEdThreads];     // and list positions, -1: none; -2 - position: FP64 orientation wanted
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
    for (int i = tid; i < 3 * NT; i += kEdThreads) {
        const int v = i / NT, q = i - v * NT;
        const int f = (v == 2) ? 4 : 0;
        float4 w = make_float4(p.taps.v[f][q], p.taps.v[f + 1][q], p.taps.v[f + 2][q], p.taps.v[f + 3][q]);
        if (v == 0 && (q == 0 || q == NT - 1)) w = make_float4(0.f, 0.f, 0.f, 0.f);
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
            seg[u] = p.sc.seg[q];
            dst[u] = p.sc.seg_dst[q];
        }
        sum += seg[u].y;
    }
    int total;
    int run = block_excl_scan<kEdThreads>(sum, s_warp, &total);
    if (total == 0) return;
    // pixels x0 - r - 1 .. x0 + 30 + r, rows y0 - r - 1 .. y0 + nrow + r, zero
    // outside the image, by TMA where the detection kernel's rows came so
    const int px = sc * kInner - R - 1, py = y0 - R - 1;
    const int x_al = floor4(px - 1), shift = px - x_al;  // as the detection's boxes, of columns px - 1 ..
    const uint32_t bar = smem_addr(&sBar);
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
        const int nr = nrow + 2 * R + 2;
        constexpr int NC = (E::TW + 31) / 32;
#pragma unroll 4
        for (int r = wid; r < nr; r += kEdThreads / 32) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int col = lane + 32 * c;
                if (col < E::TW) {
                    const int y = py + r, x = px + col;
                    float v = 0.f;
                    if ((unsigned)y < (unsigned)H && (unsigned)x < (unsigned)W) {
                        const long long o = (long long)y * im.pitch + x;
                        v = im.dtype == TOED_U8 ? (float)__ldg(static_cast<const unsigned char*>(im.src) + o)
                                                : __ldg(static_cast<const float*>(im.src) + o);
                    }
                    sPix[r * TP + shift + col] = v;
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
        if (im.tma && c0 == 0 && !mbar_wait(bar, 0) && tid == 0) atomicOr(&p.sc.words[2], TOED_FLAG_TIMEOUT);
        const int n = min(kEdChunk, total - c0);
        Staged e = {};
        int pos = -1;
        if (tid < n) {
            const int2 l = sList[tid];
            if (l.y < cap && l.x < p.sc.staging_cap) {
                pos = l.y;
                e = load_staged(p.sc, l.x);
            }
        }
        const bool odd = (e.idx - e.idx / W2 * W2) & 1;
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
            sRec[to] = e;
            sPos[to] = pos;
        }
        __syncthreads();
        pos = sPos[tid];
        if (__any_sync(0xffffffffu, pos >= 0)) {
            e = sRec[pos >= 0 ? tid : (wid * 32)];  // a warp's first slot is used if any is
            const int Gr = e.idx / W2, Gc = e.idx - Gr * W2;
            const int a = Gr & 1, b = Gc & 1;
            const float* win = sPix + ((Gr >> 1) - y0) * TP + (Gc >> 1) - sc * kInner + shift;
            float d7[7];
            if (32 * wid < n0)
                window7<R, 0>(win, a, sTab + (a ? 2 : b) * NT, p.taps, d7);
            else
                window7<R, 1>(win, a, sTab + (a ? 2 : b) * NT, p.taps, d7);
            float tix, tiy, ori;
            to_vec32(e.gx, e.gy, d7, &tix, &tiy);
            const Fitted ft =
                fit_edgel(e, p.nms_to ? tix : e.gx, p.nms_to ? tiy : e.gy, p.nms_to != 0, p.hyb != 0, Gr, Gc);
            if (p.hyb) {
                ori = (tix == 0.f && tiy == 0.f) ? __int_as_float(0x7fc00000) : atan2f(tix, -tiy);
                if (pos >= 0 && cancels(e.gx, e.gy, d7, tix, tiy)) {
                    sPos[tid] = -2 - pos;
                    sFlag[atomicAdd(&sFlags, 1)] = (unsigned char)tid;
                }
            } else {
                const float fxx = d7[0], fxy = d7[1], fyy = d7[2], fxxy = d7[3], fxyy = d7[4], fxxx = d7[5], fyyy = d7[6];
                const float gx = e.gx, gy = e.gy;
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
                const int idx = sRec[sFlag[f]].idx;
                const int Gr = idx / W2, Gc = idx - Gr * W2;
                refine_edgel(p, sPix + ((Gr >> 1) - y0) * TP + (Gc >> 1) - sc * kInner + shift, TP, Gr & 1, Gc & 1, lane,
                             sD64[wid][m]);
            }
            __syncwarp();
            if (lane < m) {
                const int pos = -2 - sPos[sFlag[f0 + lane * (kEdThreads / 32)]];
                const float ori = orientation64(sD64[wid][lane]);
                if (p.out_f64)
                    static_cast<double*>(im.out)[4LL * pos + 2] = (double)ori;
                else
                    static_cast<float*>(im.out)[4LL * pos + 2] = ori;
            }
            __syncwarp();
        }
        __syncthreads();  // the next chunk overwrites the lists
    }
}

struct EdEntry {
    const void* func;
    size_t smem;  // at p.ed_rows
};

static EdEntry edgels_entry(int radius, int rows)
{
    switch (radius) {
#define TOED_ED_CASE(R) \
    case R: return {(const void*)fin_edgels<R>, EdCfg<R>::smem(rows)};
        TOED_ED_CASE(1) TOED_ED_CASE(2) TOED_ED_CASE(3) TOED_ED_CASE(4) TOED_ED_CASE(5) TOED_ED_CASE(6)
        TOED_ED_CASE(7) TOED_ED_CASE(8) TOED_ED_CASE(9) TOED_ED_CASE(10) TOED_ED_CASE(11) TOED_ED_CASE(12)
#undef TOED_ED_CASE
    default: return {nullptr, 0};
    }
}

static_assert(kEdRowsMax <= kEdThreads && kEdThreads % 32 == 0, "two segments a thread");

// The scan reads and writes whole 16-byte groups of an image's padded segments.
static const void* scan_fn(int seg_tile)
{
    return seg_tile == kScanTileMax ? (const void*)fin_scan<kScanTileMax / kScanThreads>
                                    : (const void*)fin_scan<kSegTile / kScanThreads>;
}

cudaError_t preload_edgels(int radius)
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, scan_fn(kSegTile));
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, scan_fn(kScanTileMax));
    return e == cudaSuccess ? prepare_edgels(radius) : e;
}

cudaError_t prepare_edgels(int radius)
{
    const EdEntry ent = edgels_entry(radius, kEdRowsMax);
    if (!ent.func) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(ent.func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ent.smem);
}

cudaError_t launch_edgels(const BatchParams& p, cudaStream_t stream)
{
    const EdEntry ent = edgels_entry(p.radius, p.ed_rows);
    if (!ent.func) return cudaErrorInvalidValue;
    void* args[] = {const_cast<BatchParams*>(&p)};
    const cudaError_t e = launch_after(scan_fn(p.seg_tile), dim3(p.n_tiles), dim3(kScanThreads), args, 0, stream);
    if (e != cudaSuccess) return e;
    return launch_after(ent.func, dim3(p.n_ed), dim3(kEdThreads), args, ent.smem, stream);
}

}  // namespace toed
