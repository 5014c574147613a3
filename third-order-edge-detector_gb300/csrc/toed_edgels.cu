// toed_edgels.cu -- from the detection's staged records and row-segment table
// to each image's edgel list in the reference's order (row-major over the 2x
// grid, cpu_toed.cpp:510-538), in two launches:
//
//   fin_scan     every segment's place in its image's list.  A tile is
//                p.seg_tile consecutive segments -- (2x-grid row, strip column)
//                pairs, row-major per image -- and one CTA's work: it scans
//                its counts and adds the sum of the image's earlier tiles,
//                which every tile publishes as soon as it has its own (the
//                single-pass scan with decoupled look-back of Merrill and
//                Garland, 2016: tiles are taken in order by a ticket, so every
//                earlier tile is running or done, and the bounded wait ends);
//   fin_edgels   the edgels themselves.  A CTA takes the segments of one strip
//                column over p.ed_rows image rows and stages the pixels that
//                their windows cover in shared memory once; then a thread per
//                edgel runs the peak fit and contracts the seven higher
//                derivatives from its (2r+3)^2 window -- each row's four
//                x responses, then their products with the row's y taps --
//                forms the third-order orientation (cpu_toed.cpp:227-232) and
//                writes the edgel.  In HYBRID precision the orientations of
//                edgels whose vector nearly cancels are formed again in FP64,
//                a warp each, and written over (toed_edgels.cuh).
//
// The edgel kernel is bound by latency and issue: 94 warp
// instructions an edgel at half the issue slots, 390 us for the 2.5 M edgels of
// 78.8 Mpixel at r = 6 (scan 35 us), against 0.6 ms of the detection kernel's
// former time and 80 us of three ordering kernels.  The lists come out bit for
// bit as they did.  (Eight lanes an edgel, a lane per window column straight
// from global memory, takes the same 394 us but sums in another order; 96 rows
// a tile instead of up to 192 leave warps a third empty.)
#include "toed_edgels.cuh"

namespace toed {

namespace {

constexpr int kScanThreads = 256;
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
    if (!TOED_IN_BOUNDS(t < p.n_tiles, p.sc.words)) return;
    const int k = find_image(p.n_img, t, [&](int i) { return p.img[i].tile_base; });
    const DetImage& im = p.img[k];
    // (an image's segments are padded to whole tiles, so whole groups are read and written)
    const long long q0 = (long long)(t - im.tile_base) * kTile + tid * PER, left = im.nseg - q0;
    const int4* seg = reinterpret_cast<const int4*>(p.sc.seg + im.seg_base + q0);
    int cnt[PER], sum = 0;
#pragma unroll
    for (int u = 0; u < PER; u += 2) {
        const int4 sg = u < left && TOED_IN_BOUNDS(im.seg_base + q0 + u + 2 <= p.sc.seg_cap, p.sc.words) ? seg[u / 2] : make_int4(0, 0, 0, 0);
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
                if (im.host_count) *im.host_count = excl + total;
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
        if (u < left && TOED_IN_BOUNDS(im.seg_base + q0 + u + 4 <= p.sc.seg_cap, p.sc.words)) dst[u / 4] = d;
    }
}

}  // namespace

// The scan reads and writes whole 16-byte groups of an image's padded segments.
static const void* scan_fn(int seg_tile)
{
    return seg_tile == kScanTileMax ? (const void*)fin_scan<kScanTileMax / kScanThreads>
                                    : (const void*)fin_scan<kSegTile / kScanThreads>;
}

cudaError_t prepare_edgels(int radius, bool qad) { return qad ? prepare_qad(radius) : prepare_edgels_as<false>(radius); }

cudaError_t preload_finalize(int radius, bool qad)
{
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, scan_fn(kSegTile));
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, scan_fn(kScanTileMax));
    return e == cudaSuccess ? prepare_edgels(radius, qad) : e;
}

cudaError_t launch_finalize(const BatchParams& p, cudaStream_t stream)
{
    void* args[] = {const_cast<BatchParams*>(&p)};
    const cudaError_t e = launch_after(scan_fn(p.seg_tile), dim3(p.n_tiles), dim3(kScanThreads), args, 0, stream);
    if (e != cudaSuccess) return e;
    return p.qad ? launch_qad(p, stream) : launch_edgels_as<false>(p, stream);
}

}  // namespace toed
