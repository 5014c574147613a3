// toed_common.cuh -- launch descriptors shared by the detection kernels and
// the host side of the C ABI.
//
// Data layout in HBM (all caller-owned except the scratch block):
//   image k      : H x pitch pixels (uint8 or float32), row-major
//   edgels k     : capacity x 4 (float32 or float64) [x, y, orientation, strength]
//   scratch      : work-queue / cursor / flags words, staging records (32 bytes
//                  an edgel), the row-segment table (int2 {staging offset, count}
//                  per (2x-grid row, strip column)), each segment's place in its
//                  list, and a word per tile of the scan.
#pragma once
#include <cstdint>
#include <cuda.h>  // CUtensorMap (the type only; encoding goes through the runtime's driver entry point)
#include <cuda_runtime.h>

#include "../../include/toed_gb300.h"

namespace toed {

constexpr int kMaxTaps = 2 * TOED_MAX_RADIUS + 3;  // taps of the widest (shifted/full) filter
constexpr int kBatchMax = 64;                      // images per launch (larger batches are chunked)
constexpr int kSizeClasses = 48;                   // launch size classes floor(log2(pixels)) of tuned shapes
constexpr int kThreads = 256;                      // threads per detection CTA
constexpr int kExt = 32;                           // strip width incl. a 1-pixel ring each side
constexpr int kInner = kExt - 2;                   // 30 output columns per strip
constexpr int kStepRows = 16;                      // original rows per sliding step (B)
constexpr int kColRows = 8;                        // rows per column-pass thread (register blocking)
constexpr int kSegTile = 1024;                     // segments per ordering-pass tile
constexpr int kEdRowsMax = 192;                    // image rows of an edgel-kernel tile at most
constexpr int kScanTileMax = 4096;                 // segments per tile of a large launch's scan
constexpr int kStageBlk = 64;                      // staging records a warp of the detection reserves at a time
// Edgels whose third-order vector cancels by more than this factor (sum of
// the terms' magnitudes over the largest component) get their orientation
// recomputed from the image in FP64 (HYBRID precision, grid orientation).
constexpr float kRefineKappa = 20.f;
// Default bound of the wait for a copy group's ready flag (polls ~256 ns
// apart: a few seconds), after which the kernel flags TOED_FLAG_TIMEOUT and
// skips the units whose pixels have not arrived (BatchParams::ready_spins).
constexpr int kReadySpinLimit = 1 << 24;

// Bounds-checked builds (-DTOED_DEBUG_BOUNDS, a separate debug library):
// TOED_IN_BOUNDS(cond, words) guards a shared- or global-memory access; a
// failed check skips the access, sets TOED_FLAG_BOUNDS in words[2] and
// records the source line of the first failure in words[4] -- a status the
// host reads, never a trap.  In release builds the macro is `true` and every
// guard compiles away.
#ifdef TOED_DEBUG_BOUNDS
__device__ __forceinline__ bool debug_in_bounds(bool ok, int* words, int line)
{
    if (!ok) {
        atomicOr(&words[2], TOED_FLAG_BOUNDS);
        atomicCAS(&words[4], 0, line);
    }
    return ok;
}
#define TOED_IN_BOUNDS(cond, words) ::toed::debug_in_bounds((cond), (words), __LINE__)
#else
#define TOED_IN_BOUNDS(cond, words) true
#endif
constexpr int kWords = 8;  // scratch words: [0] queue [1] cursor [2] flags [3] tile ticket [4] first bad line

// Floats of a staged input row of the detection (a multiple of 16 bytes): the
// window of kExt outputs at radius r, up to three floats of alignment before
// it and one past an odd window's last pair.
// An odd number of 16-byte groups: eight rows apart before a column meets its bank again.
__host__ __device__ constexpr int staged_width(int r) { return ((kExt + 2 * r + 2 + 4 + (r & 1) + 3) / 4 | 1) * 4; }

// 1-D taps, index k <-> offset x = k - (r+1) (+0.5 for the shifted set).
// Filters: 0 G, 1 Gx, 2 Gxx, 3 Gxxx, 4..7 the same shifted by +0.5.
// Passed by value as a kernel parameter, so unrolled loops read each tap as
// a constant-bank operand of the FMA.
struct TapBlock {
    float v[8][kMaxTaps];
};

// The same taps in FP64, for the orientation recomputation.
struct TapBlock64 {
    double v[8][kMaxTaps];
};

struct DetImage {
    const void* src;
    long long pitch;     // elements
    void* out;           // edgels
    int* count;          // user count word
    int* index;          // optional grid index output
    long long seg_base;  // first segment of this image (tile aligned)
    long long nseg;      // segments of this image (rows x strip/tile columns)
    int H, W;
    int dtype;
    int cap;
    int nsc, nsr;        // strip columns / strip rows
    int S;               // strip inner rows of this image's work units (multiple of kStepRows minus 2)
    int unit_base;       // first work unit
    int tile_base;       // first ordering tile
    int ed_base;         // first edgel-kernel tile
    int band_base;       // first band (row of edgel-kernel tiles) in Scratch::band
    void* host_out;      // mapped host memory that the list is copied to as its bands are complete, or null
    int* host_index;
    int* host_count;
    int tma;             // 1: rows arrive by TMA through BatchParams::tmap[k]; 0: by loads
    int wait_slot;       // 0: pixels ready at launch; g > 0: the copy engine is still bringing them in,
                         // BatchParams::ready[g - 1] reads ready_epoch once they are complete
};

struct Scratch {
    int* words;          // kWords: [0] unit queue, [1] staging cursor, [2] flags, [3] the scan's tile
                         // ticket, [4] (bounds-checked builds) source line of the first failed check
    double4_32a* staging;  // staged edgels, 32 bytes each: TO correction (x, y, orientation, strength);
                           // the detection two float4 (det_stage)
    int* staging_idx;      // TO correction: pixel of each staged edgel
    long long staging_cap;
    int2* seg;           // per segment {staging offset, count}
    long long seg_cap;   // segments `seg` holds
    int* tile_sum;       // TO correction: per ordering tile
    long long* img_base; // TO correction: per map, exclusive prefix of its first segment
    int* band;           // per band of an image with host_out: edgel-kernel tiles done
    int* seg_dst;        // per segment: its place in its image's list
    unsigned long long* tile_state;  // per scan tile: {0, 1 its count, 2 the count of its image's
                                     // tiles up to it} << 32 | count
};

// The detection's staged edgel, two float4: (Ix, Iy, |grad I| at the axis and
// the diagonal neighbour ahead), (the same behind, the 2x-grid index's bits,
// unused).
__device__ __forceinline__ float4* det_stage(const Scratch& sc) { return reinterpret_cast<float4*>(sc.staging); }

__device__ __forceinline__ float sqrt_approx(float x)
{
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// |grad I| at a 2x-grid point from its (Ix, Iy); the NMS decision and the
// peak fit both use this one expression.
__device__ __forceinline__ float grad_mag(float2 g) { return sqrt_approx(fmaf(g.x, g.x, g.y * g.y)); }

// The third-order vector (cpu_toed.cpp:227-230) in FP32 with its shared
// products factored out, d = fxx, fxy, fyy, fxxy, fxyy, fxxx, fyyy:
// TIx = 2 (fx (fxx^2 + fxy^2) + fy fxy (fxx + fyy) + fx fy fxxy) + fy^2 fxyy + fx^2 fxxx
// TIy = 2 (fx fxy (fxx + fyy) + fy (fyy^2 + fxy^2) + fx fy fxyy) + fx^2 fxxy + fy^2 fyyy
__device__ __forceinline__ void to_vec32(float gx, float gy, const float (&d)[7], float* tix, float* tiy)
{
    const float fxx = d[0], fxy = d[1], fyy = d[2], fxxy = d[3], fxyy = d[4], fxxx = d[5], fyyy = d[6];
    const float a2 = fmaf(fxx, fxx, fxy * fxy), c2 = fmaf(fyy, fyy, fxy * fxy), bc = fxy * (fxx + fyy);
    const float pxy = gx * gy, x2 = gx * gx, y2 = gy * gy;
    *tix = fmaf(2.f, fmaf(gx, a2, fmaf(gy, bc, pxy * fxxy)), fmaf(y2, fxyy, x2 * fxxx));
    *tiy = fmaf(2.f, fmaf(gx, bc, fmaf(gy, c2, pxy * fxyy)), fmaf(x2, fxxy, y2 * fyyy));
}

struct BatchParams {
    CUtensorMap tmap[kBatchMax];  // per image: 2-D map, box (staged_width x kStepRows), OOB zero fill
    TapBlock taps;
    TapBlock64 taps64;
    float2 ytap[2][kMaxTaps];  // (Gy, G) of the whole and the half-pixel shifted set: the column pass's pairs
    float thr;
    float thr2;          // candidate prefilter on |grad I|^2: a little below thr^2 (-1 when thr < 0)
    int border;
    int S;               // strip inner rows of most work units (multiple of kStepRows minus 2); the
                         // images at the end of the queue may use shorter ones (DetImage::S)
    int n_img;
    int n_units;
    int n_tiles;
    int out_f64;
    int radius;
    int stage_blk;       // staging records a warp reserves per atomic (1: exactly each step's edgels)
    int seg_tile;        // segments per ordering tile: kSegTile, or kScanTileMax
    int ed_rows;         // image rows of an edgel-kernel tile (one strip column wide), up to kEdRowsMax
    int n_ed;            // such tiles
    int n_bands;         // bands to count (0: no list goes to host memory)
    int hyb;             // 1: peak fit on exact FP32 differences, FP64 recomputation of ill-conditioned
                         // orientations (TOED_HYBRID)
    int qad;             // 1: orientation from derivatives interpolated at the subpixel point (TOED_ORI_QAD)
    int nms_to;          // 1: NMS and peak fit along the corrected normal (TOED_NMS_TO_NORMAL)
    const int* ready;    // per copy group: ready_epoch once the group's images are in device memory
    int ready_epoch;
    int ready_spins;     // polls of a ready flag before the wait gives up (TOED_FLAG_TIMEOUT)
    Scratch sc;
    DetImage img[kBatchMax];
};
static_assert(sizeof(BatchParams) <= 32764, "BatchParams is passed as one kernel parameter");

// Block-wide exclusive scan of one int per thread (NT threads); leaves the
// block total in *total.  s_warp: 33 ints of shared memory.
template <int NT>
__device__ __forceinline__ int block_excl_scan(int v, int* s_warp, int* total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        constexpr int NW = NT / 32;
        int w = (lane < NW) ? s_warp[lane] : 0;
        int wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi += y;
        }
        if (lane < NW) s_warp[lane] = wi - w;
        if (lane == NW - 1) s_warp[32] = wi;
    }
    __syncthreads();
    const int r = incl - v + s_warp[wid];
    *total = s_warp[32];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// TMA staging of input rows (cp.async.bulk.tensor + mbarrier)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One thread: one box of kStepRows rows at (x, y) of image map `tm` into `dst`.
__device__ __forceinline__ void tma_copy_rows(const CUtensorMap* tm, uint32_t dst, uint32_t bar, int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_rows(const CUtensorMap* tm, uint32_t dst, uint32_t bar, int x, int y,
                                              uint32_t bytes)
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    tma_copy_rows(tm, dst, bar, x, y);
}

// Bounded wait for the mbarrier phase: gives up after ~2^20 polls (each poll
// may suspend briefly) instead of hanging the SM.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase)
{
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(bar), "r"(phase)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Programmatic dependent launch: a kernel launched so (launch_after) may start
// while its predecessor in the stream still runs, once all of that one's CTAs
// have called launch_dependents() or ended; what it reads of the predecessors'
// results it reads after grid_wait(), which returns when they are complete.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

inline cudaError_t launch_after(const void* func, dim3 grid, dim3 block, void** args, size_t smem, cudaStream_t stream)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, func, args);
}

// Four 8-bit pixels of a row at once: lane l of 16 takes the 4-byte aligned
// word l of the row from column x0 on.  `c` is the word's first column less x0
// (-3..0 for l = 0); bytes outside the image (or the word, where it is not
// wholly inside the row) read as zero.
struct Bytes4 {
    unsigned w;
    int c;
};
__device__ __forceinline__ Bytes4 fetch_bytes(const void* src, long long pitch, int H, int W, int y, int x0, int l, int n)
{
    const unsigned char* row = static_cast<const unsigned char*>(src) + (long long)y * pitch + x0;
    Bytes4 b;
    b.c = 4 * l - (int)(reinterpret_cast<uintptr_t>(row) & 3u);
    b.w = 0u;
    const int x = x0 + b.c;
    if ((unsigned)y < (unsigned)H && b.c < n) {
        if (x >= 0 && x + 3 < W) {
            b.w = __ldg(reinterpret_cast<const unsigned*>(row + b.c));
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if ((unsigned)(x + e) < (unsigned)W) b.w |= (unsigned)__ldg(row + b.c + e) << (8 * e);
        }
    }
    return b;
}

// x rounded down to a multiple of 4 (floats: 16 bytes, where a TMA box may start).
__device__ __forceinline__ int floor4(int x) { return x >= 0 ? x & ~3 : -((3 - x) & ~3); }

// Index of the image whose [base, next base) range holds `u` (bases ascending).
template <typename GetBase>
__device__ __forceinline__ int find_image(int n_img, int u, GetBase base)
{
    int lo = 0, hi = n_img - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (base(mid) <= u) lo = mid; else hi = mid - 1;
    }
    return lo;
}

}  // namespace toed
