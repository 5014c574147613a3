// toed_groups.h -- which aligned groups of four pixels of an image the adjoint
// copies to shared memory, as host and device code (the CPU tests run it over
// small images of every size, pitch and alignment).
//
// An image's storage is its `span` = (H - 1) pitch + W pixels from the first to
// the last.  The first lies `skew` pixels past a group boundary, and pixels
// count from that boundary: storage is [skew, skew + span).  A group that lies
// only partly in it, the storage's first or last, is never copied: its other
// pixels are not the caller's.  An edgel whose window needs such a group is
// evaluated from single pixels instead (window_cut).
#pragma once

#ifdef __CUDACC__
#define TOED_HD __host__ __device__ __forceinline__
#else
#define TOED_HD inline
#endif

namespace toed {

// Groups wholly in storage start less than this many pixels past its first.
TOED_HD unsigned whole_groups(long long span) { return span >= 4 ? (unsigned)(span - 3) : 0u; }

// Whether the group of pixel `at` is copied for a window row of NU pixels, of
// which this is the l-th group: at = the row's first pixel + 4 l.  (A row of
// NU = 1 (mod 4) pixels needs CH groups wherever it starts.)
template <int NU, int CH>
TOED_HD bool group_copied(int at, int l, int skew, unsigned whole)
{
    const bool of_row = NU % 4 == 1 ? l < CH : 4 * l - (at & 3) < NU;
    return of_row && (unsigned)((at & ~3) - skew) < whole;
}

// Whether the NU x NU window with corner (wy, wx), which reaches the image,
// holds an image pixel of a group that is not copied.  For W >= 4 those are up
// to three pixels at the first row's start and up to three at the last row's end.
TOED_HD bool window_cut(int wy, int wx, int NU, int H, int W, int skew, long long span)
{
    const int tail = (int)((skew + span) & 3);
    return (skew != 0 && wy <= 0 && wx + skew <= 3) || (tail != 0 && wy + NU >= H && wx + NU > W - tail);
}

}  // namespace toed
