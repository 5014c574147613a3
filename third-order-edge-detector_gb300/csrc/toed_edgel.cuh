// toed_edgel.cuh -- one staged edgel of the detection: its record and the
// peak fit, shared by the edgel kernels (toed_edgels.cu, toed_qad.cu).
#pragma once
#include "toed_common.cuh"

namespace toed {

struct Staged {
    float gx, gy;              // Ix, Iy at the 2x-grid point
    float Map, Mdp, Mam, Mdm;  // |grad I| at the axis / diagonal neighbours ahead, then behind
    int idx;                   // 2x-grid index
};

__device__ __forceinline__ Staged load_staged(const Scratch& sc, long long src)
{
    const float4* r = det_stage(sc) + 2 * src;
    const float4 a = r[0], b = r[1];
    return {a.x, a.y, a.z, a.w, b.x, b.y, __float_as_int(b.z)};
}

struct Fitted {
    double x, y;  // output position ((pos - 1) / 2, cpu_toed.cpp:516-521)
    float str;
};

// Peak fit (cpu_toed.cpp:465-489) along (dx, dy): the gradient, or the
// third-order vector in the corrected-normal mode (tod).
__device__ __forceinline__ Fitted fit_edgel(const Staged& e, float dx, float dy, bool tod, bool hyb, int Gr, int Gc)
{
    Fitted o;
    const float mv = grad_mag(make_float2(e.gx, e.gy));
    float nx, ny;
    if (tod) {
        const float tm = sqrtf(fmaf(dx, dx, dy * dy));
        nx = dx / tm;
        ny = dy / tm;
    } else {
        nx = __fdividef(dx, mv);
        ny = __fdividef(dy, mv);
    }
    const float ax = fabsf(dx), ay = fabsf(dy);
    const float sl = __fdividef(fminf(ax, ay), fmaxf(ax, ay));
    if (hyb) {
        // fp - fm and fm + fp - 2f cancel.  With fp = Map + s (Mdp - Map) and
        // fm = Mam + s (Mdm - Mam) both are formed from differences of nearly
        // equal FP32 magnitudes (exact within a factor 2 of each other), the
        // interpolation weight applied last:
        //   fp - fm        = dA + s (dD - dA),  dA = Map - Mam, dD = Mdp - Mdm
        //   fm + fp - 2f   = eA + s (eD - eA),  eA = (Map - f) + (Mam - f), eD likewise
        // so no full-scale sum is rounded before the cancellation.
        const float dA = e.Map - e.Mam, dD = e.Mdp - e.Mdm;
        const float eA = (e.Map - mv) + (e.Mam - mv), eD = (e.Mdp - mv) + (e.Mdm - mv);
        const float num = fmaf(sl, dD - dA, dA);
        const float den = fmaf(sl, eD - eA, eA);
        const float ss = sqrtf(1.f + sl * sl);
        const float sst = -0.5f * num * ss / den;           // s* = -B / (2A)
        const float maxf = mv - 0.125f * num * num / den;   // A s*^2 + B s* + C
        // the grid coordinate is exact, so the FP32 subpixel offset added in
        // FP64 keeps its digits at large coordinates
        const float x = 0.5f * sst * nx, y = 0.5f * sst * ny;
        o.x = (double)(0.5f * (float)(Gc - 1)) + (double)x;
        o.y = (double)(0.5f * (float)(Gr - 1)) + (double)y;
        o.str = sqrtf((maxf * nx) * (maxf * nx) + (maxf * ny) * (maxf * ny));
    } else {
        const float fp = e.Map * (1.f - sl) + e.Mdp * sl;
        const float fm = e.Mam * (1.f - sl) + e.Mdm * sl;
        const float num = fp - fm, den = fm + fp - 2.f * mv;
        const float ss = sqrtf(1.f + sl * sl);
        const float sst = -0.5f * num * ss / den;
        const float maxf = mv - 0.125f * num * num / den;
        const float x = (float)Gc + sst * nx;  // the FP32 position on the 2x grid
        const float y = (float)Gr + sst * ny;
        o.x = ((double)x - 1.0) * 0.5;
        o.y = ((double)y - 1.0) * 0.5;
        o.str = sqrtf((maxf * nx) * (maxf * nx) + (maxf * ny) * (maxf * ny));
    }
    return o;
}

// How much the third-order vector (tix, tiy) cancels, against its bound: true
// when the sum of its terms' magnitudes is over kRefineKappa times its larger
// component.  The FP32 derivatives' rounding reaches the angle multiplied by
// that ratio, so such an edgel's is formed again in FP64.
__device__ __forceinline__ bool cancels(float gx, float gy, const float (&d)[7], float tix, float tiy)
{
    const float fxx = d[0], fxy = d[1], fyy = d[2], fxxy = d[3], fxyy = d[4], fxxx = d[5], fyyy = d[6];
    const float ax = fabsf(gx), ay = fabsf(gy), pxx = fabsf(fxx * fxy), pyy = fabsf(fyy * fxy);
    const float sabs = 2.f * ax * (fxx * fxx + fxy * fxy) + 2.f * ay * (fyy * fyy + fxy * fxy) +
                       2.f * (ax + ay) * (pxx + pyy) + 2.f * ax * ay * (fabsf(fxxy) + fabsf(fxyy)) +
                       ay * ay * (fabsf(fxyy) + fabsf(fyyy)) + ax * ax * (fabsf(fxxx) + fabsf(fxxy));
    return sabs > kRefineKappa * fmaxf(fabsf(tix), fabsf(tiy));
}

// An edgel into its image's list.
__device__ __forceinline__ void write_edgel(const BatchParams& p, const DetImage& im, long long d, double x, double y,
                                            float ori, float str, int idx)
{
    if (p.out_f64) {  // two 16-byte stores: the caller's buffer need only be 16-byte aligned
        double2* o = reinterpret_cast<double2*>(im.out) + 2 * d;
        o[0] = make_double2(x, y);
        o[1] = make_double2((double)ori, (double)str);
    } else {
        reinterpret_cast<float4*>(im.out)[d] = make_float4((float)x, (float)y, ori, str);
    }
    if (im.index) im.index[d] = idx;
}

}  // namespace toed
