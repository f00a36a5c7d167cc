// 2-D fan-beam distance-driven and separable-footprint pair (geom/fbct):
//   fan_proj_kernel<TF>   proj,dd  geom/fbct/fbct_proj.c:153-289, proj,tf :292-464
//   fan_back_kernel<TF>   back,dd  geom/fbct/fbct_back.c:80-222,  back,tf :225-393
// Image float[ny][nx], sinogram float[noviews][nu].  Both kernels reproduce the
// reference's float/double operations and its summation order:
// * A is a per-bin gather: a block per (64 detector bins, view) enumerates the pixels whose
//   footprint can reach its bins row by row (the projected centre is monotone along a row), in
//   the reference's (iy, ix) order.  Six warps evaluate 192 of them at a time; two more, a
//   lane per bin, add the previous 192's contributions to their bins in that order.  Where the
//   rays run along the rows, a row's pixels all fall into a few bins and the additions of a
//   step would follow one another, so each bin gathers its own pixels there, four lanes
//   evaluating (a 256^2 pair at 180 views took 1.1 ms with steps alone, all of it in the views
//   near 90 degrees).
// * A^T is pixel-driven: a block per 32 pixels evaluates 32 views at a time (eight warps, four
//   views each) and one warp adds them in order.
// The footprints are chains of exactly rounded divisions and the sums are serial, so both are
// bound by latency; what helps is to evaluate ahead of the sums, in parallel.  Measured on
// B200, DD pair at 256^2, 360 bins, 180 views: 1.95 -> 0.81 ms (A 0.70, A^T 0.11) against one warp
// per 32 bins and one thread per pixel, doing both in turn.  Those still serve the wide footprints
// (fan_proj_warp_kernel), the few views and the large images (fan_back_pixel_kernel) for which
// they are the faster ones (fan_wide, fan_back_by_pixel).  Results do not depend on the launch.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ctsim_b200.h"
#include "kernels.cuh"

using namespace ctsim;

extern ctsim_status ctsim_set_last_error(ctsim_status s, const char *msg);

namespace {

struct FanGeom {
    int nx, ny, nu, det;
    float dx, dy, sad, sdd, du;
    float wx, wy, wu, sdd_du;
    float margin;  // candidate window margin of the forward projector (bins)
    float reach;   // bins from a pixel's projected centre to its footprint's edge, at most
};

struct FanView {
    float sin_a, cos_a, dx_sin_2, dx_cos_2, dy_sin_2, n_dy_cos_2;
};

__device__ __forceinline__ float fan_u(const FanGeom &g, float num, float den) {
    if (g.det == 1) return fsub(fdiv(fmul(g.sdd_du, num), den), g.wu);
    return (float)__dsub_rn(__dmul_rn((double)g.sdd_du, atan((double)fdiv(num, den))), (double)g.wu);
}

// Amplitude and the sorted DD edges t[0..1] (or SF corners t[0..3]) of pixel (ix, iy):
// fbct_proj.c:199-246 (DD), :342-404 (SF).
template <bool TF>
__device__ __forceinline__ float fan_pixel(const FanGeom &g, const FanView &v, int ix, int iy, float *t) {
    const float xc = fmul(fadd((float)ix, g.wx), g.dx);
    const float yc = fmul(fadd((float)iy, g.wy), g.dy);
    const float tp = fsub(fmul(xc, v.cos_a), fmul(yc, v.sin_a));
    const float ds = fadd(fadd(g.sad, fmul(xc, v.sin_a)), fmul(yc, v.cos_a));
    const float r = __fsqrt_rn(fadd(fmul(tp, tp), fmul(ds, ds)));
    const float cg = fdiv(ds, r), sg = fdiv(tp, r);
    const float cphi = fabsf(fsub(fmul(v.cos_a, cg), fmul(v.sin_a, sg)));
    const float sphi = fabsf(fadd(fmul(v.sin_a, cg), fmul(v.cos_a, sg)));
    const float amp = fdiv(fdiv(g.dx, cphi > sphi ? cphi : sphi), 10.0f);
    if (!TF) {
        if (cphi > sphi) {
            t[0] = fan_u(g, fadd(tp, v.dx_cos_2), fadd(ds, v.dx_sin_2));
            t[1] = fan_u(g, fsub(tp, v.dx_cos_2), fsub(ds, v.dx_sin_2));
        } else {
            t[0] = fan_u(g, fadd(tp, v.dy_sin_2), fadd(ds, v.n_dy_cos_2));
            t[1] = fan_u(g, fsub(tp, v.dy_sin_2), fsub(ds, v.n_dy_cos_2));
        }
        if (t[0] >= t[1]) { const float s = t[1]; t[1] = t[0]; t[0] = s; }
        return amp;
    }
    t[0] = fan_u(g, fadd(fadd(tp, v.dx_cos_2), v.dy_sin_2), fadd(fadd(ds, v.dx_sin_2), v.n_dy_cos_2));
    t[1] = fan_u(g, fadd(fsub(tp, v.dx_cos_2), v.dy_sin_2), fadd(fsub(ds, v.dx_sin_2), v.n_dy_cos_2));
    t[2] = fan_u(g, fsub(fadd(tp, v.dx_cos_2), v.dy_sin_2), fsub(fadd(ds, v.dx_sin_2), v.n_dy_cos_2));
    t[3] = fan_u(g, fsub(fsub(tp, v.dx_cos_2), v.dy_sin_2), fsub(fsub(ds, v.dx_sin_2), v.n_dy_cos_2));
    float s;
    if (t[0] > t[1]) { s = t[0]; t[0] = t[1]; t[1] = s; }
    if (t[2] > t[3]) { s = t[2]; t[2] = t[3]; t[3] = s; }
    if (t[0] > t[2]) { s = t[0]; t[0] = t[2]; t[2] = s; }
    if (t[1] > t[3]) { s = t[1]; t[1] = t[3]; t[3] = s; }
    if (t[1] > t[2]) { s = t[1]; t[1] = t[2]; t[2] = s; }
    return amp;
}

// Trapezoid area of bin iu (fbct_proj.c:430-456).
__device__ __forceinline__ float fan_tf_weight(int iu, const float *t) {
    float w = 0.0f;
    const float bl = (float)((double)iu - 0.5), br = (float)((double)iu + 0.5);
    float xl = bl > t[0] ? bl : t[0], xr = br < t[1] ? br : t[1];
    if (xr > xl) {
        const float a = fsub(xr, t[0]), b = fsub(xl, t[0]);
        w = fadd(w, fdiv(fdiv(fsub(fmul(a, a), fmul(b, b)), fsub(t[1], t[0])), 2.0f));
    }
    xl = bl > t[1] ? bl : t[1]; xr = br < t[2] ? br : t[2];
    if (xr > xl) w = fadd(w, fsub(xr, xl));
    xl = bl > t[2] ? bl : t[2]; xr = br < t[3] ? br : t[3];
    if (xr > xl) {
        const float a = fsub(xl, t[3]), b = fsub(xr, t[3]);
        w = fadd(w, fdiv(fdiv(fsub(fmul(a, a), fmul(b, b)), fsub(t[3], t[2])), 2.0f));
    }
    return w;
}

// umin = max(lo + 0.5, 0), umax = min(hi + 0.5, nu) and the bins.  The reference forms and
// compares the sums in double and stores them as float; a float plus 0.5 rounds to the same
// float directly.
__device__ __forceinline__ bool fan_range(const FanGeom &g, float lo, float hi, float &umin, float &umax, int &ilo,
                                          int &ihi) {
    const float a = fadd(lo, 0.5f), b = fadd(hi, 0.5f);
    umin = a > 0.0f ? a : 0.0f;
    umax = b < (float)g.nu ? b : (float)g.nu;
    if (umin > umax) return false;
    ilo = (int)floorf(umin);
    ihi = min((int)floorf(umax), g.nu - 1);
    return true;
}

constexpr int kFanMaxRows = 4096;
constexpr int kFanBins = 64;                      // bins per block: two warps of one bin per lane
constexpr int kFanChunk = 192;                    // candidates per step: six warps
constexpr int kFanThreads = kFanChunk + kFanBins;
constexpr int kFanVals = 4;                       // bins of a footprint whose contributions are kept
// Bins per pixel step along a row below which a bin gathers its pixels itself: at 256^2, 360
// bins, one view 80 degrees off takes 0.30 ms in steps and 0.44 ms gathered, 84 degrees 0.73 and
// 0.46 ms; all 180 views 0.88, 0.68 and 0.73 ms with the line at 0.1, 0.2 and 0.4; 128^2, 180 bins 0.36, 0.27 and
// 0.29; 512^2, 720 bins 2.79, 1.79 and 2.07, 360 bins 1.71, 1.84 and 2.13; 256^2, 100 bins 0.77, 0.76 and 0.93.
constexpr float kFanGatherBelow = 0.2f;
constexpr int kFanLanes = kFanThreads / kFanBins; // lanes per bin of the gather
static_assert(kFanLanes == 4, "one bin per four lanes");

// The candidates of one step: per bin the set of those that touch it, and their contributions
// to bins b = lo .. hi at val[b mod kFanVals] (in double: the sum of two floats formed in double
// and rounded to float equals their float sum, so one addition serves the reference's float
// and double sums).  wide: a footprint has more than kFanVals bins; the step's contributions
// are then formed again from pix (image index) as they are added.
struct FanStep {
    double val[kFanVals][kFanChunk];
    unsigned touch[kFanChunk / 32][kFanBins];
    int pix[kFanChunk];
    int wide;
};

// What pixel value x with corners t (fan_pixel) adds to bin iu of its bins lo .. hi, and
// whether the reference adds it in double.
template <bool TF>
__device__ __forceinline__ double fan_contribution(int iu, int lo, int hi, float amp, const float *t, float umin,
                                                   float umax, float x) {
    if (TF) return (double)fmul(fan_tf_weight(iu, t), fmul(amp, x));  // voxel = amplitude * image
    if (lo == hi) return (double)fmul(fmul(amp, fsub(umax, umin)), x);
    if (iu == lo)  // amplitude * (iumin + 1.0 - umin) * image, in double
        return __dmul_rn(__dmul_rn((double)amp, __dsub_rn(__dadd_rn((double)lo, 1.0), (double)umin)), (double)x);
    if (iu == hi) return (double)fmul(fmul(amp, fsub(umax, (float)hi)), x);
    return (double)fmul(amp, x);
}

// Bin iu of view v by four consecutive lanes: row by row the pixels whose centre projects to
// within `reach` bins of the bin -- u(x) >= c is linear in x, x (cos - r sin) >= r (sad + y cos)
// + y sin with r the tangent at u = c (an edge 90 degrees off the axis and more bounds nothing)
// -- four at a time, their contributions added in order by all four lanes alike.
template <bool TF>
__device__ __forceinline__ float fan_gather(const FanGeom &g, const FanView &v, const float *__restrict__ image, int iu,
                                            float reach) {
    const int q = threadIdx.x & (kFanLanes - 1);
    // tangent r and slope a at u; both 0 where the edge bounds nothing
    auto edge = [&](float u, float &r, float &a) {
        r = (u + g.wu - 0.5f) / g.sdd_du;
        const bool bounds = g.det == 1 || fabsf(r) < 1.57f;
        if (g.det != 1) r = bounds ? tanf(r) : 0.0f;
        a = bounds ? v.cos_a - r * v.sin_a : 0.0f;
    };
    float r0, a0, r1, a1;
    edge((float)iu - reach, r0, a0);
    edge((float)(iu + 1) + reach, r1, a1);
    // pixels [first, last) of a row that may meet a0 x >= b0 and a1 x <= b1 (one pixel of slack)
    auto range = [&](int iy, int &first, int &last) {
        const float yc = ((float)iy + g.wy) * g.dy;
        const float b0 = r0 * (g.sad + yc * v.cos_a) + yc * v.sin_a, b1 = r1 * (g.sad + yc * v.cos_a) + yc * v.sin_a;
        float lo = 0.0f, hi = (float)(g.nx - 1);
        const float x0 = b0 / (a0 * g.dx) - g.wx, x1 = b1 / (a1 * g.dx) - g.wx;
        // near-zero slopes leave the row in if either end may hold (x0, x1 may be inf or NaN)
        if (a0 > 0.0f) lo = fmaxf(lo, x0 - 1.0f); else if (a0 < 0.0f) hi = fminf(hi, x0 + 1.0f);
        if (a1 > 0.0f) hi = fminf(hi, x1 + 1.0f); else if (a1 < 0.0f) lo = fmaxf(lo, x1 - 1.0f);
        first = (int)floorf(fminf(lo, (float)g.nx));
        last = (int)ceilf(fmaxf(hi, -1.0f)) + 1;
    };
    double acc = 0.0;  // a float's value
    int iy = -1, c = 0, last = 0;
    if (iu >= g.nu) iy = g.ny;
    for (;;) {  // the warp's eight bins stay together
        while (c >= last && iy < g.ny) {
            iy++;
            if (iy < g.ny) range(iy, c, last);
        }
        if (!__any_sync(0xffffffffu, iy < g.ny)) break;
        const int ix = c + q;
        double add = 0.0;
        bool hit = false;
        if (iy < g.ny && ix < min(last, g.nx)) {
            float tt[4], umin, umax;
            int lo, hi;
            const float amp = fan_pixel<TF>(g, v, ix, iy, tt);
            if (fan_range(g, tt[0], TF ? tt[3] : tt[1], umin, umax, lo, hi) && iu >= lo && iu <= hi) {
                hit = true;
                add = fan_contribution<TF>(iu, lo, hi, amp, tt, umin, umax, image[(size_t)iy * g.nx + ix]);
            }
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit) >> (threadIdx.x & 28);
#pragma unroll
        for (int s = 0; s < kFanLanes; s++) {
            const double d = __shfl_sync(0xffffffffu, add, s, kFanLanes);
            if (hits >> s & 1u) acc = (double)(float)__dadd_rn(acc, d);
        }
        c += kFanLanes;
    }
    return (float)acc;
}

template <bool TF>
__global__ void __launch_bounds__(kFanThreads) fan_proj_kernel(FanGeom g, const FanView *__restrict__ views,
                                                               const float *__restrict__ image,
                                                               float *__restrict__ proj, int view_begin,
                                                               int view_stride) {
    extern __shared__ double fsm[];
    FanStep *step = reinterpret_cast<FanStep *>(fsm);  // two
    int *row_first = reinterpret_cast<int *>(step + 2);  // [ny]
    int *row_off = row_first + g.ny;                     // [ny + 1]
    const int t = threadIdx.x, lane = t & 31;
    const int iu0 = blockIdx.x * kFanBins;
    const int k = blockIdx.y;
    const FanView v = views[view_begin + k * view_stride];
    // bins that a pixel step along a row moves the centre by, at the axis: where it is small the
    // additions of a step crowd into few bins
    if (fabsf(v.cos_a) * g.dx * g.sdd_du < kFanGatherBelow * g.sad) {
        const int iu = iu0 + t / kFanLanes;
        const float sum = fan_gather<TF>(g, v, image, iu, g.reach);
        if (iu < g.nu && (t & (kFanLanes - 1)) == 0) proj[(size_t)k * g.nu + iu] = sum;
        return;
    }
    const float ulo = (float)iu0 - g.margin, uhi = (float)(iu0 + kFanBins) + g.margin;
    // approximate projected centre (candidate search only; footprints are exact below)
    auto centre = [&](int ix, int iy) {
        const float xc = ((float)ix + g.wx) * g.dx, yc = ((float)iy + g.wy) * g.dy;
        const float r = (xc * v.cos_a - yc * v.sin_a) / (g.sad + xc * v.sin_a + yc * v.cos_a);
        return (g.det == 1 ? g.sdd_du * r : g.sdd_du * atanf(r)) - g.wu + 0.5f;
    };
    for (int iy = t; iy < g.ny; iy += kFanThreads) {
        const bool inc = centre(g.nx - 1, iy) >= centre(0, iy);
        int lo = 0, hi = g.nx;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float f = centre(mid, iy);
            if (inc ? (f < ulo) : (f > uhi)) lo = mid + 1; else hi = mid;
        }
        const int first = lo;
        hi = g.nx;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float f = centre(mid, iy);
            if (inc ? (f > uhi) : (f < ulo)) hi = mid; else lo = mid + 1;
        }
        row_first[iy] = first;
        row_off[iy] = lo - first;
    }
    for (int i = t; i < 2 * kFanBins * (kFanChunk / 32); i += kFanThreads) {
        const int b = i / (kFanBins * (kFanChunk / 32)), o = i % (kFanBins * (kFanChunk / 32));
        (&step[b].touch[0][0])[o] = 0u;
        if (o == 0) step[b].wide = 0;
    }
    __syncthreads();
    if (t < 32) {  // exclusive scan of the per-row counts (lane owns a contiguous run of rows)
        const int per = (g.ny + 31) / 32;
        const int b = min(lane * per, g.ny), e = min(b + per, g.ny);
        int sum = 0;
        for (int iy = b; iy < e; iy++) sum += row_off[iy];
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        __syncwarp();
        int run = incl - sum;
        for (int iy = b; iy < e; iy++) {
            const int c = row_off[iy];
            row_off[iy] = run;
            run += c;
        }
        if (lane == 31) row_off[g.ny] = incl;
    }
    __syncthreads();
    const int ncand = row_off[g.ny];
    const int nsteps = (ncand + kFanChunk - 1) / kFanChunk;
    const int bin = t - kFanChunk;  // of an adding thread
    auto evaluate = [&](int pix, float *tt, float &amp, float &umin, float &umax, int &lo, int &hi) {
        const int iy = pix / g.nx;
        amp = fan_pixel<TF>(g, v, pix - iy * g.nx, iy, tt);
        return fan_range(g, tt[0], TF ? tt[3] : tt[1], umin, umax, lo, hi);
    };
    double acc = 0.0;  // a float's value
    for (int i = 0; i <= nsteps; i++) {
        if (t < kFanChunk) {
            const int c = i * kFanChunk + t;
            if (i < nsteps && c < ncand) {
                FanStep &S = step[i & 1];
                int a = 0, z = g.ny - 1;  // last row with row_off <= c
                while (a < z) {
                    const int mid = (a + z + 1) >> 1;
                    if (row_off[mid] <= c) a = mid; else z = mid - 1;
                }
                const int pix = a * g.nx + row_first[a] + (c - row_off[a]);
                const float x = image[pix];
                float tt[4], amp, umin, umax;
                int lo, hi;
                if (evaluate(pix, tt, amp, umin, umax, lo, hi)) {
                    S.pix[t] = pix;
                    if (hi - lo >= kFanVals) S.wide = 1;
                    for (int b = max(lo, iu0); b <= min(hi, iu0 + kFanBins - 1); b++) {
                        S.val[b % kFanVals][t] = fan_contribution<TF>(b, lo, hi, amp, tt, umin, umax, x);
                        atomicOr(&S.touch[t >> 5][b - iu0], 1u << lane);
                    }
                }
            }
        } else if (i > 0) {
            FanStep &S = step[(i - 1) & 1];
            const int iu = iu0 + bin;
            const double *val = S.val[iu % kFanVals];
            const bool wide = S.wide != 0;
            int wd = 0;
            unsigned m = S.touch[0][bin];
            for (;;) {
                while (m == 0u && ++wd < kFanChunk / 32) m = S.touch[wd][bin];
                if (m == 0u) break;
                const int c = wd * 32 + __ffs(m) - 1;
                m &= m - 1;
                double add = val[c];
                if (wide) {
                    float tt[4], amp, umin, umax;
                    int lo, hi;
                    evaluate(S.pix[c], tt, amp, umin, umax, lo, hi);
                    add = fan_contribution<TF>(iu, lo, hi, amp, tt, umin, umax, image[S.pix[c]]);
                }
                acc = (double)(float)__dadd_rn(acc, add);
            }
#pragma unroll
            for (int q = 0; q < kFanChunk / 32; q++) S.touch[q][bin] = 0u;
            // every adding thread has read `wide` before the evaluating ones may set it again
            asm volatile("bar.sync 1, %0;" ::"n"(kFanBins) : "memory");
            if (bin == 0) S.wide = 0;
        }
        __syncthreads();
    }
    if (bin >= 0 && iu0 + bin < g.nu) proj[(size_t)k * g.nu + iu0 + bin] = (float)acc;
}

// Footprints of three bins and more: one warp per (32 bins, view), a candidate per lane, then
// each candidate's bins in turn.  Many lanes add at once there, and nothing is evaluated twice.
// Shared memory: per row the first candidate column and the running candidate count, then one
// candidate record per lane.
template <bool TF>
__global__ void __launch_bounds__(32) fan_proj_warp_kernel(FanGeom g, const FanView *__restrict__ views,
                                                      const float *__restrict__ image, float *__restrict__ proj,
                                                      int view_begin, int view_stride) {
    extern __shared__ int fsw[];
    int *row_first = fsw;                      // [ny]
    int *row_off = fsw + g.ny;                 // [ny + 1]
    float *c_t = reinterpret_cast<float *>(row_off + g.ny + 1);  // [4][32]
    float *c_amp = c_t + 4 * 32;               // [32]: DD amplitude, SF amplitude * pixel
    float *c_x = c_amp + 32;                   // [32]: DD pixel value
    int *c_lo = reinterpret_cast<int *>(c_x + 32);
    int *c_hi = c_lo + 32;
    const int lane = threadIdx.x;
    const int iu0 = blockIdx.x * 32;
    const int k = blockIdx.y;
    const FanView v = views[view_begin + k * view_stride];
    const float ulo = (float)iu0 - g.margin, uhi = (float)(iu0 + 32) + g.margin;
    // approximate projected centre (candidate search only; footprints are exact below)
    auto centre = [&](int ix, int iy) {
        const float xc = ((float)ix + g.wx) * g.dx, yc = ((float)iy + g.wy) * g.dy;
        const float r = (xc * v.cos_a - yc * v.sin_a) / (g.sad + xc * v.sin_a + yc * v.cos_a);
        return (g.det == 1 ? g.sdd_du * r : g.sdd_du * atanf(r)) - g.wu + 0.5f;
    };
    for (int iy = lane; iy < g.ny; iy += 32) {
        const bool inc = centre(g.nx - 1, iy) >= centre(0, iy);
        int lo = 0, hi = g.nx;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float f = centre(mid, iy);
            if (inc ? (f < ulo) : (f > uhi)) lo = mid + 1; else hi = mid;
        }
        const int first = lo;
        hi = g.nx;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float f = centre(mid, iy);
            if (inc ? (f > uhi) : (f < ulo)) hi = mid; else lo = mid + 1;
        }
        row_first[iy] = first;
        row_off[iy] = lo - first;
    }
    __syncwarp();
    {   // exclusive scan of the per-row counts (lane owns a contiguous run of rows)
        const int per = (g.ny + 31) / 32;
        const int b = min(lane * per, g.ny), e = min(b + per, g.ny);
        int sum = 0;
        for (int iy = b; iy < e; iy++) sum += row_off[iy];
        int incl = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        __syncwarp();
        int run = incl - sum;
        for (int iy = b; iy < e; iy++) {
            const int c = row_off[iy];
            row_off[iy] = run;
            run += c;
        }
        if (lane == 31) row_off[g.ny] = incl;
    }
    __syncwarp();
    const int ncand = row_off[g.ny];
    const int iu = iu0 + lane;
    float acc = 0.0f;
    for (int c0 = 0; c0 < ncand; c0 += 32) {
        const int c = c0 + lane;
        int lo = 0, hi = -1;
        if (c < ncand) {
            int a = 0, z = g.ny - 1;  // last row with row_off <= c
            while (a < z) {
                const int mid = (a + z + 1) >> 1;
                if (row_off[mid] <= c) a = mid; else z = mid - 1;
            }
            const int iy = a, ix = row_first[a] + (c - row_off[a]);
            float t[4];
            const float amp = fan_pixel<TF>(g, v, ix, iy, t);
            float umin, umax;
            if (fan_range(g, t[0], TF ? t[3] : t[1], umin, umax, lo, hi)) {
                const float x = image[(size_t)iy * g.nx + ix];
                if (TF) {
                    for (int q = 0; q < 4; q++) c_t[q * 32 + lane] = t[q];
                    c_amp[lane] = fmul(amp, x);  // voxel = amplitude * image
                } else {
                    c_t[lane] = umin;
                    c_t[32 + lane] = umax;
                    c_amp[lane] = amp;
                    c_x[lane] = x;
                }
            } else {
                lo = 0;
                hi = -1;
            }
        }
        c_lo[lane] = lo;
        c_hi[lane] = hi;
        __syncwarp();
        const int ns = min(32, ncand - c0);
        for (int s = 0; s < ns; s++) {
            const int slo = c_lo[s], shi = c_hi[s];
            if (iu < slo || iu > shi) continue;
            if (TF) {
                float t[4] = {c_t[s], c_t[32 + s], c_t[64 + s], c_t[96 + s]};
                acc = fadd(acc, fmul(fan_tf_weight(iu, t), c_amp[s]));
            } else {
                const float umin = c_t[s], umax = c_t[32 + s], amp = c_amp[s], x = c_x[s];
                if (slo == shi) {
                    acc = fadd(acc, fmul(fmul(amp, fsub(umax, umin)), x));
                } else if (iu == slo) {  // amplitude * (iumin + 1.0 - umin) * image, in double
                    const double w = __dsub_rn(__dadd_rn((double)slo, 1.0), (double)umin);
                    acc = (float)__dadd_rn((double)acc, __dmul_rn(__dmul_rn((double)amp, w), (double)x));
                } else if (iu == shi) {
                    acc = fadd(acc, fmul(fmul(amp, fsub(umax, (float)shi)), x));
                } else {
                    acc = fadd(acc, fmul(amp, x));
                }
            }
        }
        __syncwarp();
    }
    if (iu < g.nu) proj[(size_t)k * g.nu + iu] = acc;
}

// One pixel in one view: what the view adds to the pixel (0 where it has no bin).
template <bool TF>
__device__ __forceinline__ float fan_back_view(const FanGeom &g, const FanView &v, const float *__restrict__ p, int ix,
                                               int iy) {
    float t[4];
    const float amp = fan_pixel<TF>(g, v, ix, iy, t);
    float temp = 0.0f;
    if (!TF) {
        float umin, umax;
        int lo, hi;
        if (!fan_range(g, t[0], t[1], umin, umax, lo, hi)) return 0.0f;
        if (lo == hi) {
            temp = fmul(fsub(umax, umin), __ldg(p + lo));
        } else {
            for (int iu = lo; iu <= hi; iu++) {
                const float pv = __ldg(p + iu);
                if (iu == lo) {
                    const double w = __dsub_rn(__dadd_rn((double)lo, 1.0), (double)umin);
                    temp = (float)__dadd_rn((double)temp, __dmul_rn(w, (double)pv));
                } else if (iu == hi) {
                    temp = fadd(temp, fmul(fsub(umax, (float)hi), pv));
                } else {
                    temp = fadd(temp, pv);
                }
            }
        }
        return fmul(amp, temp);
    }
    // iumin = max(floorf(t0 + 0.5), 0), iumax = min(ceilf(t3 + 0.5), nu - 1), fbct_back.c:345-346
    const int lo = max((int)floorf(fadd(t[0], 0.5f)), 0);
    const int hi = min((int)ceilf(fadd(t[3], 0.5f)), g.nu - 1);
    for (int iu = lo; iu <= hi; iu++) temp = fadd(temp, fmul(fmul(amp, fan_tf_weight(iu, t)), __ldg(p + iu)));
    return temp;
}

// The views in order (fbct_back.c:114-218 DD, :253-388 SF): warp w of a block evaluates views
// 4 w .. 4 w + 3 of each 32 for the block's 32 pixels, warp 0 adds the 32 of the step before.
template <bool TF>
__global__ void __launch_bounds__(256) fan_back_kernel(FanGeom g, const FanView *__restrict__ views,
                                                       const float *__restrict__ proj, float *__restrict__ image,
                                                       int view_begin, int view_stride, int view_count, float scale) {
    __shared__ float val[2][32][32];  // [step parity][view][pixel]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ix = blockIdx.x * 32 + lane;
    const int iy = blockIdx.y;
    const int nsteps = (view_count + 31) / 32;
    float img = 0.0f;
    for (int i = 0; i <= nsteps; i++) {
        if (i < nsteps && ix < g.nx)
            for (int q = 0; q < 4; q++) {
                const int s = 4 * warp + q, k = 32 * i + s;
                if (k < view_count)
                    val[i & 1][s][lane] =
                        fan_back_view<TF>(g, views[view_begin + k * view_stride], proj + (size_t)k * g.nu, ix, iy);
            }
        if (i > 0 && warp == 0) {
            const int n = min(32, view_count - 32 * (i - 1));
            for (int s = 0; s < n; s++) img = fadd(img, val[(i - 1) & 1][s][lane]);
        }
        __syncthreads();
    }
    if (warp == 0 && ix < g.nx) {
        if (scale != 1.0f) img = img * scale;
        image[(size_t)iy * g.nx + ix] = img;
    }
}

// One thread per pixel, the views in order.
template <bool TF>
__global__ void __launch_bounds__(128) fan_back_pixel_kernel(FanGeom g, const FanView *__restrict__ views,
                                                             const float *__restrict__ proj, float *__restrict__ image,
                                                             int view_begin, int view_stride, int view_count,
                                                             float scale) {
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y;
    if (ix >= g.nx) return;
    float img = 0.0f;
    for (int k = 0; k < view_count; k++)
        img = fadd(img, fan_back_view<TF>(g, views[view_begin + k * view_stride], proj + (size_t)k * g.nu, ix, iy));
    if (scale != 1.0f) img = img * scale;
    image[(size_t)iy * g.nx + ix] = img;
}

}  // namespace

struct ctsim_fan_plan {
    ctsim_fan_geom geom;
    FanGeom g;
    int device = 0;
    FanView *d_views = nullptr;
};

static size_t fan_proj_smem(int ny) { return 2 * sizeof(FanStep) + (size_t)(2 * ny + 1) * 4; }
static size_t fan_proj_warp_smem(int ny) { return (size_t)(2 * ny + 1) * 4 + 32 * 6 * 4 + 32 * 2 * 4; }

// Whether A takes a warp per 32 bins: footprints so wide (in bins, nearest the source; SF's at 45
// degrees) that some touch more bins than a step keeps contributions of and would be evaluated
// again for each.  DD, pixels of 2.5, 2.7 and 3 bins (3.1, 3.4 and 3.8 at the nearest), 90 views, steps
// over warps: 64^2 0.58, 1.75, 2.06, 256^2 0.57, 2.00, 3.39, 512^2 0.68, 1.49, 2.34; SF, pixels of 2, 2.04
// and 2.5 bins (3.6, 3.7 and 4.5): 64^2 0.35, 0.37, 1.21, 256^2 0.35, 0.37, 0.67, 512^2 0.42, 0.38, 0.80, on
// curved detectors 0.49, 0.54, 1.79; 0.35, 0.38, 0.97; 0.44, 0.41, 1.12.
constexpr float kFanWideDD = 3.25f, kFanWideTF = 3.75f;
static bool fan_wide(const ctsim_fan_plan *p, int method) {
    const ctsim_fan_geom &G = p->geom;
    if (method != CTSIM_PROJ_DD) return 2.0f * p->g.reach >= kFanWideTF;
    return 2.0f * p->g.reach * std::max(G.dx, G.dy) / std::hypot(G.dx, G.dy) >= kFanWideDD;
}

// Whether A^T takes a thread per pixel: where the image alone fills the GPU, or the views leave
// most of a block's warps without one.  Block kernel over pixel kernel, DD, flat: 1, 8, 16, 32 and
// 64 views at 64^2 0.86, 0.75, 0.46, 0.27, 0.21; 256^2 1.45, 1.29, 0.95, 0.69, 0.62; 512^2 2.59, 1.83,
// 1.25, 0.94, 0.91; 1024^2 4.51, 2.12, 1.31, 1.02, 0.99; 2000^2 5.79, 2.20, 1.34, 1.04, 1.01.
static bool fan_back_by_pixel(const ctsim_fan_geom &G, int view_count) {
    const long long pixels = (long long)G.nx * G.ny;
    return view_count < 8 || pixels >= (view_count < 16 ? 1 << 15 : view_count < 32 ? 1 << 18 : 1 << 20);
}

// A kernel with its dynamic shared memory; the launch's error.
template <class K, class... Args>
static cudaError_t fan_launch(K kernel, dim3 grid, int threads, size_t smem, void *stream, Args... args) {
    cudaError_t e = allow_dynamic_smem((const void *)kernel, smem);
    if (e != cudaSuccess) return e;
    kernel<<<grid, threads, smem, (cudaStream_t)stream>>>(args...);
    return cudaGetLastError();
}

extern "C" ctsim_status ctsim_fan_plan_create(const ctsim_fan_geom *geom, const double *betas, ctsim_fan_plan **out) {
    if (!geom || !betas || !out) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    *out = nullptr;
    const ctsim_fan_geom G = *geom;
    if (G.nx < 1 || G.ny < 1 || G.nu < 1 || G.noviews < 1)
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "sizes must be positive");
    if (!(G.dx > 0 && G.dy > 0 && G.du > 0 && G.sad > 0 && G.sdd > 0))
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "spacings and distances must be positive");
    if (G.detector_type != 0 && G.detector_type != 1)
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "detector_type must be 1 (flat) or 0 (curved)");
    if (G.ny > kFanMaxRows) return ctsim_set_last_error(CTSIM_ERR_UNSUPPORTED, "fan-beam images support ny <= 4096");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return ctsim_set_last_error(CTSIM_ERR_NO_DEVICE, cudaGetErrorString(e));
    ctsim_fan_plan *p = new ctsim_fan_plan();
    p->geom = G;
    p->device = dev;
    FanGeom &g = p->g;
    g.nx = G.nx; g.ny = G.ny; g.nu = G.nu; g.det = G.detector_type;
    g.dx = G.dx; g.dy = G.dy; g.sad = G.sad; g.sdd = G.sdd; g.du = G.du;
    g.wx = (float)(-((double)G.nx - 1.0) / 2.0 + (double)G.offset_x);
    g.wy = (float)(-((double)G.ny - 1.0) / 2.0 + (double)G.offset_y);
    g.wu = (float)(-((double)G.nu - 1.0) / 2.0 + (double)G.offset_u);
    g.sdd_du = G.sdd / G.du;
    // margin: half the pixel diagonal magnified at the nearest pixel, stretched at the
    // detector's edge for a flat panel, plus slack for the approximate centre
    double rmax = 0.0;
    for (int cx = 0; cx < 2; cx++)
        for (int cy = 0; cy < 2; cy++) {
            const double xc = ((cx ? G.nx - 1 : 0) + (double)g.wx) * G.dx, yc = ((cy ? G.ny - 1 : 0) + (double)g.wy) * G.dy;
            rmax = std::max(rmax, std::sqrt(xc * xc + yc * yc));
        }
    const double diag = std::sqrt((double)G.dx * G.dx + (double)G.dy * G.dy);
    const double dmin = (double)G.sad - rmax - diag;
    if (!(dmin > 0.0)) {
        delete p;
        return ctsim_set_last_error(CTSIM_ERR_UNSUPPORTED, "the source orbit must lie outside the image (SAD > radius)");
    }
    const double umm = std::max(std::fabs((double)g.wu * G.du), std::fabs(((double)G.nu - 1 + g.wu) * G.du)) + G.du;
    const double stretch = G.detector_type == 1 ? 1.0 + (umm / G.sdd) * (umm / G.sdd) : 1.0;
    g.margin = (float)std::ceil(0.5 * diag * G.sdd / dmin / G.du * stretch) + 2.0f;
    g.reach = (float)(0.5 * diag * G.sdd / dmin / G.du * stretch * 1.0001 + 0.05);
    std::vector<FanView> views(G.noviews);
    for (int ib = 0; ib < G.noviews; ib++) {
        FanView &v = views[ib];
        v.sin_a = (float)std::sin(betas[ib]);
        v.cos_a = (float)std::cos(betas[ib]);
        v.dx_sin_2 = (float)((double)(G.dx * v.sin_a) / 2.0);
        v.dx_cos_2 = (float)((double)(G.dx * v.cos_a) / 2.0);
        v.dy_sin_2 = (float)((double)(G.dy * v.sin_a) / 2.0);
        v.n_dy_cos_2 = (float)((double)(-G.dy * v.cos_a) / 2.0);
    }
    if ((e = cudaMalloc(&p->d_views, sizeof(FanView) * G.noviews)) != cudaSuccess ||
        (e = cudaMemcpy(p->d_views, views.data(), sizeof(FanView) * G.noviews, cudaMemcpyHostToDevice)) != cudaSuccess) {
        cudaFree(p->d_views);
        delete p;
        return ctsim_set_last_error(CTSIM_ERR_ALLOC, cudaGetErrorString(e));
    }
    *out = p;
    return CTSIM_OK;
}

extern "C" ctsim_status ctsim_fan_plan_destroy(ctsim_fan_plan *p) {
    if (p) {
        cudaFree(p->d_views);
        delete p;
    }
    return CTSIM_OK;
}

static ctsim_status fan_views_ok(const ctsim_fan_plan *p, int vb, int vs, int vc) {
    if (vc < 1 || vs < 1 || vb < 0 || (long long)vb + (long long)(vc - 1) * vs >= p->geom.noviews)
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "view selection outside the plan's views");
    return CTSIM_OK;
}

extern "C" ctsim_status ctsim_fan_project(ctsim_fan_plan *p, int method, const float *d_image, float *d_sino,
                                          int view_begin, int view_stride, int view_count, void *stream) {
    if (!p || !d_image || !d_sino) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    if (method != CTSIM_PROJ_DD && method != CTSIM_PROJ_TF)
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "unknown forward method");
    ctsim_status s = fan_views_ok(p, view_begin, view_stride, view_count);
    if (s != CTSIM_OK) return s;
    const bool dd = method == CTSIM_PROJ_DD;
    cudaError_t e;
    if (fan_wide(p, method))
        e = fan_launch(dd ? fan_proj_warp_kernel<false> : fan_proj_warp_kernel<true>, dim3((p->g.nu + 31) / 32, view_count),
                       32, fan_proj_warp_smem(p->g.ny), stream, p->g, p->d_views, d_image, d_sino, view_begin,
                       view_stride);
    else
        e = fan_launch(dd ? fan_proj_kernel<false> : fan_proj_kernel<true>,
                       dim3((p->g.nu + kFanBins - 1) / kFanBins, view_count), kFanThreads, fan_proj_smem(p->g.ny), stream,
                       p->g, p->d_views, d_image, d_sino, view_begin, view_stride);
    return e == cudaSuccess ? CTSIM_OK : ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
}

extern "C" ctsim_status ctsim_fan_backproject(ctsim_fan_plan *p, int method, const float *d_sino, float *d_image,
                                              int view_begin, int view_stride, int view_count, float scale,
                                              void *stream) {
    if (!p || !d_image || !d_sino) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    if (method != CTSIM_BACK_DD && method != CTSIM_BACK_TF)
        return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "unknown fan-beam backprojection method");
    ctsim_status s = fan_views_ok(p, view_begin, view_stride, view_count);
    if (s != CTSIM_OK) return s;
    const bool dd = method == CTSIM_BACK_DD;
    const bool pixel = fan_back_by_pixel(p->geom, view_count);
    const dim3 grid((p->g.nx + (pixel ? 127 : 31)) / (pixel ? 128 : 32), p->g.ny);
    const auto kernel = pixel ? (dd ? fan_back_pixel_kernel<false> : fan_back_pixel_kernel<true>)
                              : (dd ? fan_back_kernel<false> : fan_back_kernel<true>);
    kernel<<<grid, pixel ? 128 : 256, 0, (cudaStream_t)stream>>>(p->g, p->d_views, d_sino, d_image, view_begin, view_stride,
                                                                 view_count, scale);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CTSIM_OK : ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
}

// Host-pointer entry with the reference's fan-beam MEX dispatch (geom/fbct/fbct_geom_mex.c:243-278):
// proj,dd / proj,tf / back,dd / back,tf; synchronous, never exits.
extern "C" bool ctsim_fbct_geom(const char *type, int nx, int ny, float dx, float dy, float offset_x, float offset_y,
                                int nu, float du, float offset_u, float sad, float add, float sdd, int noviews,
                                const double *betas, int detector_type, const float *data, float *out) {
    if (!type || !betas || !data || !out) {
        ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
        return false;
    }
    int method;
    if (!std::strcmp(type, "proj,dd")) method = CTSIM_PROJ_DD;
    else if (!std::strcmp(type, "proj,tf")) method = CTSIM_PROJ_TF;
    else if (!std::strcmp(type, "back,dd")) method = CTSIM_BACK_DD;
    else if (!std::strcmp(type, "back,tf")) method = CTSIM_BACK_TF;
    else {
        ctsim_set_last_error(CTSIM_ERR_UNSUPPORTED, "unknown or unsupported fan-beam geom type");
        return false;
    }
    const ctsim_fan_geom G = {nx, ny, dx, dy, offset_x, offset_y, nu, du, offset_u, sad, add, sdd, noviews,
                              detector_type};
    ctsim_fan_plan *p = nullptr;
    if (ctsim_fan_plan_create(&G, betas, &p) != CTSIM_OK) return false;
    const bool fwd = method == CTSIM_PROJ_DD || method == CTSIM_PROJ_TF;
    const size_t nimg = (size_t)nx * ny, nsino = (size_t)nu * noviews;
    const size_t nin = fwd ? nimg : nsino, nout = fwd ? nsino : nimg;
    float *din = nullptr, *dout = nullptr;
    bool ok = false;
    cudaError_t e;
    if ((e = cudaMalloc(&din, nin * 4)) == cudaSuccess && (e = cudaMalloc(&dout, nout * 4)) == cudaSuccess &&
        (e = cudaMemcpy(din, data, nin * 4, cudaMemcpyHostToDevice)) == cudaSuccess) {
        const ctsim_status s = fwd ? ctsim_fan_project(p, method, din, dout, 0, 1, noviews, nullptr)
                                   : ctsim_fan_backproject(p, method, din, dout, 0, 1, noviews, 1.0f, nullptr);
        if (s == CTSIM_OK) {
            if ((e = cudaDeviceSynchronize()) == cudaSuccess && (e = cudaMemcpy(out, dout, nout * 4, cudaMemcpyDeviceToHost)) == cudaSuccess)
                ok = true;
            else
                ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
        }
    } else {
        ctsim_set_last_error(CTSIM_ERR_ALLOC, cudaGetErrorString(e));
    }
    cudaFree(din);
    cudaFree(dout);
    ctsim_fan_plan_destroy(p);
    return ok;
}
