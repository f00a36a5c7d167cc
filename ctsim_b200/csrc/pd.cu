// Voxel-driven bilinear backprojection for sm_100a: FDK back,pd / back,hpd
// (geom/cbct/cbct_back.c:7-133) and the variance backprojection back,var
// (geom/cbct/cbct_back_var.c).
//
// Layouts (reference MEX conventions): image[iz][iy][ix], proj[view][iu][iv].
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "packed.cuh"

namespace ctsim {

// One sinogram sample of storage type DT (kF32, kBF16, kF16) at a byte address, as float
// (exact widening).
template <int DT>
__device__ __forceinline__ float ld_sino(uintptr_t a) {
    if (DT == kBF16) return __uint_as_float((unsigned)__ldg(reinterpret_cast<const unsigned short *>(a)) << 16);
    if (DT == kF16) return __half2float(__ushort_as_half(__ldg(reinterpret_cast<const unsigned short *>(a))));
    return __ldg(reinterpret_cast<const float *>(a));
}

// Correctly rounded a / d (div_by of common.cuh) on one or two values.
template <class V>
__device__ __forceinline__ V pdiv_by(V a, float d, float r) {
    using P = Packed<V>;
    if (r == 0.0f) return P::make([&](int i) { return __fdiv_rn(P::get(a, i), d); });
    const V q = pmul(a, P::all(r));
    const V e = pfma(q, P::all(-d), a);
    return pfma(e, P::all(r), q);
}

// A warp per voxel column, lanes along z, 8 columns (consecutive ix) per block; lane l
// accumulates the voxels iz0 + l + 32 m, m < MZ, over the views in the reference's order
// with its exact float operations (the result equals the reference's bit for bit on flat
// panels).  Per view, the quantities that a column's voxels share -- the detector column,
// the u weights, w2 and w2s -- are computed by the lane that the view falls to in a 32-view
// chunk and read from a per-warp table.
//
// What bounds it: instruction issue, then the FP32 pipe (23 scalar FP32 operations per
// voxel and view) and the latency of the four loads.  So two voxels share every FP32
// instruction (V = f32x2), and a pass takes up to eight 32-voxel blocks (MZ), which spreads
// a view's table loads, unpacking and branches over them and puts their loads in flight
// together.
//
// sum: the FP32 image holds the view sum of earlier view chunks (scale 1), which the
// kernel continues in the same view order.  DT: the sinogram's storage type, read as it
// is (widening to FP32 is exact, so the result equals that of an FP32 copy bit for bit).
// The image is written as (sum * scale) * scale2.  one: 1.0f (padd_product).
struct PdArgs {
    const View *views;
    const void *proj;
    void *image;
    int out_dtype, view_begin, view_stride, view_count;
    float scale, scale2, one;
    bool sum;
};

// One pass: NP registers of W voxels per lane from slice iz0 (the last ones may lie past
// the volume: they sample clamped rows and are not stored).  vtab: the warp's view table.
template <int MODE, int NP, class V, int DT>
__device__ __forceinline__ void pd_pass(const Geom &g, const PdArgs &A, float4 (*vtab)[2], int ix, int iy, int iz0,
                                        bool on) {
    using P = Packed<V>;
    constexpr int W = P::kWidth;
    constexpr bool OFF = MODE != kPdClamp, VAR = MODE == kPdVar;
    constexpr unsigned kSize = DT == kF32 ? 4 : 2;
    const int lane = threadIdx.x & 31;
    const size_t nxy = (size_t)g.nx * g.ny;
    const size_t nuv = (size_t)g.nu * g.nv;
    const size_t out0 = (size_t)(iz0 + lane) * nxy + (size_t)iy * g.nx + ix;
    const int izn = g.nz - iz0;
    const float xc = fmul(fadd((float)ix, g.wx), g.dx);
    const float yc = fmul(fadd((float)iy, g.wy), g.dy);
    const V two23 = P::all(kTwo23), one = P::all(A.one), wv = P::all(g.wv), dz = P::all(g.dz);
    const float v_lo = OFF ? 0.0f : 0.5f, v_hi = OFF ? g.v_hi : g.v_clamp_hi;
    const unsigned col_bytes = (unsigned)g.nv * kSize;
    V acc[NP], zc0[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        acc[p] = P::all(0.0f);
        // (iz + wz) * dz (cbct_back.c:100); back,var: iz, its wz is the view's
        const V iz = P::make([&](int i) { return (float)(iz0 + lane + 32 * (W * p + i)); });
        zc0[p] = VAR ? iz : pmul(padd(iz, P::all(g.wz_pd)), dz);
        if (A.sum)
            acc[p] = P::make([&](int i) {
                const int dzi = 32 * (W * p + i);
                return lane + dzi < izn ? static_cast<const float *>(A.image)[out0 + (size_t)dzi * nxy] : 0.0f;
            });
    }
    if (on) {
        for (int k0 = 0; k0 < A.view_count; k0 += 32) {
            const int kl = k0 + lane;
            // {wul, 1 - wul, w2, w2s}, {couch, 0, address of the detector column (low, high word)};
            // address 0: u is off the detector
            float4 ta = make_float4(0.f, 0.f, 0.f, 0.f), tb = make_float4(0.f, 0.f, 0.f, 0.f);
            if (kl < A.view_count) {
                const View v = A.views[A.view_begin + kl * A.view_stride];
                const float xr = fsub(fmul(xc, v.cos_a), fmul(yc, v.sin_a));
                const float yr = fadd(fmul(xc, v.sin_a), fmul(yc, v.cos_a));
                const float den = fadd(g.sad, yr);
                float u, w2, w2s;
                if (g.det == 1) {  // cbct_back.c:68-77
                    w2 = fdiv(g.sdd, den);
                    w2s = fmul(w2, w2);
                    u = fsub(fdiv(fmul(xr, w2), g.du), g.wu);
                } else {           // cbct_back.c:78-88, cbct_back_var.c:68-77
                    const float xo = fsub(xr, VAR ? g.roff_var : g.roff);
                    const double at = atan((double)fdiv(xo, den));
                    u = (float)__dsub_rn(__ddiv_rn(__dmul_rn(at, (double)g.sdd), (double)g.du), (double)g.wu);
                    w2s = fdiv(fmul(g.sdd, g.sdd), fadd(fmul(den, den), fmul(xo, xo)));
                    w2 = fdiv(g.sdd, den);
                }
                if (u >= g.u_lo && u <= g.u_hi) {  // cbct_back.c:90
                    float fiu;
                    const int iu = floor_pos(u, &fiu);
                    const float wul = fsub(u, fiu);
                    // w2s * (...) (cbct_back.c:120); w2s * w2s * (...) (cbct_back_var.c:116)
                    ta = make_float4(wul, fsub(1.0f, wul), w2, VAR ? fmul(w2s, w2s) : w2s);
                    const uintptr_t a = reinterpret_cast<uintptr_t>(A.proj) +
                                        ((size_t)kl * nuv + (size_t)iu * g.nv) * kSize;
                    tb = make_float4(VAR ? v.wz : v.couch_pd, 0.f, __uint_as_float((unsigned)a),
                                     __uint_as_float((unsigned)(a >> 32)));
                }
            }
            __syncwarp();  // the previous chunk's reads are done
            vtab[lane][0] = ta;
            vtab[lane][1] = tb;
            __syncwarp();
            const int nk = min(32, A.view_count - k0);
            for (int j = 0; j < nk; j++) {
                const float4 b = vtab[j][1];
                uintptr_t col0 = ((uintptr_t)__float_as_uint(b.w) << 32) | __float_as_uint(b.z);
                if (col0 == 0) continue;  // u off the detector
                const float4 a = vtab[j][0];
                // row iv of the column is at col0 + kSize * bits(iv + 2^23) from here on
                col0 -= (uintptr_t)0x4B000000u * kSize;
                const uintptr_t col1 = col0 + col_bytes;
                const V wul = P::all(a.x), omu = P::all(a.y), w2 = P::all(a.z), w2s = P::all(a.w), cj = P::all(b.x);
#pragma unroll
                for (int p = 0; p < NP; p++) {
                    // (iz + wz) * dz + couch (cbct_back.c:100), with the view's wz in cbct_back_var.c:41, :89
                    const V zc = VAR ? pmul(padd(zc0[p], cj), dz) : padd_product(zc0[p], one, cj);
                    const V vv = psub(pdiv_by<V>(pmul(zc, w2), g.dv, g.rdv), wv);  // cbct_back.c:102
                    // hpd: v clamped (cbct_back.c:110-111); pd, var: rows off the detector add nothing
                    // (cbct_back.c:105-108) and sample a clamped row here.  floor(v) <= nv - 2 both ways.
                    const V vc = P::make([&](int i) { return fminf(fmaxf(P::get(vv, i), v_lo), v_hi); });
                    const V t = padd_rd(vc, two23);
                    const V wvl = psub(vc, psub(t, two23));
                    const V omv = psub(P::all(1.0f), wvl);
                    float s[4][W];
#pragma unroll
                    for (int i = 0; i < W; i++) {
                        const uintptr_t o = (uintptr_t)__float_as_uint(P::get(t, i)) * kSize;
                        s[0][i] = ld_sino<DT>(col0 + o);
                        s[1][i] = ld_sino<DT>(col0 + o + kSize);
                        s[2][i] = ld_sino<DT>(col1 + o);
                        s[3][i] = ld_sino<DT>(col1 + o + kSize);
                    }
                    auto at = [&](int k) { return P::make([&](int i) { return s[k][i]; }); };
                    const V s0 = padd_product(pmul(omv, at(0)), one, pmul(wvl, at(1)));
                    const V s1 = padd_product(pmul(omv, at(2)), one, pmul(wvl, at(3)));
                    const V val = padd_product(pmul(omu, s0), one, pmul(wul, s1));
                    const V sum = padd_product(pmul(w2s, val), one, acc[p]);
                    if (OFF)
                        acc[p] = P::make([&](int i) {
                            const float x = P::get(vv, i);
                            return x >= g.v_lo && x <= g.v_hi ? P::get(sum, i) : P::get(acc[p], i);
                        });
                    else
                        acc[p] = sum;
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < NP; p++)
#pragma unroll
        for (int i = 0; i < W; i++) {
            const int dzi = 32 * (W * p + i);
            if (lane + dzi < izn) {
                float r = on ? P::get(acc[p], i) : 0.0f;
                if (A.scale != 1.0f) r = r * A.scale;
                if (A.scale2 != 1.0f) r = r * A.scale2;
                store_from_float(A.image, out0 + (size_t)dzi * nxy, r, A.out_dtype);
            }
        }
}

// A full pass of MZ 32-voxel blocks, or the shortest one that covers the remaining slices.
template <int MODE, int NP, class V, int DT>
__device__ __forceinline__ void pd_pass_of(int np, const Geom &g, const PdArgs &A, float4 (*vtab)[2], int ix, int iy,
                                           int iz0, bool on) {
    if constexpr (NP > 1)
        if (np < NP) {
            pd_pass_of<MODE, NP - 1, V, DT>(np, g, A, vtab, ix, iy, iz0, on);
            return;
        }
    pd_pass<MODE, NP, V, DT>(g, A, vtab, ix, iy, iz0, on);
}

// Blocks per SM: four of the packed kernels (registers capped at 64); six of the scalar one, whose
// loads only other warps hide (back,hpd of 512^2 x 32, 720 views of 72 rows: 13.5 ms with five, 10.9
// with six; pd, 40 rows 11.6 and 10.8 ms).  The geometry stays in the parameters (a copy's size
// decides how the kernel compiles: back,hpd of 128^2 x 64, 360 views 0.54 -> 0.60 ms).
template <int MODE, int MZ, class V, int DT>
__global__ void __launch_bounds__(256, MZ == 1 ? 6 : 4) pd_kernel(const __grid_constant__ Geom g, PdArgs A, const uint8_t *__restrict__ map) {
    constexpr int W = Packed<V>::kWidth, NP = MZ / W;
    const int warp = threadIdx.x >> 5;
    const int tiles_x = (g.nx + 7) >> 3;
    const int iy = blockIdx.x / tiles_x;
    const int ix = (blockIdx.x % tiles_x) * 8 + warp;
    if (ix >= g.nx || iy >= g.ny) return;
    __shared__ float4 vtab[8][32][2];
    const bool on = map[iy * g.nx + ix] != 0;
    for (int iz0 = 0; iz0 < g.nz; iz0 += 32 * MZ) {
        const int np = min(NP, (g.nz - iz0 + 32 * W - 1) / (32 * W));
        pd_pass_of<MODE, NP, V, DT>(np, g, A, vtab[warp], ix, iy, iz0, on);
    }
}

// Sinogram bytes of a view chunk.  back,hpd in chunks of 64, 160 and 320 MB and in one launch: 300^2
// x 160, 900 views of 720 x 260 20.0, 21.6, 23.0, 23.3 ms; 384^2 x 320, 1200 of 560 x 500 82.6, 78.7, 84.2,
// 87.3; 256^3, 2000 of 400 x 300 40.6, 42.1, 45.9, 47.7; 512^2 x 64, 1440 of 1024 x 110 31.9, 32.8, 36.0,
// 36.0; 512^2 x 256, 720 of 1024 x 384 66.9, 66.1, 71.0, 88.2 (L2 flushed before each).
constexpr size_t kPdChunkBytes = (size_t)160 << 20;

template <int MODE, int MZ>
static cudaError_t launch_pd_mz(const Geom &g, const View *views, const void *proj, int in_dtype, const uint8_t *map,
                                void *image, int out_dtype, int vb, int vs, int vc, float scale, float scale2,
                                bool accumulate, cudaStream_t st) {
    using V = std::conditional_t<MZ == 1, float, f32x2>;
    const int blocks = g.ny * ((g.nx + 7) / 8);
    auto k = in_dtype == kBF16  ? pd_kernel<MODE, MZ, V, kBF16>
             : in_dtype == kF16 ? pd_kernel<MODE, MZ, V, kF16>
                                : pd_kernel<MODE, MZ, V, kF32>;
    // Blocks of a long launch drift apart over the views until the detector columns they read
    // no longer meet in L2 (a 512^2 x 256 volume: 7.1 ms for 90 views, 70.4 ms for 720).  So an
    // FP32 image takes a sinogram of more than two chunks chunk by chunk, continuing its sums:
    // for 720 views of 1.6 MB, 70.4 ms in one launch, 67.1, 60.7, 58.7, 58.2 and 62.3 ms in
    // chunks of 32, 64, 96, 128 and 192 views (a chunk costs the volume's read and write).
    const size_t view_bytes = (size_t)g.nu * g.nv * (in_dtype == kF32 ? 4 : 2);
    const int chunk = std::max(32, (int)(kPdChunkBytes / view_bytes / 32 * 32));
    const bool split = out_dtype == kF32 && vc > 2 * chunk;
    for (int c = 0; c < vc;) {
        const int n = split ? std::min(chunk, vc - c) : vc;
        const bool last = c + n == vc;
        const PdArgs A{views, static_cast<const char *>(proj) + (size_t)c * view_bytes, image, out_dtype, vb + c * vs,
                       vs, n, last ? scale : 1.0f, last ? scale2 : 1.0f, 1.0f, accumulate || c > 0};
        k<<<blocks, 256, 0, st>>>(g, A, map);
        c += n;
    }
    return cudaGetLastError();
}

cudaError_t launch_pd(int mode, int mz, const Geom &g, const View *views, const void *proj, const uint8_t *map,
                      void *image, int out_dtype, int vb, int vs, int vc, float scale, cudaStream_t st,
                      bool accumulate, int in_dtype, float scale2) {
    if (accumulate && (out_dtype != kF32 || scale != 1.0f || in_dtype != kF32)) return cudaErrorInvalidValue;
    if (in_dtype != kF32 && in_dtype != kBF16 && in_dtype != kF16) return cudaErrorInvalidValue;
#define CTSIM_PD_CASE(O, Z)                                                                                   \
    if (mode == O && mz == Z)                                                                                 \
        return launch_pd_mz<O, Z>(g, views, proj, in_dtype, map, image, out_dtype, vb, vs, vc, scale, scale2, \
                                  accumulate, st);
    CTSIM_PD_CASE(kPdOff, 1) CTSIM_PD_CASE(kPdOff, 2) CTSIM_PD_CASE(kPdOff, 4) CTSIM_PD_CASE(kPdOff, 8)
    CTSIM_PD_CASE(kPdClamp, 1) CTSIM_PD_CASE(kPdClamp, 2) CTSIM_PD_CASE(kPdClamp, 4) CTSIM_PD_CASE(kPdClamp, 8)
    CTSIM_PD_CASE(kPdVar, 1) CTSIM_PD_CASE(kPdVar, 2) CTSIM_PD_CASE(kPdVar, 4) CTSIM_PD_CASE(kPdVar, 8)
#undef CTSIM_PD_CASE
    return cudaErrorInvalidValue;
}

}  // namespace ctsim
