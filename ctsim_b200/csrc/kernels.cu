// Projector kernels for sm_100a.
//
//   back_kernel<METHOD,MZ>   matched backprojection A^T (distance-driven / separable footprint)
//   prefix_kernel            per-column axial prefix sums of the volume (input of A)
//   proj_kernel<METHOD>      forward projection A
//
// The voxel-driven FDK backprojection is in pd.cu.
//
// Layouts (reference MEX conventions): image[iz][iy][ix], proj[view][iu][iv].
#include "kernels.cuh"

#include <map>
#include <mutex>
#include <utility>

namespace ctsim {

constexpr unsigned kFull = 0xffffffffu;

// Rows r0 .. r0+3 of one detector column of a sinogram source (element offset off of row
// r0), times ampv at the same element for the unscaled sources.  VEC: nv a multiple of 4
// and the source aligned (one 16-byte FP32 or 8-byte 16-bit load); otherwise rows at or
// past nv read as 0.
template <int SRC, bool VEC>
__device__ __forceinline__ float4 load_rows4(const void *__restrict__ src, const float *__restrict__ ampv, size_t off,
                                             size_t aoff, int r0, int nv) {
    float4 p;
    if (SRC == kSrcScaled || SRC == kSrcF32) {
        const float *pr = static_cast<const float *>(src) + off;
        if (VEC) {
            p = __ldg(reinterpret_cast<const float4 *>(pr));
        } else {
            p.x = __ldg(pr);
            p.y = r0 + 1 < nv ? __ldg(pr + 1) : 0.f;
            p.z = r0 + 2 < nv ? __ldg(pr + 2) : 0.f;
            p.w = r0 + 3 < nv ? __ldg(pr + 3) : 0.f;
        }
    } else {
        const unsigned short *pr = static_cast<const unsigned short *>(src) + off;
        unsigned short h[4];
        if (VEC) {
            const uint2 u = __ldg(reinterpret_cast<const uint2 *>(pr));
            h[0] = (unsigned short)(u.x & 0xffffu); h[1] = (unsigned short)(u.x >> 16);
            h[2] = (unsigned short)(u.y & 0xffffu); h[3] = (unsigned short)(u.y >> 16);
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) h[i] = r0 + i < nv ? __ldg(pr + i) : (unsigned short)0;
        }
        float f[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            f[i] = SRC == kSrcBF16 ? __uint_as_float((unsigned)h[i] << 16) : __half2float(__ushort_as_half(h[i]));
        p = make_float4(f[0], f[1], f[2], f[3]);
    }
    if (SRC != kSrcScaled) {  // axial amplitude applied here instead of in a scratch copy
        const float *ar = ampv + aoff;
        float4 a;
        if (VEC) {
            a = __ldg(reinterpret_cast<const float4 *>(ar));
        } else {
            a.x = __ldg(ar);
            a.y = r0 + 1 < nv ? __ldg(ar + 1) : 0.f;
            a.z = r0 + 2 < nv ? __ldg(ar + 2) : 0.f;
            a.w = r0 + 3 < nv ? __ldg(ar + 3) : 0.f;
        }
        p.x *= a.x; p.y *= a.y; p.z *= a.z; p.w *= a.w;
    }
    return p;
}

// ---------------------------------------------------------------------------
// A^T: one warp per voxel column, lanes along z; 8 columns (consecutive ix) per block.
// For each view the warp forms, in shared memory, the u-weighted detector column
//     q[iv] = sum_iu w_u(iu) * ps[iu][iv]        (ps = proj * ampv)
// over the rows the column's voxels can touch (4 rows per lane, float4 loads).  Each
// voxel then sums q over the rows its axial extent covers with the distance-driven
// row weights of geom/cbct/cbct_back.c:318-357, its edges vmin/vmax computed with the
// reference's float operations (usually two or three rows per voxel).  The edges sit
// hundreds of rows up the detector, where one float rounding moves a voxel's weight by
// ~1e-5 of itself; evaluating them exactly as the reference does keeps each voxel's
// value within a few float roundings of the reference's instead of adding noise of
// that size.  Accumulation over views stays in registers; no atomics.
// ---------------------------------------------------------------------------
// The work of one block (8 columns of one row iy), as a device function: the plain
// kernel runs it for blockIdx.x, the batched kernel for each of its work items.
// 32-bit shared load ordered after the warp's earlier shared stores (compiler barrier).
__device__ __forceinline__ float lds_ordered(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <int METHOD, int MZ, bool VEC, int SRC, bool SUM = false>
__device__ __forceinline__ void back_block(const Geom g, const View *__restrict__ views, const void *__restrict__ ps,
                                           const uint8_t *__restrict__ map, void *__restrict__ image, int out_dtype,
                                           int view_begin, int view_stride, int view_count, float scale, int qcap,
                                           int *__restrict__ err, const float *__restrict__ ampv, float *smem,
                                           int block) {
    constexpr int kWS = 17;  // row stride of the per-warp weight table (conflict-free writes)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *wtab = smem + warp * (32 * kWS + 32 * 8 + qcap);  // [32 views][17] u weights of the view chunk
    // [32 views] per-view scalars of the chunk, written by the view's own lane:
    // {ampu, zinc, vstart, iumin | nb << 16}, {rbase | r_hi << 16, path + 1 (0: no rows), -, -}
    float4 *vtab = reinterpret_cast<float4 *>(wtab + 32 * kWS);  // 16-byte aligned: 32 * 17 * 4 = 2176
    float *Q = wtab + 32 * kWS + 32 * 8;                         // [qcap] q per row
    const int tiles_x = (g.nx + 7) >> 3;
    const int iy = block / tiles_x;
    const int ix = (block % tiles_x) * 8 + warp;
    if (ix >= g.nx || iy >= g.ny) return;
    const size_t nxy = (size_t)g.nx * g.ny;
    const size_t nuv = (size_t)g.nu * g.nv;
    const bool on = map[iy * g.nx + ix] != 0;
    const float fnv = (float)g.nv;
    const int nvm1 = g.nv - 1;
    const int zpass = 32 * MZ;
    for (int iz0 = 0; iz0 < g.nz; iz0 += zpass) {
        const int izn = min(zpass, g.nz - iz0);
        const float fz_first = (float)iz0, fz_last = (float)(iz0 + izn - 1);
        float acc[MZ];
#pragma unroll
        for (int m = 0; m < MZ; m++) acc[m] = 0.0f;
        const float fz_lane = (float)(iz0 + lane);
        if (SUM) {
            // continue the per-voxel view sum (scale 1) that the previous view chunk left in
            // the FP32 image; the sum runs in view order either way
            const float *src = static_cast<const float *>(image) + (size_t)(iz0 + lane) * nxy + (size_t)iy * g.nx + ix;
#pragma unroll
            for (int m = 0; m < MZ; m++)
                if (lane + 32 * m < izn) acc[m] = src[(size_t)(32 * m) * nxy];
        }
        if (on) {
            for (int k0 = 0; k0 < view_count; k0 += 32) {
                ColumnFP my;
                my.hit = false;
                const int kl = k0 + lane;
                if (kl < view_count) my = column_footprint<METHOD>(g, views[view_begin + kl * view_stride], ix, iy);
                // lane-parallel u weights of this lane's view (geom/cbct/cbct_back.c:288-301, :549-578)
                // A voxel's vmax - vmin is zinc within 1.5 float ulps of nv (< 2^-10 for nv <=
                // 8192), so away from zinc = 1 and 2 by a margin every voxel of the view covers
                // the same number of rows give or take one: n = k_hi - k_lo is 0 or 1 (zinc < 1)
                // or 1 or 2 (1 < zinc < 2).  Those views run branch-free (paths 1 and 2 below).
                constexpr float kMargin = 1.0f / 256.0f;
                __syncwarp();  // the previous chunk's reads of wtab and vtab are done
                {
                    int path1 = 0, rows = 0;
                    if (my.hit) {
                        const int nb = my.iumax - my.iumin + 1;
                        for (int b = 0; b < nb; b++)
                            wtab[lane * kWS + b] =
                                u_weight<METHOD>(my.iumin + b, my.iumin, my.iumax, my.p0, my.p1, my.p2, my.p3);
                        // rows reachable by voxels [iz0, iz0+izn) (the reference's clamped
                        // extents, monotone in iz)
                        const float zinc = my.zinc, vstart = my.vstart;
                        const float a0u = fadd(fadd(vstart, fmul(fz_first, zinc)), 0.5f);
                        const float b1u = fadd(fadd(fadd(vstart, fmul(fz_last, zinc)), zinc), 0.5f);
                        const float a0 = fmaxf(a0u, 0.0f), b1 = fminf(b1u, fnv);
                        if (a0 < fnv && b1 >= 0.0f) {
                            const int r_lo = floor_pos(a0);
                            int r_hi = min(floor_pos(b1), nvm1);
                            if (r_lo <= r_hi) {
                                const int rbase = r_lo & ~3;
                                // every voxel of the pass exists and lies inside the detector
                                bool inside = a0u > 0.0f && b1u < fnv && izn == zpass;
                                if (r_hi - rbase + 1 > qcap) {  // rows rbase..r_hi must fit
                                    atomicOr(err, 1);
                                    r_hi = rbase + qcap - 1;
                                    inside = false;
                                }
                                path1 = 1 + (!inside ? 0 : zinc < 1.0f - kMargin ? 1
                                                     : (zinc > 1.0f + kMargin && zinc < 2.0f - kMargin) ? 2 : 0);
                                rows = rbase | (r_hi << 16);
                            }
                        }
                        vtab[2 * lane] = make_float4(my.ampu, zinc, vstart, __int_as_float(my.iumin | (nb << 16)));
                    }
                    vtab[2 * lane + 1] = make_float4(__int_as_float(rows), __int_as_float(path1), 0.f, 0.f);
                }
                __syncwarp();
                const int nk = min(32, view_count - k0);
                for (int j = 0; j < nk; j++) {
                    const float4 pb = vtab[2 * j + 1];
                    const int path1 = __float_as_int(pb.y);
                    if (path1 == 0) continue;  // no footprint or no rows
                    const float4 pa = vtab[2 * j];
                    const float ampu = pa.x, zinc = pa.y, vstart = pa.z;
                    const int iumin = __float_as_int(pa.w) & 0xffff, nb = __float_as_int(pa.w) >> 16;
                    const int rbase = __float_as_int(pb.x) & 0xffff, r_hi = __float_as_int(pb.x) >> 16;
                    // q over rows [rbase, r_hi], 128 rows per pass (the voxels read rows
                    // [r_lo, r_hi] only)
                    const float *wj = wtab + j * kWS;
                    const size_t pv = (size_t)(k0 + j) * nuv + (size_t)iumin * g.nv;  // element offsets
                    const size_t av = (size_t)iumin * g.nv;
                    for (int c = rbase; c <= r_hi; c += 128) {
                        const int r0 = c + 4 * lane;
                        float q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
                        if (r0 <= r_hi) {
                            for (int b = 0; b < nb; b++) {
                                const float w = wj[b];
                                const float4 p = load_rows4<SRC, VEC>(ps, ampv, pv + (size_t)b * g.nv + r0,
                                                                      av + (size_t)b * g.nv + r0, r0, g.nv);
                                q0 = fmaf(w, p.x, q0); q1 = fmaf(w, p.y, q1);
                                q2 = fmaf(w, p.z, q2); q3 = fmaf(w, p.w, q3);
                            }
                        }
                        *reinterpret_cast<float4 *>(Q + (r0 - rbase)) = make_float4(q0, q1, q2, q3);
                    }
                    __syncwarp();
                    // Each voxel: the reference's clamped extent and row weights
                    // (geom/cbct/cbct_back.c:318-357); rows [k_lo, k_hi] lie in [r_lo, r_hi]
                    // because the edges are monotone in iz.
                    const float *qb = Q - rbase;
                    // shared address of row k is qadj + 4 * bits(k + 2^23) (mod 2^32)
                    const uint32_t qadj = (uint32_t)__cvta_generic_to_shared(Q) - 4u * (uint32_t)rbase -
                                          (0x4B000000u << 2);
                    // Paths 1 and 2 always read the rows k_lo .. k_lo + 1 (+ 2) (the row buffer has 4
                    // spare floats; rows past r_hi may hold anything, so their terms are selected,
                    // never multiplied by zero).
                    const int path = path1 - 1;
                    if (path == 1) {
#pragma unroll
                        for (int m = 0; m < MZ; m++) {
                            const float izv = fz_lane + (float)(32 * m);  // exact
                            const float vpre = fadd(vstart, fmul(izv, zinc));
                            const float vmin = fadd(vpre, 0.5f);
                            const float vmax = fadd(fadd(vpre, zinc), 0.5f);
                            const float tlo = __fadd_rd(vmin, kTwo23), thi = __fadd_rd(vmax, kTwo23);
                            const uint32_t qa = qadj + (__float_as_uint(tlo) << 2);
                            const float q0 = lds_ordered(qa), q1 = lds_ordered(qa + 4u);
                            // one row: (vmax - vmin) q0; two: (k_lo + 1 - vmin) q0 + (vmax - k_hi) q1,
                            // where k_hi = k_lo + 1 (kf, exact)
                            const float one = fsub(vmax, vmin) * q0;
                            const float kf = fsub(tlo, kTwo23 - 1.0f);
                            const float two = fmaf(fsub(vmax, kf), q1, fsub(kf, vmin) * q0);
                            acc[m] = fmaf(ampu, thi == tlo ? one : two, acc[m]);
                        }
                    } else if (path == 2) {
#pragma unroll
                        for (int m = 0; m < MZ; m++) {
                            const float izv = fz_lane + (float)(32 * m);
                            const float vpre = fadd(vstart, fmul(izv, zinc));
                            const float vmin = fadd(vpre, 0.5f);
                            const float vmax = fadd(fadd(vpre, zinc), 0.5f);
                            const float tlo = __fadd_rd(vmin, kTwo23), thi = __fadd_rd(vmax, kTwo23);
                            const uint32_t qa = qadj + (__float_as_uint(tlo) << 2);
                            const float q0 = lds_ordered(qa), q1 = lds_ordered(qa + 4u), q2 = lds_ordered(qa + 8u);
                            const bool three = fsub(thi, tlo) == 2.0f;
                            const float wl = fsub(vmax, fsub(thi, kTwo23));
                            // two rows: w0 q0 + wl q1; three: w0 q0 + q1 + wl q2 (the reference's row order)
                            float vox = fmaf(three ? 1.0f : wl, q1, fsub(fsub(tlo, kTwo23 - 1.0f), vmin) * q0);
                            vox = three ? fmaf(wl, q2, vox) : vox;
                            acc[m] = fmaf(ampu, vox, acc[m]);
                        }
                    } else {
#pragma unroll
                        for (int m = 0; m < MZ; m++) {
                            const float izv = fz_lane + (float)(32 * m);  // exact
                            const float vpre = fadd(vstart, fmul(izv, zinc));                // vstart + iz * zinc
                            const float vmin = fmaxf(fadd(vpre, 0.5f), 0.0f);                 // max(vmin + 0.5, 0)
                            const float vmax = fminf(fadd(fadd(vpre, zinc), 0.5f), fnv);      // min(vmax + 0.5, nv)
                            if (izv <= fz_last && vmin <= vmax) {
                                float flo, fhi;
                                const int klo = floor_pos(vmin, &flo);
                                int khi = floor_pos(vmax, &fhi);
                                if (khi > nvm1) { khi = nvm1; fhi = fsub(fnv, 1.0f); }
                                if (khi > klo + (kMaxRowsV - 1)) {
                                    khi = klo + (kMaxRowsV - 1);
                                    fhi = fadd(flo, (float)(kMaxRowsV - 1));
                                }
                                khi = min(khi, r_hi);  // only after a row-buffer overflow (flagged above)
                                float vox = 0.0f;
                                if (klo == khi) {
                                    vox = fsub(vmax, vmin) * qb[klo];
                                } else if (klo < khi) {
                                    vox = fsub(fadd(flo, 1.0f), vmin) * qb[klo];
                                    for (int k = klo + 1; k < khi; k++) vox += qb[k];
                                    vox = fmaf(fsub(vmax, fhi), qb[khi], vox);
                                }
                                acc[m] = fmaf(ampu, vox, acc[m]);
                            }
                        }
                    }
                    __syncwarp();
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int m = 0; m < MZ; m++) {
            const int dz = lane + 32 * m;
            if (dz < izn)
                store_from_float(image, (size_t)(iz0 + dz) * nxy + (size_t)iy * g.nx + ix, on ? acc[m] * scale : 0.0f,
                                 out_dtype);
        }
    }
}

// ps = proj * ampv (the axial amplitude the reference applies to the backprojected
// view in place, geom/cbct/cbct_back.c:196-214), into scratch.
// Four resident blocks per SM (registers capped at 64): measured on B200 at config 2,
// DD 110 -> 100 ms and SF 143 -> 104 ms against the uncapped 80-118 registers.
template <int METHOD, int MZ, bool VEC, int SRC = kSrcScaled, bool SUM = false>
__global__ void __launch_bounds__(256, 4) back_kernel(Geom g, const View *__restrict__ views,
                                                   const void *__restrict__ ps, const uint8_t *__restrict__ map,
                                                   void *__restrict__ image, int out_dtype, int view_begin,
                                                   int view_stride, int view_count, float scale, int qcap,
                                                   int *__restrict__ err, const float *__restrict__ ampv,
                                                   int block_base) {
    extern __shared__ float smem[];
    back_block<METHOD, MZ, VEC, SRC, SUM>(g, views, ps, map, image, out_dtype, view_begin, view_stride,
                                                view_count, scale, qcap, err, ampv, smem, block_base + blockIdx.x);
}

__global__ void prescale_kernel(const void *__restrict__ proj, int in_dtype, const float *__restrict__ ampv,
                                float *__restrict__ ps, size_t nuv, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        ps[i] = load_as_float(proj, i, in_dtype) * (ampv ? ampv[i % nuv] : 1.0f);
}

// ---------------------------------------------------------------------------
// Axial prefix sums of every voxel column (input of the forward projector),
// X[k] = sum_{j<k} image[j][col], k = 0..nz, col = iy*nx + ix, in one of two layouts:
// * PAIRS: xc[col][k] = (X[k], X[k+1] - X[k]) as float2, with the top pair (X[nz], 0), so
//   X(s) = X[k] + (s - k) * slope is one aligned 8-byte load and one FMA for 0 <= s <= nz;
// * single: xc[col][k] = X[k] as float (half the bytes: better when the volume's prefix
//   does not stay cache-resident; measured on B200 at 512^2 x 256), columns xstride =
//   prefix_stride(nz) floats apart, with X[nz] repeated above X[nz] up to the stride.
// 32 columns per block; a 32x32 tile is transposed through shared memory so that the
// image reads and the prefix writes are coalesced.
// ---------------------------------------------------------------------------
template <bool PAIRS>
__global__ void __launch_bounds__(256) prefix_kernel(const void *__restrict__ image, int in_dtype,
                                                     float *__restrict__ xs, int nxy, int nz, int xstride) {
    __shared__ float tile[32][33];
    __shared__ float carry[32];
    const int c0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const size_t stride = PAIRS ? (size_t)nz + 1 : (size_t)xstride;
    if (threadIdx.x < 32) carry[threadIdx.x] = 0.0f;
    for (int z0 = 0; z0 < nz; z0 += 32) {
        __syncthreads();
        for (int zz = ty; zz < 32; zz += 8) {
            const int z = z0 + zz, c = c0 + tx;
            tile[zz][tx] = (z < nz && c < nxy) ? load_as_float(image, (size_t)z * nxy + c, in_dtype) : 0.0f;
        }
        __syncthreads();
        // warp ty scans columns ty, ty+8, ty+16, ty+24 along z (lane = z)
        for (int cc = ty; cc < 32; cc += 8) {
            float v = tile[tx][cc];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float n = __shfl_up_sync(kFull, v, o);
                if (tx >= o) v += n;
            }
            const float base = carry[cc];
            const float xtop = base + v;                        // X[z + 1]
            const float xprev = __shfl_up_sync(kFull, xtop, 1);  // X[z] from the lane below
            const float xbot = tx == 0 ? base : xprev;
            const int c = c0 + cc, z = z0 + tx;
            if (c < nxy && z < nz) {
                if (PAIRS) reinterpret_cast<float2 *>(xs)[(size_t)c * stride + z] = make_float2(xbot, xtop - xbot);
                else xs[(size_t)c * stride + z + 1] = xtop;
            }
            const float tot = __shfl_sync(kFull, v, 31);
            __syncwarp();
            if (tx == 0) carry[cc] = base + tot;
        }
    }
    __syncthreads();
    if (threadIdx.x < 32 && c0 + threadIdx.x < nxy) {
        const size_t c = c0 + threadIdx.x;
        if (PAIRS) {
            reinterpret_cast<float2 *>(xs)[c * stride + nz] = make_float2(carry[threadIdx.x], 0.0f);
        } else {
            xs[c * stride] = 0.0f;
            for (size_t k = nz + 1; k < stride; k++) xs[c * stride + k] = carry[threadIdx.x];
        }
    }
}

constexpr int kTU = kProjGroupWidth;
constexpr int kProjMaxThreads = 256;
constexpr int kMaxLines = 2048;

// X(s): integral of a voxel column from its bottom edge to axial position s (in
// voxels, already clamped to [0, nz]) from the column's prefix (x: its first entry).
template <bool PAIRS>
__device__ __forceinline__ float column_integral(const float *__restrict__ x, float s, int nzm1, float fnzm1) {
    float fl;
    int k = floor_pos(s, &fl);
    if (PAIRS) {
        const float2 p = __ldg(reinterpret_cast<const float2 *>(x) + k);
        return fmaf(s - fl, p.y, p.x);
    }
    if (k > nzm1) { k = nzm1; fl = fnzm1; }
    const float a = __ldg(x + k), b = __ldg(x + k + 1);
    return fmaf(s - fl, b - a, a);
}

// Dynamic shared-memory layout of proj_kernel.
// groups: candidate-parallel thread groups, each with its own accumulator copy.
struct ProjSmem {
    int nq, nt, nlines, groups;
    __host__ __device__ size_t acc_bytes() const { return (size_t)groups * kTU * nq * 16; }
    __host__ __device__ size_t bytes() const {
        return acc_bytes() + (size_t)nt * (6 + kTU) * 4 + (size_t)(2 * nlines + 1 + 32) * 4;
    }
};

// A: one block per (group of kTU detector columns, view).  Candidate voxel columns
// are enumerated line by line (lines across the ray direction; the projected column
// centre is monotone along a line, so a line's candidates form one interval found by
// binary search).  Each candidate's footprint is evaluated exactly.  Thread t owns
// detector rows 4t..4t+3 and adds, for every candidate hitting its group,
//     w_u(iu) * ampu * zinc * (X(iv+1) - X(iv))
// -- the integral form of the distance-driven axial weights
// (geom/cbct/cbct_proj.c:382-420) -- into float4 shared-memory accumulators that only
// it touches: no atomics, deterministic.  A block of NT threads holds NT / R groups
// of R row threads (R a multiple of 32, passed by the launcher): group g takes candidates
// g, g + groups, ... into its own accumulators, summed in group order at the store,
// so short detectors (few rows) still keep 8 warps busy per block.
template <int METHOD, int GROUPS, bool PAIRS>
__device__ __forceinline__ void proj_block(const Geom g, const View *__restrict__ views, const float *__restrict__ xs,
                                           const float *__restrict__ ampv, const uint8_t *__restrict__ map,
                                           void *__restrict__ proj, int out_dtype, int view_begin, int view_stride,
                                           float margin, float4 *acc4, int bx, int by) {
    // acc4: [GROUPS][kTU][nq] row quads, then the arrays below (dynamic shared memory)
    const int NT = blockDim.x;
    constexpr int groups = GROUPS;
    const int R = NT / GROUPS;
    const int nq0 = (g.nv + 3) >> 2;
    const int nlines0 = max(g.nx, g.ny);
    int *s_col = reinterpret_cast<int *>(acc4 + groups * kTU * nq0);
    float *s_b0 = reinterpret_cast<float *>(s_col + NT);
    float *s_iz = s_b0 + NT;
    int *s_rlo = reinterpret_cast<int *>(s_iz + NT);
    int *s_rhi = s_rlo + NT;
    int *s_j = s_rhi + NT;
    float *s_wf = reinterpret_cast<float *>(s_j + NT);  // [NT][kTU]
    int *line_start = reinterpret_cast<int *>(s_wf + NT * kTU);
    int *line_off = line_start + nlines0;
    int *s_warp_tot = line_off + nlines0 + 1;

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int grp = GROUPS == 1 ? 0 : t / R;  // candidate group
    const int gwarp = GROUPS == 1 ? warp : (t - grp * R) >> 5;  // warp within the group
    const int iu0 = bx * kTU;
    const int k = by;
    const View v = views[view_begin + k * view_stride];
    const int nv = g.nv;
    const int nq = (nv + 3) >> 2;
    for (int i = t; i < groups * kTU * nq; i += NT) acc4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 *gacc = acc4 + grp * kTU * nq;

    // lines of constant iy when the rays run mostly along y, else lines of constant ix
    const bool rows = fabsf(v.cos_a) >= fabsf(v.sin_a);
    const int nlines = rows ? g.ny : g.nx;
    const int npos = rows ? g.nx : g.ny;
    const float ulo = (float)iu0 - margin, uhi = (float)(iu0 + kTU) + margin;

    auto centre_u = [&](int ix, int iy) -> float {
        const float xcf = ((float)ix + g.wx) * g.dx;
        const float ycf = ((float)iy + g.wy) * g.dy;
        const float tp = xcf * v.cos_a - ycf * v.sin_a;
        const float ds = g.sad + xcf * v.sin_a + ycf * v.cos_a;
        const float r = __fdividef(tp, ds);
        float u;
        if (g.det == 1) {
            u = g.sdd_du * r;
        } else if (g.det == 0) {
            u = g.sdd_du * atanf(r);
        } else {  // arc (candidate search only; the footprints are exact)
            const float gam = atanf(r);
            u = (gam + asinf(g.sad_add * sinf(gam))) * g.add / g.du;
        }
        return u - g.wu + 0.5f;
    };

    // 1. candidate interval of every line (binary search on the monotone centre projection)
    for (int L = t; L < nlines; L += NT) {
        auto f = [&](int p) { return rows ? centre_u(p, L) : centre_u(L, p); };
        const bool inc = f(npos - 1) >= f(0);
        int lo = 0, hi = npos;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float fm = f(mid);
            if (inc ? (fm < ulo) : (fm > uhi)) lo = mid + 1; else hi = mid;
        }
        const int first = lo;
        hi = npos;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const float fm = f(mid);
            if (inc ? (fm > uhi) : (fm < ulo)) hi = mid; else lo = mid + 1;
        }
        line_start[L] = first;
        line_off[L] = lo - first;  // count, turned into offsets below
    }
    __syncthreads();
    // 2. exclusive scan of the counts
    {
        const int per = (nlines + NT - 1) / NT;
        const int b = t * per, e = min(b + per, nlines);
        int sum = 0;
        for (int L = b; L < e; L++) sum += line_off[L];
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int n = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += n;
        }
        if (lane == 31) s_warp_tot[warp] = incl;
        __syncthreads();
        int wbase = 0;
        for (int w = 0; w < warp; w++) wbase += s_warp_tot[w];
        int run = wbase + incl - sum;
        __syncthreads();
        for (int L = b; L < e; L++) {
            const int c = line_off[L];
            line_off[L] = run;
            run += c;
        }
        if (t == NT - 1) line_off[nlines] = run;
    }
    __syncthreads();
    const int ncand = line_off[nlines];
    const float fnz = (float)g.nz;
    const int nzm1 = g.nz - 1;
    const float fnzm1 = (float)nzm1;
    const int rows_per_pass = 4 * R;

    for (int c0 = 0; c0 < ncand; c0 += NT) {
        // 3. exact footprints of this chunk of candidates
        {
            const int c = c0 + t;
            bool valid = false;
            if (c < ncand) {
                int a = 0, bnd = nlines - 1;  // last line with line_off <= c
                while (a < bnd) {
                    const int mid = (a + bnd + 1) >> 1;
                    if (line_off[mid] <= c) a = mid; else bnd = mid - 1;
                }
                const int pos = line_start[a] + (c - line_off[a]);
                const int ix = rows ? pos : a, iy = rows ? a : pos;
                const int col = iy * g.nx + ix;
                if (map[col]) {
                    const ColumnFP fp = column_footprint<METHOD>(g, v, ix, iy);
                    if (fp.hit && fp.iumax >= iu0 && fp.iumin <= iu0 + kTU - 1) {
                        const int jlo = max(fp.iumin, iu0) - iu0, jhi = min(fp.iumax, iu0 + kTU - 1) - iu0;
                        const float scl = fp.ampu * fp.zinc;
#pragma unroll
                        for (int j = 0; j < kTU; j++) {
                            float w = 0.0f;
                            if (j >= jlo && j <= jhi)
                                w = u_weight<METHOD>(iu0 + j, fp.iumin, fp.iumax, fp.p0, fp.p1, fp.p2, fp.p3) * scl;
                            s_wf[t * kTU + j] = w;
                        }
                        const float b0 = fp.vstart + 0.5f;
                        const float btop = fmaf(fnz, fp.zinc, b0);
                        const int rlo = max((int)floorf(b0) - 1, 0);
                        const int rhi = min((int)floorf(btop) + 1, nv - 1);
                        if (rlo <= rhi) {
                            valid = true;
                            s_col[t] = col;
                            s_b0[t] = b0;
                            s_iz[t] = 1.0f / fp.zinc;
                            s_rlo[t] = rlo;
                            s_rhi[t] = rhi;
                            s_j[t] = jlo | (jhi << 8);
                        }
                    }
                }
            }
            if (!valid) s_j[t] = -1;
        }
        __syncthreads();
        // 4. row quads: R(iv) = X(iv+1) - X(iv) from the column's prefix pairs
        const int nslot = min(NT, ncand - c0);
        for (int s = grp; s < nslot; s += groups) {
            const int jj = s_j[s];
            if (jj < 0) continue;
            const int rlo = s_rlo[s], rhi = s_rhi[s];
            const float b0 = s_b0[s], izc = s_iz[s];
            const float *x = xs + (size_t)s_col[s] * (PAIRS ? 2 * (g.nz + 1) : g.xstride);
            const int jlo = jj & 0xff, jhi = jj >> 8;
            // groups of one warp own all their accumulator rows, so the warp walks the
            // candidate's own rows from rlo (128 per pass); wider groups own fixed bands
            const bool walk = R == 32;
            const int pstart = walk ? (rlo & ~3) : 0, pend = walk ? rhi + 1 : nv;
            for (int pbase = pstart; pbase < pend; pbase += rows_per_pass) {
                const int wrow = pbase + 128 * gwarp;  // first row of this warp's 128
                if (wrow > rhi || wrow + 127 < rlo) continue;  // warp-uniform
                const int iv0 = wrow + 4 * lane;
                const float f0 = small_int_to_float(iv0) - b0;
                float X0, X1, X2, X3;
                X0 = column_integral<PAIRS>(x, fminf(fmaxf(f0 * izc, 0.0f), fnz), nzm1, fnzm1);
                X1 = column_integral<PAIRS>(x, fminf(fmaxf((f0 + 1.0f) * izc, 0.0f), fnz), nzm1, fnzm1);
                X2 = column_integral<PAIRS>(x, fminf(fmaxf((f0 + 2.0f) * izc, 0.0f), fnz), nzm1, fnzm1);
                X3 = column_integral<PAIRS>(x, fminf(fmaxf((f0 + 3.0f) * izc, 0.0f), fnz), nzm1, fnzm1);
                float X4 = __shfl_down_sync(kFull, X0, 1);
                if (lane == 31) X4 = column_integral<PAIRS>(x, fminf(fmaxf((f0 + 4.0f) * izc, 0.0f), fnz), nzm1, fnzm1);
                if (iv0 <= rhi && iv0 + 3 >= rlo && iv0 < nv) {
                    const float R0 = X1 - X0, R1 = X2 - X1, R2 = X3 - X2, R3 = X4 - X3;
                    float4 *a = gacc + (iv0 >> 2);
                    for (int j = jlo; j <= jhi; j++) {
                        const float w = s_wf[s * kTU + j];
                        float4 r = a[j * nq];
                        r.x = fmaf(w, R0, r.x); r.y = fmaf(w, R1, r.y);
                        r.z = fmaf(w, R2, r.z); r.w = fmaf(w, R3, r.w);
                        a[j * nq] = r;
                    }
                }
            }
        }
        __syncthreads();
    }
    // 5. sum of the groups (in group order), axial amplitude and store
    const size_t obase = (size_t)k * g.nu * nv;
    const float *accf = reinterpret_cast<const float *>(acc4);
    const int gstride = kTU * 4 * nq;
    for (int j = 0; j < kTU; j++) {
        const int iu = iu0 + j;
        if (iu >= g.nu) break;
        for (int iv = t; iv < nv; iv += NT) {
            float a = accf[j * 4 * nq + iv];
#pragma unroll
            for (int q = 1; q < groups; q++) a += accf[q * gstride + j * 4 * nq + iv];
            store_from_float(proj, obase + (size_t)iu * nv + iv, a * ampv[(size_t)iu * nv + iv], out_dtype);
        }
    }
}

template <int METHOD, int GROUPS, bool PAIRS>
__global__ void __launch_bounds__(kProjMaxThreads) proj_kernel(Geom g, const View *__restrict__ views,
                                                               const float *__restrict__ xs,
                                                               const float *__restrict__ ampv,
                                                               const uint8_t *__restrict__ map,
                                                               void *__restrict__ proj, int out_dtype,
                                                               int view_begin, int view_stride, float margin,
                                                               int ngx, int vc) {
    extern __shared__ float4 acc4_smem[];
    int bx, by;
    view_grouped_block(blockIdx.x, ngx, vc, bx, by);
    proj_block<METHOD, GROUPS, PAIRS>(g, views, xs, ampv, map, proj, out_dtype, view_begin, view_stride, margin,
                                      acc4_smem, bx, by);
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
// The dynamic shared-memory limit is a per-function, per-device attribute shared by
// every plan, stream and captured graph of the process; it is only ever raised, so
// a launch recorded earlier (another request's stream, a CUDA graph) stays valid.
cudaError_t allow_dynamic_smem(const void *kfn, size_t bytes) {
    static std::mutex m;
    static std::map<std::pair<int, const void *>, size_t> granted;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(m);
    size_t &g = granted[{dev, kfn}];
    if (bytes <= g) return cudaSuccess;
    e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) g = bytes;
    return e;
}

// per warp: the u weights of 32 views and the row buffer; 4 spare floats past the last
// warp's buffer for the branch-free row reads
size_t back_smem_bytes(int qcap) { return ((size_t)8 * (32 * 17 + 32 * 8 + qcap) + 4) * sizeof(float); }

template <int METHOD, int MZ, bool VEC, int SRC, bool SUM>
static cudaError_t launch_back_mz(const Geom &g, const View *views, const void *ps, const float *ampv,
                                  const uint8_t *map, void *image, int out_dtype, int vb, int vs, int vc, float scale,
                                  int qcap, int *err, int y_begin, int y_end, cudaStream_t st) {
    const int tiles_x = (g.nx + 7) / 8;
    const int blocks = (y_end - y_begin) * tiles_x;
    if (blocks <= 0) return cudaSuccess;
    const size_t sm = back_smem_bytes(qcap);
    auto kfn = back_kernel<METHOD, MZ, VEC, SRC, SUM>;
    cudaError_t e = allow_dynamic_smem((const void *)kfn, sm);
    if (e != cudaSuccess) return e;
    kfn<<<blocks, 256, sm, st>>>(g, views, ps, map, image, out_dtype, vb, vs, vc, scale, qcap, err, ampv,
                                 y_begin * tiles_x);
    return cudaGetLastError();
}

cudaError_t launch_prescale(const void *proj, int in_dtype, const float *ampv, float *ps, size_t nuv, size_t n,
                            cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 32);
    prescale_kernel<<<blocks, 256, 0, st>>>(proj, in_dtype, ampv, ps, nuv, n);
    return cudaGetLastError();
}

cudaError_t launch_back(int method, int mz, const Geom &g, const View *views, const void *ps, const uint8_t *map,
                        void *image, int out_dtype, int vb, int vs, int vc, float scale, int qcap, int *err,
                        cudaStream_t st, bool accumulate, int y_begin, int y_end, int src, const float *ampv) {
    if (accumulate && (out_dtype != kF32 || scale != 1.0f || src != kSrcScaled)) return cudaErrorInvalidValue;
    if (src != kSrcScaled && src != kSrcBF16 && src != kSrcF16) return cudaErrorInvalidValue;
    if (src != kSrcScaled && !ampv) return cudaErrorInvalidValue;
    if (y_end < 0) y_end = g.ny;
    if (y_begin < 0 || y_end > g.ny || y_begin > y_end) return cudaErrorInvalidValue;
    const size_t align = src == kSrcScaled ? 16 : 8;  // one float4, or four 16-bit values, per load
    const bool vec = (g.nv % 4) == 0 && (reinterpret_cast<uintptr_t>(ps) % align) == 0 &&
                     (reinterpret_cast<uintptr_t>(ampv) % 16) == 0;
    // accumulate: the image holds the FP32 view sum of earlier views, which the kernel
    // continues (separate instantiations, so the plain kernel keeps its registers)
#define CTSIM_BACK_ARGS g, views, ps, ampv, map, image, out_dtype, vb, vs, vc, scale, qcap, err, y_begin, y_end, st
#define CTSIM_BACK_CASE(M, Z)                                                                            \
    if (method == M && mz == Z) {                                                                        \
        if (accumulate)                                                                                  \
            return vec ? launch_back_mz<M, Z, true, kSrcScaled, true>(CTSIM_BACK_ARGS)                   \
                       : launch_back_mz<M, Z, false, kSrcScaled, true>(CTSIM_BACK_ARGS);                 \
        if (src == kSrcBF16)                                                                             \
            return vec ? launch_back_mz<M, Z, true, kSrcBF16, false>(CTSIM_BACK_ARGS)                    \
                       : launch_back_mz<M, Z, false, kSrcBF16, false>(CTSIM_BACK_ARGS);                  \
        if (src == kSrcF16)                                                                              \
            return vec ? launch_back_mz<M, Z, true, kSrcF16, false>(CTSIM_BACK_ARGS)                     \
                       : launch_back_mz<M, Z, false, kSrcF16, false>(CTSIM_BACK_ARGS);                   \
        return vec ? launch_back_mz<M, Z, true, kSrcScaled, false>(CTSIM_BACK_ARGS)                      \
                   : launch_back_mz<M, Z, false, kSrcScaled, false>(CTSIM_BACK_ARGS);                    \
    }
    CTSIM_BACK_CASE(kDD, 1) CTSIM_BACK_CASE(kDD, 2) CTSIM_BACK_CASE(kDD, 4) CTSIM_BACK_CASE(kDD, 8)
    CTSIM_BACK_CASE(kTF, 1) CTSIM_BACK_CASE(kTF, 2) CTSIM_BACK_CASE(kTF, 4) CTSIM_BACK_CASE(kTF, 8)
#undef CTSIM_BACK_CASE
#undef CTSIM_BACK_ARGS
    return cudaErrorInvalidValue;
}

cudaError_t launch_prefix(const void *image, int in_dtype, float *xs, int nxy, int nz, bool pairs, int xstride,
                          cudaStream_t st) {
    const int blocks = (nxy + 31) / 32;
    if (pairs) prefix_kernel<true><<<blocks, 256, 0, st>>>(image, in_dtype, xs, nxy, nz, 0);
    else prefix_kernel<false><<<blocks, 256, 0, st>>>(image, in_dtype, xs, nxy, nz, xstride);
    return cudaGetLastError();
}

// Row threads R (one per 4 detector rows, whole warps, at most kProjMaxThreads) and
// candidate groups (1, 2, 4 or 8, with R * groups <= kProjMaxThreads).  Default: two
// groups wherever they fit (R <= 128, up to 512 rows) -- the fastest count on every
// shape measured on B200 (nv 72..384); one group above.  A plan's autotuner may pick
// another valid count.
static int proj_row_threads(int nv) {
    return std::min(kProjMaxThreads, std::max(32, ((nv + 3) / 4 + 31) / 32 * 32));
}
int proj_default_groups(int nv) { return proj_row_threads(nv) <= kProjMaxThreads / 2 ? 2 : 1; }
int proj_default_rows(int nv) { return proj_row_threads(nv); }
// rows: row threads of a group, a multiple of 32 up to the ones that cover nv in one
// pass (fewer loop over the rows in passes; 32 walks each candidate's own rows)
bool proj_shape_valid(int nv, int groups, int rows) {
    return (groups == 1 || groups == 2 || groups == 4 || groups == 8) && rows >= 32 && rows % 32 == 0 &&
           rows <= proj_row_threads(nv) && rows * groups <= kProjMaxThreads;
}
bool proj_groups_valid(int nv, int groups) { return proj_shape_valid(nv, groups, proj_row_threads(nv)); }
size_t proj_smem_bytes(int nv, int nx, int ny, int groups, int rows) {
    ProjSmem L{(nv + 3) / 4, rows * groups, std::max(nx, ny), groups};
    return L.bytes();
}
size_t proj_smem_bytes(int nv, int nx, int ny, int groups) {
    return proj_smem_bytes(nv, nx, ny, groups, proj_row_threads(nv));
}
int proj_max_lines() { return kMaxLines; }


cudaError_t launch_proj(int method, int groups, int rows, bool pairs, const Geom &g, const View *views,
                        const float *xc, const float *ampv, const uint8_t *map, void *proj, int out_dtype, int vb,
                        int vs, int vc, float margin, cudaStream_t st) {
    if (!proj_shape_valid(g.nv, groups, rows)) return cudaErrorInvalidValue;
    const size_t sm = proj_smem_bytes(g.nv, g.nx, g.ny, groups, rows);
    const int ngx = (g.nu + kTU - 1) / kTU;
    const int nblocks = ngx * vc;
    // one thread per 4 detector rows (rows threads per group, more rows loop), groups
    // of those threads share the candidates
    const int nt = rows * groups;
#define CTSIM_PROJ_CASE(M, GR, P)                                                                     \
    if (method == M && groups == GR && pairs == P) {                                                  \
        cudaError_t e = allow_dynamic_smem((const void *)proj_kernel<M, GR, P>, sm);                  \
        if (e != cudaSuccess) return e;                                                               \
        proj_kernel<M, GR, P><<<nblocks, nt, sm, st>>>(g, views, xc, ampv, map, proj, out_dtype, vb, vs, margin, \
                                                       ngx, vc);                                      \
        return cudaGetLastError();                                                                    \
    }
    CTSIM_PROJ_CASE(kDD, 1, false) CTSIM_PROJ_CASE(kDD, 2, false) CTSIM_PROJ_CASE(kDD, 4, false)
    CTSIM_PROJ_CASE(kDD, 8, false) CTSIM_PROJ_CASE(kTF, 1, false) CTSIM_PROJ_CASE(kTF, 2, false)
    CTSIM_PROJ_CASE(kTF, 4, false) CTSIM_PROJ_CASE(kTF, 8, false)
    CTSIM_PROJ_CASE(kDD, 1, true) CTSIM_PROJ_CASE(kDD, 2, true) CTSIM_PROJ_CASE(kDD, 4, true)
    CTSIM_PROJ_CASE(kDD, 8, true) CTSIM_PROJ_CASE(kTF, 1, true) CTSIM_PROJ_CASE(kTF, 2, true)
    CTSIM_PROJ_CASE(kTF, 4, true) CTSIM_PROJ_CASE(kTF, 8, true)
#undef CTSIM_PROJ_CASE
    return cudaErrorInvalidValue;
}

// A^T reading the unscaled sinogram (axial amplitude applied on the fly); used by the
// entry point that allocates nothing (noalloc.cu).
template <int METHOD, int MZ>
static cudaError_t launch_back_unscaled_mz(const Geom &g, const View *views, const float *proj, const float *ampv,
                                           const uint8_t *map, float *image, int vc, int qcap, int *err,
                                           cudaStream_t st) {
    const int blocks = g.ny * ((g.nx + 7) / 8);
    const size_t sm = back_smem_bytes(qcap);
    auto kfn = back_kernel<METHOD, MZ, false, kSrcF32>;
    cudaError_t e = allow_dynamic_smem((const void *)kfn, sm);
    if (e != cudaSuccess) return e;
    kfn<<<blocks, 256, sm, st>>>(g, views, proj, map, image, kF32, 0, 1, vc, 1.0f, qcap, err, ampv, 0);
    return cudaGetLastError();
}

cudaError_t launch_back_unscaled(int mz, const Geom &g, const View *views, const float *proj, const float *ampv,
                                 const uint8_t *map, float *image, int vc, int qcap, int *err, cudaStream_t st) {
    switch (mz) {
    case 1: return launch_back_unscaled_mz<kDD, 1>(g, views, proj, ampv, map, image, vc, qcap, err, st);
    case 2: return launch_back_unscaled_mz<kDD, 2>(g, views, proj, ampv, map, image, vc, qcap, err, st);
    case 4: return launch_back_unscaled_mz<kDD, 4>(g, views, proj, ampv, map, image, vc, qcap, err, st);
    case 8: return launch_back_unscaled_mz<kDD, 8>(g, views, proj, ampv, map, image, vc, qcap, err, st);
    }
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Batched launches.  One persistent grid (the resident blocks of the whole GPU) walks
// the flat block list of up to kBatchMax tasks -- plans of different geometries -- and
// runs each block's work with its task's tables; the task table is a __grid_constant__
// kernel parameter, so a batch needs no device allocation and can be graph-captured.
// ---------------------------------------------------------------------------
// LOWP: outputs in each task's storage type; otherwise FP32 (a compile-time store).
template <int METHOD, int GROUPS, bool PAIRS, bool LOWP>
__global__ void __launch_bounds__(kProjMaxThreads) proj_batch_kernel(const __grid_constant__ ProjBatch b) {
    extern __shared__ float4 acc4_batch[];
    for (int blk = blockIdx.x; blk < b.total; blk += gridDim.x) {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b.t[mid].first <= blk) lo = mid; else hi = mid - 1;
        }
        const ProjTask &T = b.t[lo];
        int bx, by;
        view_grouped_block(blk - T.first, T.gx, T.vc, bx, by);
        proj_block<METHOD, GROUPS, PAIRS>(T.g, T.views, T.xs, T.ampv, T.map, T.proj, LOWP ? T.out_dtype : kF32, T.vb,
                                          T.vs, T.margin, acc4_batch, bx, by);
        __syncthreads();  // the next block reuses the shared accumulators
    }
}

template <int METHOD, int MZ, bool VEC, bool LOWP, int SRC>
__global__ void __launch_bounds__(256) back_batch_kernel(const __grid_constant__ BackBatch b) {
    extern __shared__ float smem_batch[];
    for (int blk = blockIdx.x; blk < b.total; blk += gridDim.x) {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b.t[mid].first <= blk) lo = mid; else hi = mid - 1;
        }
        const BackTask &T = b.t[lo];
        back_block<METHOD, MZ, VEC, SRC>(T.g, T.views, T.ps, T.map, T.image, LOWP ? T.out_dtype : kF32, T.vb, T.vs,
                                         T.vc, T.scale, T.qcap, T.err, T.ampv, smem_batch, blk - T.first);
        // the per-warp row buffers are laid out with the task's own stride, so a warp may
        // not start the next item (possibly another task) while its neighbours still work
        __syncthreads();
    }
}

int back_task_blocks(const Geom &g) { return g.ny * ((g.nx + 7) / 8); }
int proj_row_threads_of(int nv) { return proj_row_threads(nv); }

int persistent_grid(const void *kernel, int threads, size_t smem, int total) {
    int dev = 0, sms = 148, per_sm = 1;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return std::max(1, std::min(total, sms * per_sm));
}

cudaError_t launch_proj_batch(int method, int groups, int row_threads, bool pairs, bool lowp, size_t smem,
                              const ProjBatch &b, cudaStream_t st) {
    if (b.n < 1 || b.total < 1) return cudaSuccess;
    const int nt = row_threads * groups;
#define CTSIM_PB_CASE(M, GR)                                                                          \
    if (method == M && groups == GR) {                                                                \
        auto k = pairs ? (lowp ? proj_batch_kernel<M, GR, true, true> : proj_batch_kernel<M, GR, true, false>) \
                       : (lowp ? proj_batch_kernel<M, GR, false, true> : proj_batch_kernel<M, GR, false, false>); \
        cudaError_t e = allow_dynamic_smem((const void *)k, smem);                                    \
        if (e != cudaSuccess) return e;                                                               \
        k<<<persistent_grid((const void *)k, nt, smem, b.total), nt, smem, st>>>(b);                                \
        return cudaGetLastError();                                                                    \
    }
    CTSIM_PB_CASE(kDD, 1) CTSIM_PB_CASE(kDD, 2) CTSIM_PB_CASE(kDD, 4) CTSIM_PB_CASE(kDD, 8)
    CTSIM_PB_CASE(kTF, 1) CTSIM_PB_CASE(kTF, 2) CTSIM_PB_CASE(kTF, 4) CTSIM_PB_CASE(kTF, 8)
#undef CTSIM_PB_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_back_batch(int method, int mz, bool vec, bool lowp, size_t smem, const BackBatch &b,
                              cudaStream_t st, int src) {
    if (b.n < 1 || b.total < 1) return cudaSuccess;
    if (src != kSrcScaled && src != kSrcBF16 && src != kSrcF16) return cudaErrorInvalidValue;
#define CTSIM_BB_LAUNCH(M, Z, V, S)                                                                   \
    {                                                                                                 \
        auto k = lowp ? back_batch_kernel<M, Z, V, true, S> : back_batch_kernel<M, Z, V, false, S>;   \
        cudaError_t e = allow_dynamic_smem((const void *)k, smem);                                    \
        if (e != cudaSuccess) return e;                                                               \
        k<<<persistent_grid((const void *)k, 256, smem, b.total), 256, smem, st>>>(b);                              \
        return cudaGetLastError();                                                                    \
    }
#define CTSIM_BB_CASE(M, Z, V)                                                                        \
    if (method == M && mz == Z && vec == V) {                                                         \
        if (src == kSrcBF16) CTSIM_BB_LAUNCH(M, Z, V, kSrcBF16)                                       \
        if (src == kSrcF16) CTSIM_BB_LAUNCH(M, Z, V, kSrcF16)                                         \
        CTSIM_BB_LAUNCH(M, Z, V, kSrcScaled)                                                          \
    }
    CTSIM_BB_CASE(kDD, 1, true) CTSIM_BB_CASE(kDD, 2, true) CTSIM_BB_CASE(kDD, 4, true) CTSIM_BB_CASE(kDD, 8, true)
    CTSIM_BB_CASE(kDD, 1, false) CTSIM_BB_CASE(kDD, 2, false) CTSIM_BB_CASE(kDD, 4, false) CTSIM_BB_CASE(kDD, 8, false)
    CTSIM_BB_CASE(kTF, 1, true) CTSIM_BB_CASE(kTF, 2, true) CTSIM_BB_CASE(kTF, 4, true) CTSIM_BB_CASE(kTF, 8, true)
    CTSIM_BB_CASE(kTF, 1, false) CTSIM_BB_CASE(kTF, 2, false) CTSIM_BB_CASE(kTF, 4, false) CTSIM_BB_CASE(kTF, 8, false)
#undef CTSIM_BB_CASE
#undef CTSIM_BB_LAUNCH
    return cudaErrorInvalidValue;
}

}  // namespace ctsim
