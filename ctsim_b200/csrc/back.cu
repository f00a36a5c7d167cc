// Matched backprojection A^T for sm_100a (distance-driven / separable footprint).
//
// Layouts (reference MEX conventions): image[iz][iy][ix], proj[view][iu][iv].
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"
#include "packed.cuh"

namespace ctsim {

// ---------------------------------------------------------------------------
// One warp per voxel column, lanes along z; 8 columns (consecutive ix) per block.  For each
// view the warp forms, in shared memory, the u-weighted detector column
//     q[iv] = sum_iu w_u(iu) * ps[iu][iv]        (ps = proj * ampv)
// over the rows the column's voxels can touch.  Each voxel then sums q over the rows its
// axial extent covers with the distance-driven row weights of geom/cbct/cbct_back.c:318-357,
// its edges vmin/vmax computed with the reference's float operations (usually two or three
// rows per voxel).  The edges sit hundreds of rows up the detector, where one float rounding
// moves a voxel's weight by ~1e-5 of itself; evaluating them exactly as the reference does
// keeps each voxel's value within a few float roundings of the reference's instead of adding
// noise of that size.  Accumulation over views stays in registers; no atomics.
//
// What bounds it: instruction issue.  So two voxels share every FP32 instruction; a view's
// detector columns are summed over all of its rows at once, from an address that the view's
// lane computed; and voxels whose extent covers at most two (zinc < 1) or three rows (zinc <
// 2) take their rows without a loop or a branch, on a clipped detector and in a last,
// shorter z pass too.
// ---------------------------------------------------------------------------

// Four FP32 values of a sinogram source: rows r, r + 1, r + 2, r + 3 of a detector column
// (VEC: one 16-byte FP32 or 8-byte 16-bit load), or the lane's rows r, r + 32, r + 64, r + 96.
// VEC = false: rows past r_hi read as 0.  a: the byte address of the first.
template <int SRC, bool VEC>
__device__ __forceinline__ float4 load_rows4(uintptr_t a, int r, int r_hi) {
    if (SRC == kSrcScaled || SRC == kSrcF32) {
        const float *p = reinterpret_cast<const float *>(a);
        if (VEC) return __ldg(reinterpret_cast<const float4 *>(p));
        return make_float4(r <= r_hi ? __ldg(p) : 0.f, r + 32 <= r_hi ? __ldg(p + 32) : 0.f,
                           r + 64 <= r_hi ? __ldg(p + 64) : 0.f, r + 96 <= r_hi ? __ldg(p + 96) : 0.f);
    }
    const unsigned short *p = reinterpret_cast<const unsigned short *>(a);
    unsigned short h[4];
    if (VEC) {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
        h[0] = (unsigned short)(u.x & 0xffffu); h[1] = (unsigned short)(u.x >> 16);
        h[2] = (unsigned short)(u.y & 0xffffu); h[3] = (unsigned short)(u.y >> 16);
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) h[i] = r + 32 * i <= r_hi ? __ldg(p + 32 * i) : (unsigned short)0;
    }
    float f[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        f[i] = SRC == kSrcBF16 ? __uint_as_float((unsigned)h[i] << 16) : __half2float(__ushort_as_half(h[i]));
    return make_float4(f[0], f[1], f[2], f[3]);
}

// 32-bit shared load ordered after the warp's earlier shared stores (compiler barrier).
__device__ __forceinline__ float lds_ordered(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// Detector rows up to which voxels may take their rows without a loop.
constexpr int kLoopFreeRows = 8192;

// The work of one block (8 columns of one row iy), as a device function: the plain
// kernel runs it for blockIdx.x, the batched kernel for each of its work items.
// one: 1.0f (padd_product).
template <int METHOD, int MZ, bool VEC, int SRC, bool SUM = false>
__device__ __forceinline__ void back_block(const Geom &g, const View *__restrict__ views, const void *__restrict__ ps,
                                           const uint8_t *__restrict__ map, void *__restrict__ image, int out_dtype,
                                           int view_begin, int view_stride, int view_count, float scale, int qcap,
                                           int *__restrict__ err, const float *__restrict__ ampv, float one_rt,
                                           float *smem, int block) {
    using V = std::conditional_t<MZ == 1, float, f32x2>;
    using P = Packed<V>;
    constexpr int W = P::kWidth, NP = MZ / W;  // voxels per register, registers per pass
    constexpr unsigned kSize = SRC == kSrcScaled || SRC == kSrcF32 ? 4 : 2;
    constexpr int kWS = 17;  // row stride of the per-warp weight table (conflict-free writes)
    constexpr int kGeneric = 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float *wtab = smem + warp * (32 * kWS + 32 * 8 + qcap);  // [32 views][17] u weights of the view chunk
    // [32 views] per-view scalars of the chunk, written by the view's own lane: {ampu, zinc, vstart,
    // nb | path << 8 | 128-row steps << 16}, {address of row rbase of the first detector column (low,
    // high word), qadj, r_hi - rbase | r_hi << 16}; path 0: no rows.  A half word holds every r_hi - rbase
    // (below qcap, which the block's shared memory holds eight times), and r_hi up to kLoopFreeRows
    // rows; taller detectors take path 5, which reads r_hi modulo 2^16.  Entry 16 of the view's weights
    // is the element offset of that row in ampv.  qadj: row k of Q is at shared address qadj + 4 *
    // bits(k + 2^23) (mod 2^32)
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
    const uint32_t q_u32 = (uint32_t)__cvta_generic_to_shared(Q);
    const unsigned col_step = (unsigned)g.nv * kSize;
    const V one = P::all(one_rt), half = P::all(0.5f);
    for (int iz0 = 0; iz0 < g.nz; iz0 += 32 * MZ) {
        const int izn = min(32 * MZ, g.nz - iz0);
        const float fz_first = (float)iz0, fz_last = (float)(iz0 + izn - 1);
        const size_t out0 = (size_t)(iz0 + lane) * nxy + (size_t)iy * g.nx + ix;
        V acc[NP], fz[NP];
#pragma unroll
        for (int p = 0; p < NP; p++) {
            acc[p] = P::all(0.0f);
            // lanes past the last slice repeat it (and are not stored)
            fz[p] = P::make([&](int i) { return fminf((float)(iz0 + lane + 32 * (W * p + i)), fz_last); });
            if (SUM)  // continue the per-voxel view sum (scale 1) that the previous view chunk left
                      // in the FP32 image; the sum runs in view order either way
                acc[p] = P::make([&](int i) {
                    const int dz = 32 * (W * p + i);
                    return lane + dz < izn ? static_cast<const float *>(image)[out0 + (size_t)dz * nxy] : 0.0f;
                });
        }
        if (on) {
            for (int k0 = 0; k0 < view_count; k0 += 32) {
                ColumnFP my;
                my.hit = false;
                const int kl = k0 + lane;
                if (kl < view_count) my = column_footprint<METHOD>(g, views[view_begin + kl * view_stride], ix, iy);
                // lane-parallel u weights of this lane's view (geom/cbct/cbct_back.c:288-301, :549-578)
                __syncwarp();  // the previous chunk's reads of wtab and vtab are done
                float4 ta = make_float4(0.f, 0.f, 0.f, 0.f), tb = make_float4(0.f, 0.f, 0.f, 0.f);
                // no detector column (nb 0): a footprint that only meets the detector's upper edge
                const int nb = my.hit ? my.iumax - my.iumin + 1 : 0;
                if (nb > 0) {
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
                            // A voxel's vmax - vmin is zinc within 1.5 float ulps of nv (< 2^-10 for nv <=
                            // kLoopFreeRows), so below 1 and 2 by a margin every voxel of the view covers
                            // at most two or three rows: paths 1 and 2, and 3 and 4 where the detector
                            // clips some voxel of the pass.
                            constexpr float kMargin = 1.0f / 256.0f;
                            int path = zinc < 1.0f - kMargin ? 1 : zinc < 2.0f - kMargin ? 2 : kGeneric;
                            if (g.nv > kLoopFreeRows) path = kGeneric;
                            if (path != kGeneric && !(a0u > 0.0f && b1u < fnv)) path += 2;
                            if (r_hi - rbase + 1 > qcap) {  // rows rbase..r_hi must fit
                                atomicOr(err, 1);
                                r_hi = rbase + qcap - 1;
                                path = kGeneric;
                            }
                            const size_t aoff = (size_t)my.iumin * g.nv + rbase;
                            const uintptr_t a = reinterpret_cast<uintptr_t>(ps) + ((size_t)kl * nuv + aoff) * kSize;
                            ta = make_float4(my.ampu, zinc, vstart,
                                             __int_as_float(nb | (path << 8) | (((r_hi - rbase) / 128 + 1) << 16)));
                            tb = make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)),
                                             __uint_as_float(q_u32 - 4u * (uint32_t)rbase - (0x4B000000u << 2)),
                                             __int_as_float((r_hi - rbase) | (r_hi << 16)));
                            if (SRC != kSrcScaled) wtab[lane * kWS + 16] = __uint_as_float((unsigned)aoff);
                        }
                    }
                }
                vtab[2 * lane] = ta;
                vtab[2 * lane + 1] = tb;
                __syncwarp();
                const int nk = min(32, view_count - k0);
                for (int j = 0; j < nk; j++) {
                    const float4 pa = vtab[2 * j];
                    const int code = __float_as_int(pa.w);
                    if (code == 0) continue;  // no footprint or no rows
                    const float4 pb = vtab[2 * j + 1];
                    const int nb = code & 0xff, path = (code >> 8) & 0xff, steps = code >> 16;
                    const int last = __float_as_int(pb.w) & 0xffff;  // r_hi - rbase
                    // q over rows [rbase, r_hi] (the voxels read rows [r_lo, r_hi] only), 128 rows per step, a
                    // detector column added to all of a call's steps.  A lane past r_hi repeats the last row
                    // quad (VEC) or adds nothing; what it leaves in Q is not used.
                    const float *wj = wtab + j * kWS;
                    const uintptr_t col = ((uintptr_t)__float_as_uint(pb.y) << 32) | __float_as_uint(pb.x);
                    auto q_rows = [&](auto steps_c, int c) {  // steps from row rbase + c on
                        constexpr int S = decltype(steps_c)::value;
                        f32x2 q[S][2];
                        int o[S];  // this lane's first row of each step, from rbase
                        uintptr_t a[S], am[S];
#pragma unroll
                        for (int t = 0; t < S; t++) {
                            o[t] = VEC ? min(c + 128 * t + 4 * lane, last & ~3) : c + 128 * t + lane;
                            a[t] = col + (unsigned)o[t] * kSize;
                            if (SRC != kSrcScaled)
                                am[t] = reinterpret_cast<uintptr_t>(ampv) + 4 * (size_t)(__float_as_uint(wj[16]) + o[t]);
                        }
                        auto add = [&](int b, bool first) {
                            const f32x2 w = pack2(wj[b], wj[b]);
#pragma unroll
                            for (int t = 0; t < S; t++) {
                                float4 v = load_rows4<SRC, VEC>(a[t], o[t], last);
                                f32x2 lo = pack2(v.x, v.y), hi = pack2(v.z, v.w);
                                a[t] += col_step;
                                if (SRC != kSrcScaled) {  // axial amplitude applied here instead of in a scratch copy
                                    v = load_rows4<kSrcF32, VEC>(am[t], o[t], last);
                                    lo = pmul(lo, pack2(v.x, v.y));
                                    hi = pmul(hi, pack2(v.z, v.w));
                                    am[t] += 4u * (unsigned)g.nv;
                                }
                                q[t][0] = first ? pmul(w, lo) : pfma(w, lo, q[t][0]);
                                q[t][1] = first ? pmul(w, hi) : pfma(w, hi, q[t][1]);
                            }
                        };
                        add(0, true);
                        for (int b = 1; b < nb; b++) add(b, false);
#pragma unroll
                        for (int t = 0; t < S; t++) {
                            float4 v;
                            unpack2(q[t][0], v.x, v.y);
                            unpack2(q[t][1], v.z, v.w);
                            if (VEC) {
                                *reinterpret_cast<float4 *>(Q + c + 128 * t + 4 * lane) = v;
                            } else {
                                float *d = Q + o[t];
                                d[0] = v.x; d[32] = v.y; d[64] = v.z; d[96] = v.w;
                            }
                        }
                    };
                    if (steps == 1) {
                        q_rows(std::integral_constant<int, 1>{}, 0);
                    } else {
                        q_rows(std::integral_constant<int, 2>{}, 0);
                        for (int t = 2; t < steps; t++) q_rows(std::integral_constant<int, 1>{}, 128 * t);
                    }
                    __syncwarp();
                    // Each voxel: the reference's clamped extent and row weights
                    // (geom/cbct/cbct_back.c:318-357); its rows lie in [r_lo, r_hi] because the edges are
                    // monotone in iz.
                    const V ampu = P::all(pa.x), zinc = P::all(pa.y), vstart = P::all(pa.z);
                    const uint32_t qadj = __float_as_uint(pb.z);
                    const int r_hi = __float_as_int(pb.w) >> 16;
                    // ROWS rows from floor(vmin) = k on, weights min(vmax, k + 1) - vmin, min(vmax - (k + 1),
                    // 1) and vmax - (k + 2): the reference's values (one of its branches each).  A row that
                    // the extent does not reach (a negative weight, or a row off the detector) may hold
                    // anything, so its value is replaced; one it touches with weight 0 counts, as there.
                    auto voxels = [&](auto rows_c, auto clip_c) {
                        constexpr int ROWS = decltype(rows_c)::value;
                        constexpr bool CLIP = decltype(clip_c)::value;
                        const float t_hi = __int_as_float(0x4B000000 + r_hi);
#pragma unroll
                        for (int p = 0; p < NP; p++) {
                            if (p > 0 && 32 * W * p >= izn) break;  // warp-uniform
                            const V vpre = padd_product(pmul(fz[p], zinc), one, vstart);  // vstart + iz * zinc
                            V vmin = padd(vpre, half), vmax = padd(padd(vpre, zinc), half);
                            if (CLIP) {
                                vmin = P::make([&](int i) { return fmaxf(P::get(vmin, i), 0.0f); });
                                vmax = P::make([&](int i) { return fminf(P::get(vmax, i), fnv); });
                            }
                            V t = padd_rd(vmin, P::all(kTwo23));
                            if (CLIP) t = P::make([&](int i) { return fminf(P::get(t, i), t_hi); });
                            const V k1 = psub(t, P::all(kTwo23 - 1.0f));  // k + 1, exact
                            const V w0 = psub(P::make([&](int i) { return fminf(P::get(vmax, i), P::get(k1, i)); }), vmin);
                            V w1 = psub(vmax, k1), w2 = w1;
                            if (ROWS == 3) {
                                w2 = psub(vmax, psub(t, P::all(kTwo23 - 2.0f)));
                                w1 = P::make([&](int i) { return fminf(P::get(w1, i), 1.0f); });
                            }
                            float q0[W], q1[W], q2[W];
#pragma unroll
                            for (int i = 0; i < W; i++) {
                                const uint32_t qa = qadj + (__float_as_uint(P::get(t, i)) << 2);
                                q0[i] = lds_ordered(qa);
                                q1[i] = lds_ordered(qa + 4u);
                                if (ROWS == 3) q2[i] = lds_ordered(qa + 8u);
                                const float k1i = P::get(k1, i), lo = P::get(vmin, i);
                                if (CLIP) q0[i] = lo <= P::get(vmax, i) && lo < fnv ? q0[i] : 0.0f;
                                q1[i] = P::get(w1, i) >= 0.0f && (!CLIP || k1i < fnv) ? q1[i] : 0.0f;
                                if (ROWS == 3) q2[i] = P::get(w2, i) >= 0.0f && (!CLIP || k1i < fnv - 1.0f) ? q2[i] : 0.0f;
                            }
                            V vox = pfma(w1, P::make([&](int i) { return q1[i]; }),
                                         pmul(w0, P::make([&](int i) { return q0[i]; })));
                            if (ROWS == 3) vox = pfma(w2, P::make([&](int i) { return q2[i]; }), vox);
                            acc[p] = pfma(ampu, vox, acc[p]);
                        }
                    };
                    if (path == 1) {
                        voxels(std::integral_constant<int, 2>{}, std::false_type{});
                    } else if (path == 2) {
                        voxels(std::integral_constant<int, 3>{}, std::false_type{});
                    } else if (path == 3) {
                        voxels(std::integral_constant<int, 2>{}, std::true_type{});
                    } else if (path == 4) {
                        voxels(std::integral_constant<int, 3>{}, std::true_type{});
                    } else {
                        const uint32_t qrow = qadj + (0x4B000000u << 2);
                        auto qb = [&](int k) { return lds_ordered(qrow + 4u * (uint32_t)k); };
#pragma unroll
                        for (int p = 0; p < NP; p++) {
                            if (p > 0 && 32 * W * p >= izn) break;  // warp-uniform
                            acc[p] = P::make([&](int i) {
                                const float izv = P::get(fz[p], i);
                                const float vpre = fadd(pa.z, fmul(izv, pa.y));
                                const float vmin = fmaxf(fadd(vpre, 0.5f), 0.0f);             // max(vmin + 0.5, 0)
                                const float vmax = fminf(fadd(fadd(vpre, pa.y), 0.5f), fnv);  // min(vmax + 0.5, nv)
                                const float a = P::get(acc[p], i);
                                if (!(vmin <= vmax)) return a;
                                float flo, fhi;
                                const int klo = floor_pos(vmin, &flo);
                                int khi = floor_pos(vmax, &fhi);
                                if (khi > nvm1) { khi = nvm1; fhi = fsub(fnv, 1.0f); }
                                if (khi > klo + (kMaxRowsV - 1)) {
                                    khi = klo + (kMaxRowsV - 1);
                                    fhi = fadd(flo, (float)(kMaxRowsV - 1));
                                }
                                // at most r_hi, from its low half (a pass spans fewer than 2^15 rows): only
                                // after a row-buffer overflow (flagged above)
                                khi = min(khi, klo + (int)(short)(r_hi - klo));
                                float vox = 0.0f;
                                if (klo == khi) {
                                    vox = fsub(vmax, vmin) * qb(klo);
                                } else if (klo < khi) {
                                    vox = fsub(fadd(flo, 1.0f), vmin) * qb(klo);
                                    #pragma unroll 4
                                    for (int k = klo + 1; k < khi; k++) vox += qb(k);
                                    vox = fmaf(fsub(vmax, fhi), qb(khi), vox);
                                }
                                return fmaf(pa.x, vox, a);
                            });
                        }
                    }
                    __syncwarp();
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int p = 0; p < NP; p++)
#pragma unroll
            for (int i = 0; i < W; i++) {
                const int dz = 32 * (W * p + i);
                if (lane + dz < izn)
                    store_from_float(image, out0 + (size_t)dz * nxy, on ? P::get(acc[p], i) * scale : 0.0f, out_dtype);
            }
    }
}

// Four resident blocks per SM (registers capped at 64): measured on B200 at 512^2 x 256 and 720
// views, DD 110 -> 100 ms and SF 143 -> 104 ms against the uncapped 80-118 registers.  The geometry
// stays in the parameters: copied, its size decides which values spill (128^2 x 64, BF16, 360 views
// 0.995 -> 1.013 ms).
template <int METHOD, int MZ, bool VEC, int SRC = kSrcScaled, bool SUM = false>
__global__ void __launch_bounds__(256, 4) back_kernel(const __grid_constant__ Geom g, const View *__restrict__ views,
                                                   const void *__restrict__ ps, const uint8_t *__restrict__ map,
                                                   void *__restrict__ image, int out_dtype, int view_begin,
                                                   int view_stride, int view_count, float scale, int qcap,
                                                   int *__restrict__ err, const float *__restrict__ ampv, float one,
                                                   int block_base) {
    extern __shared__ float smem[];
    back_block<METHOD, MZ, VEC, SRC, SUM>(g, views, ps, map, image, out_dtype, view_begin, view_stride, view_count,
                                          scale, qcap, err, ampv, one, smem, block_base + blockIdx.x);
}

// A batch (see kernels.cuh): persistent blocks over the flat block list of many plans.
template <int METHOD, int MZ, bool VEC, bool LOWP, int SRC>
__global__ void __launch_bounds__(256) back_batch_kernel(const __grid_constant__ BackBatch b, float one) {
    extern __shared__ float smem_batch[];
    for (int blk = blockIdx.x; blk < b.total; blk += gridDim.x) {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b.t[mid].first <= blk) lo = mid; else hi = mid - 1;
        }
        const BackTask &T = b.t[lo];
        back_block<METHOD, MZ, VEC, SRC>(T.g, T.views, T.ps, T.map, T.image, LOWP ? T.out_dtype : kF32, T.vb, T.vs,
                                         T.vc, T.scale, T.qcap, T.err, T.ampv, one, smem_batch, blk - T.first);
        // the per-warp row buffers are laid out with the task's own stride, so a warp may
        // not start the next item (possibly another task) while its neighbours still work
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
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
                                 1.0f, y_begin * tiles_x);
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
    kfn<<<blocks, 256, sm, st>>>(g, views, proj, map, image, kF32, 0, 1, vc, 1.0f, qcap, err, ampv, 1.0f, 0);
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

int back_task_blocks(const Geom &g) { return g.ny * ((g.nx + 7) / 8); }

cudaError_t launch_back_batch(int method, int mz, bool vec, bool lowp, size_t smem, const BackBatch &b,
                              cudaStream_t st, int src) {
    if (b.n < 1 || b.total < 1) return cudaSuccess;
    if (src != kSrcScaled && src != kSrcBF16 && src != kSrcF16) return cudaErrorInvalidValue;
#define CTSIM_BB_LAUNCH(M, Z, V, S)                                                                   \
    {                                                                                                 \
        auto k = lowp ? back_batch_kernel<M, Z, V, true, S> : back_batch_kernel<M, Z, V, false, S>;   \
        cudaError_t e = allow_dynamic_smem((const void *)k, smem);                                    \
        if (e != cudaSuccess) return e;                                                               \
        k<<<persistent_grid((const void *)k, 256, smem, b.total), 256, smem, st>>>(b, 1.0f);                            \
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
