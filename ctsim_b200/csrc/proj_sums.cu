// Forward projector A for sm_100a with the candidates' prefix columns staged in shared memory:
// volumes whose paired sums do not stay cache-resident and whose detector rows reach more than
// three voxels (proj_staged.cu, which takes a row's voxels one by one, serves the others).
//
// One block per (group of kTU detector columns, view), candidate columns from the monotone
// projected centres of the volume's lines, exact footprints per candidate, rows accumulated as
// w_u * ampu * zinc * (X(iv + 1) - X(iv)) by the thread that owns them.  The valid candidates of
// a chunk are packed into a list, and their whole prefix columns (g.xstride floats, X[nz]
// repeated at the top) are copied from global memory into shared memory by the copy engine
// (cp.async.bulk, completion counted in bytes on an mbarrier), `slots` columns at a time into
// one of two buffers, so that the copies of the next slots overlap the row loop over the
// current ones.  Two sums bound a row whatever its length, so long rows cost no more than short
// ones; four lanes' rows share a bank, and the fixed bands of 128 rows are filled in part.
//
// Bound by instruction issue (about 60 lane-instructions per voxel and view).  Measured on
// B200, DD A, rows of 2.1, 3.2, 4 and 6 voxels against staged voxel columns (single sums for the
// last): 300^2 x 400, 16 views 1.07, 1.05, 1.09, 1.08 against 1.52, 1.25, 1.55, 2.69 ms; 512^2 x
// 256, 16 views 2.21, 1.96, 1.95, 1.96 against 2.23, 2.51, 2.40, 4.74 ms; 200^2 x 1200, 12 views
// 1.10, 1.22, 0.83, 0.80 against single sums 1.92, 1.51, 1.52, 1.64 ms.
#include <algorithm>

#include "kernels.cuh"
#include "mbar.cuh"

namespace ctsim {

namespace {

constexpr int kTU = kProjGroupWidth;
constexpr int kProjMaxThreads = 256;

// X(s) of a staged column, s clamped to [0, nz] (X[nz + 1] = X[nz] is part of the copy).
// xadj: the column's shared-memory address minus 4 * 0x4B000000 (mod 2^32), so that the
// address of X[floor(s)] is xadj + 4 * bits(s + 2^23 rounded down).
__device__ __forceinline__ float column_sum(uint32_t xadj, float s, float fnz) {
    s = fminf(fmaxf(s, 0.0f), fnz);
    const float t = __fadd_rd(s, kTwo23);
    const uint32_t a = xadj + (__float_as_uint(t) << 2);
    float x0, x1;
    asm volatile("ld.shared.f32 %0, [%2];\n\tld.shared.f32 %1, [%2+4];" : "=f"(x0), "=f"(x1) : "r"(a));
    return fmaf(s - (t - kTwo23), x1 - x0, x0);
}
// acc += w * (r0, r1, r2, r3) on the float4 at shared address a.
__device__ __forceinline__ void acc_add4(uint32_t a, float w, float r0, float r1, float r2, float r3) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    v.x = fmaf(w, r0, v.x); v.y = fmaf(w, r1, v.y); v.z = fmaf(w, r2, v.z); v.w = fmaf(w, r3, v.w);
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// Dynamic shared-memory layout: four mbarriers (first, so
// that a persistent block keeps them across work items of different shapes), the
// accumulators, the two stage buffers, the packed candidate table, the
// line tables.
struct SumsSmem {
    int nq, nt, nlines, groups, slots, xstride;
    __host__ __device__ size_t acc_bytes() const { return (size_t)groups * kTU * nq * 16; }
    __host__ __device__ size_t stage_floats() const { return (size_t)slots * xstride; }  // one buffer
    __host__ __device__ size_t bytes() const {
        return 32 + acc_bytes() + 2 * stage_floats() * 4 + (size_t)nt * (5 + kTU) * 4 +
               (size_t)(2 * nlines + 1 + 32) * 4;
    }
};

// The stage buffers form a two-deep full/empty pipeline: bar[b] ("full", one arrival plus
// the copies' bytes) completes when buffer b holds its slots, bar[2 + b] ("empty", one
// arrival per warp) when every warp has finished reading it.  A thread's `phase` holds the
// parity of the next completion it waits for: bit b for full[b], bit 2 + b for empty[b].
// The empty bits start at 1, the parity of the phase before a fresh barrier's first,
// which counts as complete, so the first copies into each buffer do not wait.
constexpr unsigned kSumsPhase0 = 0xCu;

__device__ __forceinline__ void sums_bars_init(uint64_t *bar) {
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_init(&bar[2], blockDim.x >> 5);
        mbar_init(&bar[3], blockDim.x >> 5);
        mbar_init_fence();
    }
    __syncthreads();
}

// Candidate intervals of the lines for detector columns [iu0, iu0 + kTU) of view v:
// line_start[L], and line_off[L] the exclusive scan of the counts (line_off[nlines] =
// the total).  All threads of the block call it; ends with a block barrier.
__device__ __forceinline__ int candidate_lines(const Geom &g, const View &v, int iu0, float margin, bool rows,
                                               int *line_start, int *line_off, int *s_warp_tot) {
    const int NT = blockDim.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
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
        line_off[L] = lo - first;
    }
    __syncthreads();
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
    __syncthreads();
    return line_off[nlines];
}

// The work of one block.  bar: the block's four stage mbarriers (initialised once per
// block by sums_bars_init); phase: their next-completion parities, carried across the
// items of a persistent block (kSumsPhase0 at the start); acc4: the shared memory past
// the mbarriers.  Returns false when a stage wait ran out (the block has then set
// kErrStageWait, waited for its copies in flight and must stop).
template <int METHOD, int GROUPS>
__device__ __forceinline__ bool proj_sums_block(const Geom g, const View *__restrict__ views,
                                                  const float *__restrict__ xs, const float *__restrict__ ampv,
                                                  const uint8_t *__restrict__ map, void *__restrict__ proj,
                                                  int out_dtype, int view_begin, int view_stride, float margin,
                                                  int slots, int *__restrict__ err, float4 *acc4, uint64_t *bar,
                                                  unsigned &phase, int bx, int by) {
    const int NT = blockDim.x;
    const int R = NT / GROUPS;
    const int nv = g.nv;
    const int nq = (nv + 3) >> 2;
    const int nlines0 = max(g.nx, g.ny);
    const int xst = g.xstride;
    SumsSmem L{nq, NT, nlines0, GROUPS, slots, xst};
    float *stage = reinterpret_cast<float *>(acc4 + GROUPS * kTU * nq);  // [2][slots][xst]
    // per candidate slot: {-b0 / zinc, 1 / zinc, rlo | rhi << 16, jlo | jhi << 8} (one 16-byte load)
    // (all three indexed by the candidate's position among the chunk's valid candidates)
    float4 *c_prm = reinterpret_cast<float4 *>(stage + 2 * L.stage_floats());
    int *c_col = reinterpret_cast<int *>(c_prm + NT);
    float *c_w = reinterpret_cast<float *>(c_col + NT);  // [NT][kTU]
    int *line_start = reinterpret_cast<int *>(c_w + NT * kTU);
    int *line_off = line_start + nlines0;
    int *s_warp_tot = line_off + nlines0 + 1;  // [32]

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int grp = GROUPS == 1 ? 0 : t / R;
    const int gwarp = GROUPS == 1 ? warp : (t - grp * R) >> 5;
    const int iu0 = bx * kTU;
    const View v = views[view_begin + by * view_stride];
    for (int i = t; i < GROUPS * kTU * nq; i += NT) acc4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 *gacc = acc4 + grp * kTU * nq;
    // 32-bit shared addresses of the row loop's tables
    const uint32_t acc_u32 = smem_addr(gacc), nq16 = 16u * (uint32_t)nq;
    const uint32_t prm_u32 = smem_addr(c_prm), w_u32 = smem_addr(c_w);
    const float fnz = (float)g.nz;
    // rows iv0 .. iv0 + 3 (f0 = iv0 as float) of one candidate: X at the five row edges from
    // the staged column (xadj), R = X(iv + 1) - X(iv), added with the weights at wq (16-byte
    // aligned, the first for the candidate's first column) into the accumulator columns at aq
    // (pjn + 1 of them).  Boundary iv sits at s = iv / zinc -
    // b0 / zinc (psa, piz), one rounding from iv alone, so a row's value does not depend on
    // which lane, warp or pass evaluates it; rows outside the column's shadow have both
    // edges clamped to the same end of the column and add exactly 0 (no per-lane test).
    auto row_quad = [&](int iv0, float f0, float psa, float piz, uint32_t xadj, uint32_t wq, uint32_t aq,
                           int pjn) {
        const float X0 = column_sum(xadj, fmaf(f0, piz, psa), fnz);
        const float X1 = column_sum(xadj, fmaf(f0 + 1.0f, piz, psa), fnz);
        const float X2 = column_sum(xadj, fmaf(f0 + 2.0f, piz, psa), fnz);
        const float X3 = column_sum(xadj, fmaf(f0 + 3.0f, piz, psa), fnz);
        const float X4 = column_sum(xadj, fmaf(f0 + 4.0f, piz, psa), fnz);
        if (iv0 < nv) {
            const float R0 = X1 - X0, R1 = X2 - X1, R2 = X3 - X2, R3 = X4 - X3;
            const uint32_t a = aq + 4u * (uint32_t)iv0;  // float4 of rows iv0 .. iv0 + 3
            const float4 w4 = lds_f32x4(wq);  // the candidate's first four weights
            acc_add4(a, w4.x, R0, R1, R2, R3);
            if (pjn > 0) {
                acc_add4(a + nq16, w4.y, R0, R1, R2, R3);
                if (pjn > 1) {
                    acc_add4(a + 2u * nq16, w4.z, R0, R1, R2, R3);
                    if (pjn > 2) {
                        acc_add4(a + 3u * nq16, w4.w, R0, R1, R2, R3);
                        for (int j = 4; j <= pjn; j++)
                            acc_add4(a + (uint32_t)j * nq16, lds_f32(wq + 4u * j), R0, R1, R2, R3);
                    }
                }
            }
        }
    };
    const bool rows = fabsf(v.cos_a) >= fabsf(v.sin_a);
    const int nlines = rows ? g.ny : g.nx;
    const int ncand = candidate_lines(g, v, iu0, margin, rows, line_start, line_off, s_warp_tot);
    const int rows_per_pass = 4 * R;
    const unsigned col_bytes = (unsigned)xst * 4u;
    int buf0 = 0;   // buffer of the next chunk's first slots
    int vbase = 0;  // valid candidates of the earlier chunks

    for (int c0 = 0; c0 < ncand; c0 += NT) {
        // 1. exact footprint of candidate c0 + t; the valid candidates' scalars, weights and
        // columns are packed in candidate order
        bool valid = false;
        int my_col = 0;
        float4 my_prm;
        float my_w[kTU];
        {
            const int c = c0 + t;
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
                        // weight i for detector column iu0 + jlo + i (16-byte loads in the row loop)
#pragma unroll
                        for (int i = 0; i < kTU; i++) {
                            float w = 0.0f;
                            if (jlo + i <= jhi)
                                w = u_weight<METHOD>(iu0 + jlo + i, fp.iumin, fp.iumax, fp.p0, fp.p1, fp.p2, fp.p3) *
                                    scl;
                            my_w[i] = w;
                        }
                        const float b0 = fp.vstart + 0.5f;
                        const float btop = fmaf(fnz, fp.zinc, b0);
                        const int rlo = max((int)floorf(b0) - 1, 0);
                        const int rhi = min((int)floorf(btop) + 1, nv - 1);
                        if (rlo <= rhi) {
                            valid = true;
                            const float izc = 1.0f / fp.zinc;
                            my_col = col;
                            // s(iv) = iv / zinc - b0 / zinc
                            my_prm = make_float4(-b0 * izc, izc, __int_as_float(rlo | (rhi << 16)),
                                                 __int_as_float(jlo | (jhi << 8)));
                        }
                    }
                }
            }
        }
        const unsigned bal = __ballot_sync(kFull, valid);
        if (lane == 0) s_warp_tot[warp] = __popc(bal);
        __syncthreads();
        int base = 0, nval = 0;
        for (int w = 0; w < (NT >> 5); w++) {
            const int n = s_warp_tot[w];
            base += w < warp ? n : 0;
            nval += n;
        }
        if (valid) {
            const int q = base + __popc(bal & ((1u << lane) - 1u));
            c_col[q] = my_col;
            c_prm[q] = my_prm;
#pragma unroll
            for (int j = 0; j < kTU; j++) c_w[q * kTU + j] = my_w[j];
        }
        __syncthreads();

        // 2. the packed candidates, `slots` at a time: warp 0 issues the copies of the next
        // slots into the other buffer once every warp has released it, while the warps run
        // the rows of the current ones; each warp releases a buffer when it is done with it
        const int nsub = (nval + slots - 1) / slots;
        bool failed = false;
        auto issue = [&](int sub, int buf) {
            const int p0 = sub * slots, n = min(slots, nval - p0);
            const bool free = mbar_wait(&bar[2 + buf], (phase >> (2 + buf)) & 1u);
            phase ^= 4u << buf;
            failed |= !free;
            // a buffer that was not released gets no copies: its full phase completes empty
            // and the block stops at the end of the chunk
            if (lane == 0) mbar_arrive_expect(&bar[buf], free ? (unsigned)n * col_bytes : 0u);
            __syncwarp();
            if (!free) return;
            float *dst = stage + (size_t)buf * L.stage_floats();
            for (int i = lane; i < n; i += 32)
                bulk_copy_g2s(dst + (size_t)i * xst, xs + (size_t)c_col[p0 + i] * xst, col_bytes, &bar[buf]);
        };
        if (nsub > 0 && warp == 0) issue(0, buf0);
        for (int sub = 0; sub < nsub; sub++) {
            const int buf = (buf0 + sub) & 1;
            if (sub + 1 < nsub && warp == 0) issue(sub + 1, buf ^ 1);
            failed |= !mbar_wait(&bar[buf], (phase >> buf) & 1u);
            phase ^= 1u << buf;
            const uint32_t sb = smem_addr(stage + (size_t)buf * L.stage_floats()) - (0x4B000000u << 2);
            const int p0 = sub * slots, p1 = min(nval, p0 + slots);
            // group g takes the valid candidates whose position in the block's whole sequence of
            // valid candidates (vbase + p) is g mod GROUPS, in order: the same split and order
            // whatever the chunk, row-thread or slot counts
            const int pstart0 = p0 + (((grp - vbase - p0) % GROUPS) + GROUPS) % GROUPS;
            if (R == 32) {
                // one-warp groups walk each candidate's own rows (every row of the group is theirs)
                for (int p = pstart0; p < p1; p += GROUPS) {
                    const float4 prm = lds_f32x4(prm_u32 + 16u * (uint32_t)p);
                    const int rr = __float_as_int(prm.z), jj = __float_as_int(prm.w);
                    const int prlo = rr & 0xffff, prhi = rr >> 16;
                    const int pjlo = jj & 0xff;
                    const uint32_t xadj = sb + (uint32_t)((p - p0) * xst) * 4u;
                    for (int wrow = prlo & ~3; wrow <= prhi; wrow += 128)
                        row_quad(wrow + 4 * lane, small_int_to_float(wrow + 4 * lane), prm.x, prm.y, xadj,
                                    w_u32 + 4u * (uint32_t)(p * kTU), acc_u32 + nq16 * (uint32_t)pjlo,
                                    (jj >> 8) - pjlo);
                }
            } else {
                // fixed bands: warp gwarp owns rows pbase + 128 gwarp .. + 127 of each pass
                for (int pbase = 0; pbase < nv; pbase += rows_per_pass) {
                    const int wrow = pbase + 128 * gwarp;
                    const int iv0 = wrow + 4 * lane;
                    const float f0 = small_int_to_float(iv0);
                    for (int p = pstart0; p < p1; p += GROUPS) {
                        const float4 prm = lds_f32x4(prm_u32 + 16u * (uint32_t)p);
                        const int rr = __float_as_int(prm.z), jj = __float_as_int(prm.w);
                        if (wrow > (rr >> 16) || wrow + 127 < (rr & 0xffff)) continue;  // warp-uniform
                        const int pjlo = jj & 0xff;
                        row_quad(iv0, f0, prm.x, prm.y, sb + (uint32_t)((p - p0) * xst) * 4u,
                                    w_u32 + 4u * (uint32_t)(p * kTU), acc_u32 + nq16 * (uint32_t)pjlo,
                                    (jj >> 8) - pjlo);
                    }
                }
            }
            // this warp is done with buffer `buf`
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar[2 + buf]);
        }
        // every warp is done with this chunk's candidate tables before the next chunk
        // rewrites them
        if (__syncthreads_or(failed)) {
            if (t == 0) atomicOr(err, kErrStageWait);
            // let copies still in flight land before the block stops (bounded waits: a
            // phase that completed, or never began, returns at once)
            mbar_wait(&bar[0], (phase & 1u) ^ 1u);
            mbar_wait(&bar[1], ((phase >> 1) & 1u) ^ 1u);
            return false;
        }
        buf0 = (buf0 + nsub) & 1;
        vbase += nval;
    }
    if (ncand == 0) __syncthreads();
    // 3. sum of the groups (in group order), axial amplitude and store
    const size_t obase = (size_t)by * g.nu * nv;
    const float *accf = reinterpret_cast<const float *>(acc4);
    const int gstride = kTU * 4 * nq;
    for (int j = 0; j < kTU; j++) {
        const int iu = iu0 + j;
        if (iu >= g.nu) break;
        for (int iv = t; iv < nv; iv += NT) {
            float a = accf[j * 4 * nq + iv];
#pragma unroll
            for (int q = 1; q < GROUPS; q++) a += accf[q * gstride + j * 4 * nq + iv];
            store_from_float(proj, obase + (size_t)iu * nv + iv, a * ampv[(size_t)iu * nv + iv], out_dtype);
        }
    }
    return true;
}

template <int METHOD, int GROUPS>
__global__ void __launch_bounds__(kProjMaxThreads, 3) proj_sums_kernel(Geom g, const View *__restrict__ views,
                                                                      const float *__restrict__ xs,
                                                                      const float *__restrict__ ampv,
                                                                      const uint8_t *__restrict__ map,
                                                                      void *__restrict__ proj, int out_dtype,
                                                                      int view_begin, int view_stride, float margin,
                                                                      int slots, int *__restrict__ err, int ngx,
                                                                      int vc) {
    extern __shared__ float4 smem_sums[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_sums);
    sums_bars_init(bar);
    unsigned phase = kSumsPhase0;
    int bx, by;
    view_grouped_block(blockIdx.x, ngx, vc, bx, by);
    proj_sums_block<METHOD, GROUPS>(g, views, xs, ampv, map, proj, out_dtype, view_begin, view_stride, margin,
                                      slots, err, smem_sums + 2, bar, phase, bx, by);
}

// The projector over the flat blocks of many plans (same group count,
// row threads and slots; each task its own geometry and scratch); the mbarriers and their
// phases persist across the items of a block.
template <int METHOD, int GROUPS, bool LOWP>
__global__ void __launch_bounds__(kProjMaxThreads, 3) proj_sums_batch_kernel(const __grid_constant__ ProjBatch b,
                                                                               int slots) {
    extern __shared__ float4 smem_sums_batch[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_sums_batch);
    sums_bars_init(bar);
    unsigned phase = kSumsPhase0;
    for (int blk = blockIdx.x; blk < b.total; blk += gridDim.x) {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b.t[mid].first <= blk) lo = mid; else hi = mid - 1;
        }
        const ProjTask &T = b.t[lo];
        int bx, by;
        view_grouped_block(blk - T.first, T.gx, T.vc, bx, by);
        if (!proj_sums_block<METHOD, GROUPS>(T.g, T.views, T.xs, T.ampv, T.map, T.proj, LOWP ? T.out_dtype : kF32,
                                               T.vb, T.vs, T.margin, slots, T.err, smem_sums_batch + 2, bar, phase,
                                               bx, by))
            return;
        __syncthreads();  // the next item reuses the shared accumulators and tables
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
size_t proj_sums_smem_bytes(int nv, int nx, int ny, int xstride, int groups, int rows, int slots) {
    SumsSmem L{(nv + 3) / 4, rows * groups, std::max(nx, ny), groups, slots, xstride};
    return L.bytes();
}
cudaError_t launch_proj_sums(int method, int groups, int rows, int slots, const Geom &g, const View *views,
                               const float *xs, const float *ampv, const uint8_t *map, void *proj, int out_dtype,
                               int vb, int vs, int vc, float margin, int *err, cudaStream_t st) {
    if (!proj_shape_valid(g.nv, groups, rows) || !proj_slots_valid(g.xstride, slots) ||
        g.xstride % 4 != 0 || g.xstride < g.nz + 2 || reinterpret_cast<uintptr_t>(xs) % 16 != 0)
        return cudaErrorInvalidValue;
    const size_t sm = proj_sums_smem_bytes(g.nv, g.nx, g.ny, g.xstride, groups, rows, slots);
    const int ngx = (g.nu + kTU - 1) / kTU;
    const int nblocks = ngx * vc;
    const int nt = rows * groups;
#define CTSIM_PROJ_SUMS_CASE(M, GR)                                                                 \
    if (method == M && groups == GR) {                                                                \
        cudaError_t e = allow_dynamic_smem((const void *)proj_sums_kernel<M, GR>, sm);              \
        if (e != cudaSuccess) return e;                                                               \
        proj_sums_kernel<M, GR><<<nblocks, nt, sm, st>>>(g, views, xs, ampv, map, proj, out_dtype, vb, vs,    \
                                                           margin, slots, err, ngx, vc);              \
        return cudaGetLastError();                                                                    \
    }
    CTSIM_PROJ_SUMS_CASE(kDD, 1) CTSIM_PROJ_SUMS_CASE(kDD, 2) CTSIM_PROJ_SUMS_CASE(kDD, 4)
    CTSIM_PROJ_SUMS_CASE(kDD, 8) CTSIM_PROJ_SUMS_CASE(kTF, 1) CTSIM_PROJ_SUMS_CASE(kTF, 2)
    CTSIM_PROJ_SUMS_CASE(kTF, 4) CTSIM_PROJ_SUMS_CASE(kTF, 8)
#undef CTSIM_PROJ_SUMS_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_proj_sums_batch(int method, int groups, int row_threads, int slots, bool lowp, size_t smem,
                                     const ProjBatch &b, cudaStream_t st) {
    if (b.n < 1 || b.total < 1) return cudaSuccess;
    const int nt = row_threads * groups;
#define CTSIM_PSB_CASE(M, GR)                                                                         \
    if (method == M && groups == GR) {                                                                \
        auto k = lowp ? proj_sums_batch_kernel<M, GR, true> : proj_sums_batch_kernel<M, GR, false>; \
        cudaError_t e = allow_dynamic_smem((const void *)k, smem);                                    \
        if (e != cudaSuccess) return e;                                                               \
        k<<<persistent_grid((const void *)k, nt, smem, b.total), nt, smem, st>>>(b, slots);                         \
        return cudaGetLastError();                                                                    \
    }
    CTSIM_PSB_CASE(kDD, 1) CTSIM_PSB_CASE(kDD, 2) CTSIM_PSB_CASE(kDD, 4) CTSIM_PSB_CASE(kDD, 8)
    CTSIM_PSB_CASE(kTF, 1) CTSIM_PSB_CASE(kTF, 2) CTSIM_PSB_CASE(kTF, 4) CTSIM_PSB_CASE(kTF, 8)
#undef CTSIM_PSB_CASE
    return cudaErrorInvalidValue;
}

}  // namespace ctsim
