// Projector kernels for sm_100a.
//
//   prefix_kernel            per-column axial prefix sums of the volume (input of A)
//   proj_kernel<METHOD>      forward projection A
//
// The staged forward projector is in proj_staged.cu, the matched backprojection in back.cu,
// the voxel-driven FDK backprojection in pd.cu.
//
// Layouts (reference MEX conventions): image[iz][iy][ix], proj[view][iu][iv].
#include "kernels.cuh"

#include <map>
#include <mutex>
#include <tuple>
#include <utility>

namespace ctsim {

constexpr unsigned kFull = 0xffffffffu;

// ps = proj * ampv (the axial amplitude the reference applies to the backprojected
// view in place, geom/cbct/cbct_back.c:196-214), into scratch.
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
//   does not stay cache-resident; measured on B200 at 512^2 x 256), columns xstride
//   (column_stride) floats apart, with X[nz] repeated above X[nz] up to the stride.
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

cudaError_t launch_prescale(const void *proj, int in_dtype, const float *ampv, float *ps, size_t nuv, size_t n,
                            cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 32);
    prescale_kernel<<<blocks, 256, 0, st>>>(proj, in_dtype, ampv, ps, nuv, n);
    return cudaGetLastError();
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

int proj_row_threads_of(int nv) { return proj_row_threads(nv); }

// The resident blocks of a kernel's launch shape are asked for once per device: the staged forward
// projector needs them at every launch, twelve times per OS-SQS iteration of twelve subsets.
int persistent_grid(const void *kernel, int threads, size_t smem, int total) {
    static std::mutex m;
    static std::map<std::tuple<int, const void *, int, size_t>, int> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    std::lock_guard<std::mutex> lock(m);
    int &resident = known[{dev, kernel, threads, smem}];
    if (resident == 0) {
        int sms = 148, per_sm = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        resident = sms * per_sm;
    }
    return std::max(1, std::min(total, resident));
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

}  // namespace ctsim
