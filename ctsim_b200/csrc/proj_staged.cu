// Forward projector A for sm_100a with the voxel columns staged in shared memory
// (distance-driven and separable-footprint).
//
// One work item per (group of kPart x parts detector columns, view), walked by a persistent
// grid.  A block has three producer warps and four or eight consumer warps around a ring of
// three stages in shared memory; they meet only at the ring, so the producers start the next
// item while the consumers finish the last.
//
// Producers enumerate the candidate voxel columns line by line (lines across the ray
// direction; the projected column centre is monotone along a line, so a line's candidates
// form one interval found by binary search), up to `slots` candidates per stage, one per
// lane.  A lane evaluates its candidate's footprint exactly, writes the candidate's entry
// (axial mapping and column weights) and lets the copy engine bring the whole column -- the
// image transposed to [column][z] with zeros at both ends -- into the stage (cp.async.bulk,
// completion counted in bytes on the stage's "full" mbarrier).  A stage is free again when
// every consumer warp has arrived on its "empty" mbarrier.  A footprint is a long chain of
// exactly rounded divisions (about 4000 cycles from one stage of a warp to its next), hence
// three producers, one per stage of the ring: with one, A waited for it most of the time.
//
// Consumers: the contribution of a column to detector row iv is w_u * ampu * zinc * R(iv),
// where R is the integral of the column over the row's back-projected extent [s, s +
// 1/zinc] in voxels (the axial weights of geom/cbct/cbct_proj.c:382-420 summed over the
// voxels): the overlaps with the TAPS voxels from floor(s) on, each times its voxel.  A lane
// owns single rows, 32 consecutive ones per warp, so that a tap's loads run over consecutive
// words of the staged column.  Rows go in pairs (two 32-row runs, one on each side of the
// row that the volume's middle projects to) with packed FP32 arithmetic, and a stage's
// entries run over the pairs that their shadows reach, in straight-line code for that
// number of pairs.  A warp keeps the sums of its rows over kPart detector columns in
// registers.
//
// What bounds it: instruction issue (58% of the slots) and the waits at the stages' ends.
// Measured on B200 against row threads that kept their sums in shared memory and read prefix
// sums: DD A of 512^2 x 256 and 720 views of 1024 x 384 106.4 -> 63.4 ms; against the
// unstaged projector over paired prefix sums, 128^2 x 64 and 360 views of 256 x 96 2.08 ->
// 0.91 ms.  On the way, 96 of the 720 views: one producer 14.0 ms, four on a ring of four 9.6,
// packed arithmetic through the float2 intrinsics instead of inline assembly (fewer moves) 9.2.
// Rows of more than three voxels on large volumes, and columns too tall for three stages, take
// proj_sums.cu.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"
#include "mbar.cuh"
#include "packed.cuh"

namespace ctsim {

constexpr int kPart = 4;  // detector columns of a consumer warp

// ---------------------------------------------------------------------------
// The column layout: col[ix + iy nx][k], k = 0 .. g.xstride - 1, holds g.xpad zeros, the nz
// voxels, zeros.  A 32 x 32 tile is transposed through shared memory so that the image
// reads and the column writes are coalesced.  state[col]: kColumnOn where the map has the
// column, kColumnNonFinite where a voxel of it is infinite or NaN.
// ---------------------------------------------------------------------------
constexpr int kColumnOn = 1, kColumnNonFinite = 2;

__global__ void __launch_bounds__(256) columns_kernel(const void *__restrict__ image, int in_dtype,
                                                      const uint8_t *__restrict__ map, float *__restrict__ xs,
                                                      uint8_t *__restrict__ state, int nxy, int nz, int xpad,
                                                      int xstride) {
    __shared__ float tile[32][33];
    __shared__ int non_finite[32];
    const int c0 = blockIdx.x * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    bool bad = false;
    if (threadIdx.x < 32) non_finite[threadIdx.x] = 0;
    for (int k0 = 0; k0 < xstride; k0 += 32) {
        for (int kk = ty; kk < 32; kk += 8) {
            const int z = k0 + kk - xpad, c = c0 + tx;
            const float x = (z >= 0 && z < nz && c < nxy) ? load_as_float(image, (size_t)z * nxy + c, in_dtype) : 0.0f;
            tile[kk][tx] = x;
            bad |= !isfinite(x);
        }
        __syncthreads();
        for (int cc = ty; cc < 32; cc += 8) {
            const int c = c0 + cc, k = k0 + tx;
            if (c < nxy && k < xstride) xs[(size_t)c * xstride + k] = tile[tx][cc];
        }
        __syncthreads();
    }
    if (bad) non_finite[tx] = 1;
    __syncthreads();
    if (threadIdx.x < 32 && c0 + tx < nxy)
        state[c0 + tx] = (map[c0 + tx] ? kColumnOn : 0) | (non_finite[tx] ? kColumnNonFinite : 0);
}

cudaError_t launch_columns(const void *image, int in_dtype, const uint8_t *map, float *xs, uint8_t *state, int nxy,
                           int nz, int xpad, int xstride, cudaStream_t st) {
    columns_kernel<<<(nxy + 31) / 32, 256, 0, st>>>(image, in_dtype, map, xs, state, nxy, nz, xpad, xstride);
    return cudaGetLastError();
}

// Two f32x2 values at a 16-byte aligned shared address.
__device__ __forceinline__ void lds_2x2(uint32_t a, f32x2 &x, f32x2 &y) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(y.x), "=f"(y.y) : "r"(a));
}

// The launch shape of a plan: NP row pairs per consumer warp, `warps` warps along the rows,
// `parts` along the columns and `groups` along the candidates (4 or 8 consumer warps), `split`
// blocks along the rows.  The pairs needed are ceil(nv / 64); one warp holds up to six (384
// rows).  More parts share a candidate's footprint and column copy among more columns.
StagedShape staged_shape(int nv, int groups) {
    StagedShape S;
    const int pairs = (nv + 63) / 64;
    S.np = pairs <= 2 ? pairs : pairs <= 4 ? 4 : 6;
    const int need = (pairs + S.np - 1) / S.np;
    S.warps = need >= 2 ? 2 : 1;
    S.groups = S.warps == 2 ? std::min(groups, 2) : std::min(groups, 4);
    S.parts = S.warps == 2 || S.groups == 4 ? 2 : 4;
    S.split = (need + S.warps - 1) / S.warps;
    return S;
}

// Dynamic shared memory: the ring's mbarriers and counts, the stages' columns, the sums of
// the candidate groups, the stages' entries, the line tables.  Laid out for the largest volume
// and the longest columns of a launch: while the producers fill the next item's stages, the
// consumers still read the last one's.
constexpr int kRing = 3, kProducers = 3;
// A producer that filled stage i knows stage i - kRing consumed; the parity it waits for
// before stage i + kProducers tells that stage's slot one phase back from two only if the
// use before the last one, i + kProducers - 2 kRing, is among those.
static_assert(kProducers <= kRing, "a ring shorter than the producers aliases the phases of a slot");
constexpr int kStageLast = 1, kStageNonFinite = 2;
struct StagedRing {
    uint64_t full[kRing], empty[kRing];
    int count[kRing][16];  // entries of (column part, candidate group)
    int pairs[kRing];      // row pairs that the stage's entries reach, counted from the block's first
    int flags[kRing];      // kStageLast: the item's last stage; kStageNonFinite: some column is not finite
    // a producer's or a consumer's wait ran out: read by its own role between two of the role's
    // barriers, where nobody sets it, so that all warps of the role stop at the same item
    int fail_producer, fail_consumer;
};
struct StagedSmem {
    int nlines, slots, xstride, pairs, groups, parts;  // pairs: row pairs of a block
    __host__ __device__ size_t ring_bytes() const { return (sizeof(StagedRing) + 15) & ~(size_t)15; }
    __host__ __device__ size_t column_bytes() const { return (size_t)kRing * slots * xstride * 4; }
    __host__ __device__ size_t sum_bytes() const { return groups > 1 ? (size_t)pairs * parts * kPart * 64 * 4 : 0; }
    __host__ __device__ int entries() const { return slots + groups; }  // of a stage and part
    __host__ __device__ size_t entry_bytes() const { return (size_t)kRing * parts * entries() * 48; }
    __host__ __device__ size_t bytes() const {
        return ring_bytes() + column_bytes() + sum_bytes() + entry_bytes() + (size_t)(2 * nlines + 1 + 32) * 4;
    }
};

// Position in the ring: the next stage and the parity of its "full" phase (its "empty"
// phase before the first use counts as complete: parity ^ 1).
struct RingPos {
    int stage = 0;
    unsigned parity = 0;
    __device__ __forceinline__ void advance(int k) {
        const int q = (stage + k) / kRing;
        stage += k - q * kRing;
        parity ^= (unsigned)q & 1u;
    }
};

// Barriers of the producer warps (1) and of the consumer warps (2).
__device__ __forceinline__ void role_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Candidate intervals of the lines for detector columns [iu0, iu0 + width) of view v:
// line_start[L], and line_off[L] the exclusive scan of the counts (line_off[nlines] =
// the total).  The kProducers producer warps call it; ends with their barrier.
__device__ __forceinline__ int candidate_lines(const Geom &g, const View &v, int iu0, int width, float margin, bool rows,
                                               int *line_start, int *line_off, int *s_warp_tot) {
    constexpr int NT = 32 * kProducers;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nlines = rows ? g.ny : g.nx;
    const int npos = rows ? g.nx : g.ny;
    const float ulo = (float)iu0 - margin, uhi = (float)(iu0 + width) + margin;
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
    role_barrier(1, NT);
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
    role_barrier(1, NT);
    int wbase = 0;
    for (int w = 0; w < warp; w++) wbase += s_warp_tot[w];
    int run = wbase + incl - sum;
    role_barrier(1, NT);
    for (int L = b; L < e; L++) {
        const int c = line_off[L];
        line_off[L] = run;
        run += c;
    }
    if (t == NT - 1) line_off[nlines] = run;
    role_barrier(1, NT);
    return line_off[nlines];
}

// R of the rows f (two per lane) of a staged column.  s + xpad = N sat(pa f + pb) clamps
// the extent's lower edge to [-xpad, nz] at no extra instruction: below and above the
// volume the taps read the zeros of the layout.  xadj: the column's shared-memory address
// minus 4 * 0x4B000000 (mod 2^32), so that the word of voxel floor(s) is at xadj + 4 * bits(s
// + xpad + 2^23 rounded down).  The overlaps are formed from k + 1 - s (one rounding) and
// the extent's length dl = 1 / zinc, so they stay accurate far up the column.  SAFE: a voxel
// that the extent does not reach counts as 0 whatever its value (an infinity times overlap 0
// would be NaN).
template <int TAPS, bool SAFE>
__device__ __forceinline__ f32x2 staged_rows(uint32_t xadj, f32x2 f, float pa, float pb, float dl, float n, int taps) {
    using P = Packed<f32x2>;
    const f32x2 s01 = P::make([&](int i) { return __saturatef(__fmaf_rn(P::get(f, i), pa, pb)); });
    const f32x2 t = pfma_rd(s01, P::all(n), P::all(kTwo23));
    f32x2 a = pfma(s01, P::all(-n), psub(t, P::all(kTwo23 - 1.0f)));  // k + 1 - s
    a = P::make([&](int i) { return fminf(P::get(a, i), dl); });
    uint32_t ad[2];
#pragma unroll
    for (int i = 0; i < 2; i++) ad[i] = xadj + (__float_as_uint(P::get(t, i)) << 2);
    auto tap = [&](int k, f32x2 overlap) {
        return P::make([&](int i) {
            const float x = lds_f32(ad[i] + 4u * k);
            return !SAFE || P::get(overlap, i) > 0.0f ? x : 0.0f;
        });
    };
    f32x2 rem = psub(P::all(dl), a);
    if (TAPS == 2) return pfma(rem, tap(1, rem), pmul(a, tap(0, a)));
    if (TAPS == 3) {
        const f32x2 b = P::make([&](int i) { return fminf(P::get(rem, i), 1.0f); });
        rem = psub(rem, b);
        return pfma(rem, tap(2, rem), pfma(b, tap(1, b), pmul(a, tap(0, a))));
    }
    f32x2 r = pmul(a, tap(0, a));
    for (int k = 1; k < taps; k++) {  // extents of two voxels and more
        const f32x2 b = P::make([&](int i) { return fminf(P::get(rem, i), 1.0f); });
        r = pfma(b, tap(k, b), r);
        rem = psub(rem, b);
    }
    return r;
}

// The entries at shared addresses e, e + step, ... < end over the first NA of the warp's
// row pairs, added with the weights of the warp's kPart detector columns (-0 where the
// footprint does not reach: SAFE adds nothing there).
template <int NP, int NA, int TAPS, bool SAFE = false>
__device__ __forceinline__ void staged_entries(f32x2 (&acc)[kPart][NP], const f32x2 (&frow)[NP], uint32_t e,
                                               uint32_t end, uint32_t step, float n, int taps) {
    float4 next = lds_f32x4(e);
    for (; e < end; e += step) {
        const float4 prm = next;
        next = lds_f32x4(e + step);  // the loads of the next entry's rows wait for it (past the last: unused)
        f32x2 r[NA], w[kPart];
        lds_2x2(e + 16u, w[0], w[1]);
        lds_2x2(e + 32u, w[2], w[3]);
        if constexpr (SAFE) {  // pair by pair: rare, and no more registers than the others
#pragma unroll
            for (int p = 0; p < NA; p++) {
                const f32x2 v = staged_rows<TAPS, true>(__float_as_uint(prm.w), frow[p], prm.x, prm.y, prm.z, n, taps);
#pragma unroll
                for (int j = 0; j < kPart; j++)
                    if (__float_as_uint(w[j].x) != 0x80000000u) acc[j][p] = pfma(w[j], v, acc[j][p]);
            }
            continue;
        }
#pragma unroll
        for (int p = 0; p < NA; p++)
            r[p] = staged_rows<TAPS, false>(__float_as_uint(prm.w), frow[p], prm.x, prm.y, prm.z, n, taps);
#pragma unroll
        for (int p = 0; p < NA; p++)
#pragma unroll
            for (int j = 0; j < kPart; j++) acc[j][p] = pfma(w[j], r[p], acc[j][p]);
    }
}

// u weights of detector columns c0 .. c0 + kPart - 1 (footprint scaled by scl): u_weight of
// common.cuh, with a trapezoid's two divisions replaced by r0 and r1 (half the reciprocals
// of its ramps) and its squares' differences formed as (a - b)(a + b); -0 off the footprint.
template <int METHOD>
__device__ __forceinline__ void staged_weights(const ColumnFP &fp, float scl, float r0, float r1, int c0,
                                               float (&w)[kPart]) {
#pragma unroll
    for (int j = 0; j < kPart; j++) {
        float v;
        if (METHOD == kDD) {
            v = u_weight<kDD>(c0 + j, fp.iumin, fp.iumax, fp.p0, fp.p1, 0.f, 0.f);
        } else {
            const float bl = (float)(c0 + j) - 0.5f, br = bl + 1.0f;
            float xl = fmaxf(bl, fp.p0), xr = fminf(br, fp.p1);
            v = xr > xl ? ((xr - xl) * ((xr - fp.p0) + (xl - fp.p0))) * r0 : 0.0f;
            v += fmaxf(fminf(br, fp.p2) - fmaxf(bl, fp.p1), 0.0f);
            xl = fmaxf(bl, fp.p2);
            xr = fminf(br, fp.p3);
            v += xr > xl ? ((xr - xl) * ((fp.p3 - xl) + (fp.p3 - xr))) * r1 : 0.0f;
        }
        w[j] = c0 + j >= fp.iumin && c0 + j <= fp.iumax ? v * scl : -0.0f;
    }
}

// One work item: detector columns from bx kPart parts on of launch view by, row pairs from
// bz PB on (PB: row pairs of a block).
struct StagedItem {
    const ColumnsGeom *g;
    const View *views;
    const float *xs, *ampv;
    const uint8_t *state;  // of the columns (columns_kernel)
    void *proj;
    int *err;
    int out_dtype, view_begin, view_stride, bx, by, bz;
    float margin;
};

// What both roles derive from an item.
struct StagedView {
    View v;
    int iu0, mid, Q0;
    float n;  // nz + xpad: the clamped range of s + xpad
    // the row that the volume's middle projects to (at the rotation axis) splits the rows:
    // pair q covers rows [mid - 32 (q + 1), mid - 32 q) and [mid + 32 q, mid + 32 (q + 1)); all
    // pairs together cover the detector wherever mid is clamped to
    __device__ __forceinline__ StagedView(const StagedItem &I, int parts, int PB) {
        const ColumnsGeom &g = *I.g;
        v = I.views[I.view_begin + I.by * I.view_stride];
        iu0 = I.bx * kPart * parts;
        const int half = 32 * ((g.nv + 63) / 64);
        const float zc = (v.wz + 0.5f * (float)(g.nz - 1)) * (g.dz_dv * g.sdd / g.sad) - g.wv + 0.5f;
        mid = max(g.nv - half, min(half, (int)rintf(fminf(fmaxf(zc, -1e6f), 1e6f))));
        Q0 = I.bz * PB;
        n = (float)(g.nz + g.xpad);
    }
};

// Producers: stage i of the item is filled by producer i mod kProducers.  at: the ring
// position of the item's first stage, left at the next item's.  False: a wait of an
// earlier item ran out.
template <int METHOD>
__device__ __forceinline__ bool staged_produce(const StagedItem &I, const StagedSmem &L, StagedRing *ring, RingPos &at,
                                               int PB) {
    const ColumnsGeom &g = *I.g;
    char *smem = reinterpret_cast<char *>(ring) + L.ring_bytes();
    float *columns = reinterpret_cast<float *>(smem);  // [kRing][slots][xstride]
    char *entries = smem + L.column_bytes() + L.sum_bytes();
    int *line_start = reinterpret_cast<int *>(entries + L.entry_bytes());
    int *line_off = line_start + L.nlines;
    int *s_warp_tot = line_off + L.nlines + 1;  // [32]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xst = g.xstride, nv = g.nv, groups = L.groups;
    const int width = kPart * L.parts;
    const StagedView V(I, L.parts, PB);
    const View v = V.v;
    const int iu0 = V.iu0, mid = V.mid;
    const bool rows = fabsf(v.cos_a) >= fabsf(v.sin_a);
    const int nlines = rows ? g.ny : g.nx;
    role_barrier(1, 32 * kProducers);
    const bool stop = ring->fail_producer != 0;
    const int ncand = candidate_lines(g, v, iu0, width, I.margin, rows, line_start, line_off, s_warp_tot);
    if (stop) return false;
    const int per = min(L.slots, 32);  // candidates per stage
    const int nstages = max(1, (ncand + per - 1) / per);
    RingPos my = at;
    my.advance(warp);
    at.advance(nstages);
    const double rn = 1.0 / (double)V.n;
    int out_stage = -1;  // the last stage this producer filled
    unsigned out_parity = 0;
    for (int i = warp; i < nstages; i += kProducers, my.advance(kProducers)) {
        const int c = i * per + lane;
        bool valid = false, non_finite = false;
        int na = 0, col = 0, h0 = 1, h1 = 0;  // the parts the footprint touches
        float pa = 0.f, pb = 0.f, dl = 0.f, scl = 0.f;
        ColumnFP fp;
        if (lane < per && c < ncand) {
            int a = 0, bnd = nlines - 1;  // last line with line_off <= c
            while (a < bnd) {
                const int m = (a + bnd + 1) >> 1;
                if (line_off[m] <= c) a = m; else bnd = m - 1;
            }
            const int p = line_start[a] + (c - line_off[a]);
            const int ix = rows ? p : a, iy = rows ? a : p;
            col = iy * g.nx + ix;
            const int state = I.state[col];
            const bool on = (state & kColumnOn) != 0;
            fp = column_footprint<METHOD, false>(g, v, ix, iy);
            if (on && fp.hit && fp.iumax >= iu0 && fp.iumin <= iu0 + width - 1) {
                const float b0 = fp.vstart + 0.5f;
                const float btop = fmaf((float)g.nz, fp.zinc, b0);
                const int rlo = max((int)floorf(fminf(b0, 1e6f)) - 1, 0);
                const int rhi = min((int)floorf(fmaxf(btop, -1e6f)) + 1, nv - 1);
                // the block's pairs up to the one that rows rlo .. rhi reach
                na = min(max(rhi - mid, mid - 1 - rlo) / 32 + 1 - V.Q0, PB);
                if (rlo <= rhi && na > 0) {
                    valid = true;
                    non_finite = (state & kColumnNonFinite) != 0;
                    h0 = (max(fp.iumin, iu0) - iu0) / kPart;
                    h1 = (min(fp.iumax, iu0 + width - 1) - iu0) / kPart;
                    scl = fp.ampu * fp.zinc;
                    // lower edge of row iv: s = (iv - b0) / zinc, as sat(pa iv + pb) of [-xpad, nz]; pb
                    // makes it exact at iv = mid (double: 1 / zinc and the offset each rounded once)
                    const double d = 1.0 / (double)fp.zinc;
                    const double sm = ((double)mid - (double)b0) * d + (double)g.xpad;
                    dl = (float)d;
                    pa = (float)(d * rn);
                    pb = (float)(sm * rn - (double)pa * (double)mid);
                }
            }
        }
        const float r0 = METHOD == kTF && valid ? 0.5f / (fp.p1 - fp.p0) : 0.0f;
        const float r1 = METHOD == kTF && valid ? 0.5f / (fp.p3 - fp.p2) : 0.0f;
        const unsigned all = __ballot_sync(kFull, valid);
        const unsigned reach = __reduce_max_sync(kFull, valid ? (unsigned)na : 0u);
        const bool any_non_finite = __any_sync(kFull, non_finite);
        // lanes of this lane's candidate group: (c mod groups) repeats every `groups` lanes
        unsigned same = 1u << (lane & (groups - 1));
        for (int k = groups; k < 32; k <<= 1) same |= same << k;
        const unsigned below = (1u << lane) - 1u;
        const int q = c & (groups - 1);  // groups: a power of two
        unsigned hb[4];                  // this lane's group's candidates of each part
#pragma unroll
        for (int h = 0; h < 4; h++) hb[h] = __ballot_sync(kFull, valid && h >= h0 && h <= h1) & same;
        if (!mbar_wait<100>(&ring->empty[my.stage], my.parity ^ 1u)) {
            if (lane == 0) {
                atomicOr(I.err, kErrStageWait);
                ring->fail_producer = 1;
            }
            // this producer's copies in flight land before it stops (its earlier stages were consumed)
            if (out_stage >= 0) mbar_wait(&ring->full[out_stage], out_parity);
            break;
        }
        float *dst = columns + ((size_t)my.stage * L.slots + __popc(all & below)) * L.xstride;
        const uint32_t xadj = smem_addr(dst) - (0x4B000000u << 2);
#pragma unroll
        for (int h = 0; h < 4; h++)
            if (h < L.parts && lane < groups) ring->count[my.stage][h * 4 + q] = __popc(hb[h]);
        if (valid)
            for (int h = h0; h <= h1; h++) {
                float w[kPart];
                staged_weights<METHOD>(fp, scl, r0, r1, iu0 + h * kPart, w);
                const unsigned b = h == 0 ? hb[0] : h == 1 ? hb[1] : h == 2 ? hb[2] : hb[3];
                const int k = __popc(b & below) * groups + q;
                float4 *e = reinterpret_cast<float4 *>(entries + ((size_t)(my.stage * L.parts + h) * L.entries() + k) * 48);
                e[0] = make_float4(pa, pb, dl, __uint_as_float(xadj));
                e[1] = make_float4(w[0], w[0], w[1], w[1]);
                e[2] = make_float4(w[2], w[2], w[3], w[3]);
            }
        if (lane == 0) {
            ring->pairs[my.stage] = (int)reach;
            ring->flags[my.stage] = (i == nstages - 1 ? kStageLast : 0) | (any_non_finite ? kStageNonFinite : 0);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_expect(&ring->full[my.stage], (unsigned)__popc(all) * (unsigned)xst * 4u);
        __syncwarp();
        if (valid) bulk_copy_g2s(dst, I.xs + (size_t)col * xst, (unsigned)xst * 4u, &ring->full[my.stage]);
        out_stage = my.stage;
        out_parity = my.parity;
    }
    return true;
}

// Consumers: the item's sums and its store.  A row's value depends neither on which lane or
// warp evaluates it nor on the launch shape: its extent is a function of the row and the
// candidate alone, and candidate group q takes the candidates whose number in the item's
// sequence is q mod groups, in order.  False: a wait ran out.
template <int NP, int TAPS>
__device__ __forceinline__ bool staged_consume(const StagedItem &I, const StagedSmem &L, StagedRing *ring, RingPos &at,
                                               int wg, int consumers) {
    const ColumnsGeom &g = *I.g;
    char *smem = reinterpret_cast<char *>(ring) + L.ring_bytes();
    float *sum = reinterpret_cast<float *>(smem + L.column_bytes());  // [columns][pairs][2][32]
    // [kRing][parts][entries]: {pa, pb, 1 / zinc, column address}, four weights, each twice
    // (a packed operand); entry k of candidate group q is at k * groups + q
    char *entries = smem + L.column_bytes() + L.sum_bytes();
    const int t = threadIdx.x - 128, lane = t & 31, warp = t >> 5;
    const int groups = L.groups, PB = L.pairs, nv = g.nv;
    // candidate group grp, column part, row pairs Q0 + gwarp + i wg
    const int gwarp = wg == 2 ? warp & 1 : 0, part = (wg == 2 ? warp >> 1 : warp) & (L.parts - 1);
    const int grp = warp / (wg * L.parts);
    const StagedView V(I, L.parts, PB);
    const int mid = V.mid, Q0 = V.Q0;
    const float n = V.n;
    const int taps = g.taps;
    f32x2 acc[kPart][NP], frow[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int q = Q0 + gwarp + p * wg;
        frow[p] = pack2((float)(mid - 32 * (q + 1) + lane), (float)(mid + 32 * q + lane));
#pragma unroll
        for (int j = 0; j < kPart; j++) acc[j][p] = pack2(0.0f, 0.0f);
    }
    const uint32_t ent = smem_addr(entries) + 48u * (uint32_t)(part * L.entries() + grp);
    const uint32_t ent_stage = 48u * (uint32_t)(L.parts * L.entries()), step = 48u * (uint32_t)groups;
    bool last = false;
    while (!last) {
        if (!mbar_wait(&ring->full[at.stage], at.parity)) {
            if (lane == 0) {
                atomicOr(I.err, kErrStageWait);
                ring->fail_consumer = 1;
            }
            break;
        }
        const int count = ring->count[at.stage][part * 4 + grp];
        const int na = wg == 1 ? ring->pairs[at.stage] : (ring->pairs[at.stage] - gwarp + 1) >> 1;  // wg: 1 or 2
        const int flags = ring->flags[at.stage];
        last = (flags & kStageLast) != 0;
        if (count > 0 && na > 0) {
            const uint32_t e = ent + (uint32_t)at.stage * ent_stage, end = e + (uint32_t)count * step;
            // A stage with a non-finite column: pairs that it does not reach add zeros.  With up to four
            // pairs per warp the test stands before the switch, with six it is a case of it (registers:
            // DD A of 128^2 x 64 0.917 and 0.925 ms, of 512^2 x 256 64.3 and 63.4 ms).
            const bool safe = (flags & kStageNonFinite) != 0;
            if (NP < 6 && safe) {
                staged_entries<NP, NP, TAPS, true>(acc, frow, e, end, step, n, taps);
            } else switch (NP == 6 && safe ? 0 : na) {
            case 0:
                if constexpr (NP == 6) staged_entries<NP, NP, TAPS, true>(acc, frow, e, end, step, n, taps);
                break;
            case 1: staged_entries<NP, 1, TAPS>(acc, frow, e, end, step, n, taps); break;
            case 2: staged_entries<NP, NP < 2 ? NP : 2, TAPS>(acc, frow, e, end, step, n, taps); break;
            case 3: staged_entries<NP, NP < 3 ? NP : 3, TAPS>(acc, frow, e, end, step, n, taps); break;
            case 4: staged_entries<NP, NP < 4 ? NP : 4, TAPS>(acc, frow, e, end, step, n, taps); break;
            case 5: staged_entries<NP, NP < 5 ? NP : 5, TAPS>(acc, frow, e, end, step, n, taps); break;
            default: staged_entries<NP, NP, TAPS>(acc, frow, e, end, step, n, taps); break;
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ring->empty[at.stage]);
        at.advance(1);
    }
    const size_t obase = (size_t)I.by * g.nu * nv;
    auto store = [&](int j, int q, int h, float v) {  // column j of the item, half h of pair q, this lane's row
        const int iu = V.iu0 + j, iv = (h ? mid + 32 * q : mid - 32 * (q + 1)) + lane;
        if (iu < g.nu && iv >= 0 && iv < nv)
            store_from_float(I.proj, obase + (size_t)iu * nv + iv, v * I.ampv[(size_t)iu * nv + iv], I.out_dtype);
    };
    if (groups == 1) {
        role_barrier(2, consumers);
        const bool stop = ring->fail_consumer != 0;
        role_barrier(2, consumers);
        if (stop) return false;
#pragma unroll
        for (int p = 0; p < NP; p++)
#pragma unroll
            for (int j = 0; j < kPart; j++) {
                float lo, hi;
                unpack2(acc[j][p], lo, hi);
                store(part * kPart + j, Q0 + gwarp + p * wg, 0, lo);
                store(part * kPart + j, Q0 + gwarp + p * wg, 1, hi);
            }
        return true;
    }
    // the groups' sums in group order
    for (int gi = 0; gi < groups; gi++) {
        if (grp == gi)
#pragma unroll
            for (int p = 0; p < NP; p++)
#pragma unroll
                for (int j = 0; j < kPart; j++) {
                    float lo, hi;
                    unpack2(acc[j][p], lo, hi);
                    float *d = sum + (((part * kPart + j) * PB + gwarp + p * wg) * 2) * 32 + lane;
                    d[0] = gi ? d[0] + lo : lo;
                    d[32] = gi ? d[32] + hi : hi;
                }
        role_barrier(2, consumers);
    }
    if (ring->fail_consumer) return false;
    for (int r = warp; r < kPart * L.parts * PB * 2; r += consumers >> 5) {  // 32-row runs
        const int j = r / (2 * PB), o = r - j * 2 * PB;
        store(j, Q0 + (o >> 1), o & 1, sum[r * 32 + lane]);
    }
    role_barrier(2, consumers);  // the next item's sums overwrite this one's
    return true;
}

// Registers per thread: at launch, of a producer and of a consumer (setmaxnreg; per block
// 128 threads in the producers' place, the last warp of them idle, and 128 CW consumer threads, whose shares add up to the launch's at most).
// Two pairs and fewer need no split.
template <int NP, int CW>
struct StagedRegs {
    static constexpr int kLaunch = NP <= 2 ? 64 : 80, kProducer = 56, kConsumer = CW == 1 ? 104 : 88;
    static_assert(128 * (kProducer + CW * kConsumer) <= 128 * (1 + CW) * kLaunch || NP <= 2, "register split");
};

// xstride: the columns' stride in the stages, the same for all items (0: the only plan's own).
template <int METHOD, int NP, int CW, int TAPS, class ITEM>
__device__ __forceinline__ void staged_block(int total, int groups, int parts, int slots, int xstride, int nlines,
                                             ITEM item) {
    extern __shared__ float4 smem_staged[];
    StagedRing *ring = reinterpret_cast<StagedRing *>(smem_staged);
    constexpr int consumers = 128 * CW;
    const int wg = (consumers >> 5) / (groups * parts);  // consumer warps along the rows: 1 or 2
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRing; i++) {
            mbar_init(&ring->full[i], 1);
            mbar_init(&ring->empty[i], consumers >> 5);
        }
        ring->fail_producer = ring->fail_consumer = 0;
        mbar_init_fence();
    }
    __syncthreads();
    StagedSmem L{nlines, slots, 0, wg * NP, groups, parts};
    RingPos at;
    // the first four warps are the producers' place (registers are shared out four warps at a time)
    if (threadIdx.x < 128) {
        if constexpr (NP > 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(StagedRegs<NP, CW>::kProducer));
        if (threadIdx.x >= 32 * kProducers) return;
        for (int blk = blockIdx.x; blk < total; blk += gridDim.x) {
            const StagedItem I = item(blk);
            L.xstride = xstride ? xstride : I.g->xstride;
            if (!staged_produce<METHOD>(I, L, ring, at, wg * NP)) return;
        }
    } else {
        if constexpr (NP > 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(StagedRegs<NP, CW>::kConsumer));
        for (int blk = blockIdx.x; blk < total; blk += gridDim.x) {
            const StagedItem I = item(blk);
            L.xstride = xstride ? xstride : I.g->xstride;
            if (!staged_consume<NP, TAPS>(I, L, ring, at, wg, consumers)) return;
        }
    }
}

template <int METHOD, int NP, int CW, int TAPS>
__global__ void __launch_bounds__(128 * (1 + CW), 65536 / (128 * (1 + CW) * StagedRegs<NP, CW>::kLaunch))
    proj_staged_kernel(const __grid_constant__ ColumnsGeom g, const View *__restrict__ views,
                       const float *__restrict__ xs, const float *__restrict__ ampv,
                       const uint8_t *__restrict__ state, void *__restrict__ proj,
                       int out_dtype, int view_begin, int view_stride, float margin, int groups, int parts,
                       int slots, int *__restrict__ err, int ngx, int vc, int total) {
    staged_block<METHOD, NP, CW, TAPS>(total, groups, parts, slots, 0, max(g.nx, g.ny), [&](int blk) {
        StagedItem I{&g, views, xs, ampv, state, proj, err, out_dtype, view_begin, view_stride, 0, 0, 0, margin};
        const int per = ngx * vc;
        I.bz = blk / per;
        view_grouped_block(blk - I.bz * per, ngx, vc, I.bx, I.by);
        return I;
    });
}

// The staged forward projector over the items of many plans of one launch shape and TAPS (each
// task its own geometry, scratch and storage type).  xstride, nlines: the longest columns' and
// the largest volume's.
template <int METHOD, int NP, int CW, int TAPS>
__global__ void __launch_bounds__(128 * (1 + CW), 65536 / (128 * (1 + CW) * StagedRegs<NP, CW>::kLaunch))
    proj_staged_batch_kernel(const __grid_constant__ ProjBatch b, int groups, int parts, int slots, int xstride,
                             int nlines) {
    staged_block<METHOD, NP, CW, TAPS>(b.total, groups, parts, slots, xstride, nlines, [&](int blk) {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (b.t[m].first <= blk) lo = m; else hi = m - 1;
        }
        const ProjTask &T = b.t[lo];
        StagedItem I{&T.g, T.views, T.xs, T.ampv, T.state, T.proj, T.err, T.out_dtype, T.vb, T.vs, 0, 0, 0, T.margin};
        const int per = T.gx * T.vc, l = blk - T.first;
        I.bz = l / per;
        view_grouped_block(l - I.bz * per, T.gx, T.vc, I.bx, I.by);
        return I;
    });
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
// Work items along the detector columns.
int staged_columns(const StagedShape &S, int nu) { return (nu + kPart * S.parts - 1) / (kPart * S.parts); }
size_t proj_staged_smem_bytes(const StagedShape &S, int nlines, int xstride, int slots) {
    StagedSmem L{nlines, slots, xstride, S.warps * S.np, S.groups, S.parts};
    return L.bytes();
}
size_t proj_staged_smem_bytes(int nv, int nlines, int xstride, int groups, int slots) {
    return proj_staged_smem_bytes(staged_shape(nv, groups), nlines, xstride, slots);
}
// Slots per stage: 1 .. 64 (at most 32 are used), and their bytes within an mbarrier phase's
// transaction count (< 2^20).
bool proj_slots_valid(int xstride, int slots) {
    return slots >= 1 && slots <= 64 && (size_t)slots * xstride * 4 < (1u << 20);
}

#define CTSIM_STAGED_SWITCH(KERNEL, CALL)                                        \
    do {                                                                         \
        CTSIM_STAGED_NP(KERNEL, kDD, CALL) CTSIM_STAGED_NP(KERNEL, kTF, CALL)    \
    } while (0)
#define CTSIM_STAGED_NP(KERNEL, M, CALL)                                         \
    CTSIM_STAGED_CW(KERNEL, M, 1, CALL) CTSIM_STAGED_CW(KERNEL, M, 2, CALL)      \
    CTSIM_STAGED_CW(KERNEL, M, 4, CALL) CTSIM_STAGED_CW(KERNEL, M, 6, CALL)
#define CTSIM_STAGED_CW(KERNEL, M, N, CALL)                                      \
    CTSIM_STAGED_TAPS(KERNEL, M, N, 1, CALL) CTSIM_STAGED_TAPS(KERNEL, M, N, 2, CALL)
#define CTSIM_STAGED_TAPS(KERNEL, M, N, C, CALL)                                 \
    CTSIM_STAGED_ONE(KERNEL, M, N, C, 2, CALL) CTSIM_STAGED_ONE(KERNEL, M, N, C, 3, CALL) \
    CTSIM_STAGED_ONE(KERNEL, M, N, C, 0, CALL)
#define CTSIM_STAGED_ONE(KERNEL, M, N, C, T, CALL)                               \
    if (method == M && S.np == N && S.warps * S.groups * S.parts == 4 * C && (taps <= 3 ? taps : 0) == T) { \
        auto k = KERNEL<M, N, C, T>;                                             \
        cudaError_t e = allow_dynamic_smem((const void *)k, sm);                 \
        if (e != cudaSuccess) return e;                                          \
        constexpr int nt = 128 * (1 + C);                                        \
        CALL;                                                                    \
        return cudaGetLastError();                                               \
    }

cudaError_t launch_proj_staged(int method, int groups, int slots, const ColumnsGeom &g, const View *views,
                               const float *xs, const float *ampv, const uint8_t *state, void *proj, int out_dtype,
                               int vb, int vs, int vc, float margin, int *err, cudaStream_t st) {
    if ((groups != 1 && groups != 2 && groups != 4 && groups != 8) || !proj_slots_valid(g.xstride, slots) ||
        g.xstride % 4 != 0 || g.xpad < 1 || g.taps < 2 || g.xstride < g.nz + g.xpad + g.taps ||
        reinterpret_cast<uintptr_t>(xs) % 16 != 0)
        return cudaErrorInvalidValue;
    const StagedShape S = staged_shape(g.nv, groups);
    const size_t sm = proj_staged_smem_bytes(g.nv, std::max(g.nx, g.ny), g.xstride, groups, slots);
    const int ngx = staged_columns(S, g.nu), taps = g.taps, total = ngx * vc * S.split;
    CTSIM_STAGED_SWITCH(proj_staged_kernel,
                        (k<<<persistent_grid((const void *)k, nt, sm, total), nt, sm, st>>>(
                            g, views, xs, ampv, state, proj, out_dtype, vb, vs, margin, S.groups, S.parts, slots, err, ngx,
                            vc, total)));
    return cudaErrorInvalidValue;
}

cudaError_t launch_proj_staged_batch(int method, const StagedShape &S, int taps, int slots, int xstride, int nlines,
                                     size_t sm, const ProjBatch &b, cudaStream_t st) {
    if (b.n < 1 || b.total < 1) return cudaSuccess;
    CTSIM_STAGED_SWITCH(proj_staged_batch_kernel, (k<<<persistent_grid((const void *)k, nt, sm, b.total), nt, sm, st>>>(
                                                      b, S.groups, S.parts, slots, xstride, nlines)));
    return cudaErrorInvalidValue;
}

}  // namespace ctsim
