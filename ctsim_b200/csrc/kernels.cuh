// Launcher declarations for the projector kernels (kernels.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace ctsim {

// Detector columns per block of the forward projector.
constexpr int kProjGroupWidth = 8;

// Views per group of the forward projector's launch order.
constexpr int kViewGroup = 32;

// Detector-column group bx and launch view by of the forward projector's linear block
// L: the launch views in groups of kViewGroup consecutive ones (the last group may be
// shorter), and within a group the blocks of one detector-column group over all its
// views, then the next column group -- neighbouring views share candidate columns in L2.
__device__ __forceinline__ void view_grouped_block(int L, int ngx, int vc, int &bx, int &by) {
    const int per = ngx * kViewGroup;
    const int G = L / per, r = L - G * per;
    const int n = min(kViewGroup, vc - G * kViewGroup);  // views of this group
    bx = r / n;
    by = G * kViewGroup + (r - bx * n);
}

// ps = proj (any storage type) * ampv (ampv may be null: plain conversion to FP32)
cudaError_t launch_prescale(const void *proj, int in_dtype, const float *ampv, float *ps, size_t nuv, size_t n,
                            cudaStream_t st);

// Sinogram sources of the backprojector: FP32 already multiplied by the axial amplitude
// ampv (a pre-scaled copy, or a residual written that way), or the stored sinogram in
// FP32, BF16 or FP16, multiplied by ampv as it is read.  launch_back and the batches take
// kSrcScaled, kSrcBF16 and kSrcF16 (kSrcF32 serves the entry point without allocations).
enum BackSrc { kSrcScaled = 0, kSrcF32 = 1, kSrcBF16 = 2, kSrcF16 = 3 };
cudaError_t launch_back(int method, int mz, const Geom &g, const View *views, const void *ps, const uint8_t *map,
                        void *image, int out_dtype, int view_begin, int view_stride, int view_count, float scale,
                        int qcap, int *err, cudaStream_t st, bool accumulate = false, int y_begin = 0,
                        int y_end = -1, int src = kSrcScaled, const float *ampv = nullptr);
size_t back_smem_bytes(int qcap);
cudaError_t launch_back_unscaled(int mz, const Geom &g, const View *views, const float *proj, const float *ampv,
                                 const uint8_t *map, float *image, int view_count, int qcap, int *err,
                                 cudaStream_t st);

// pairs: the (X, slope) layout of the column prefix sums (forward_pairs below)
cudaError_t launch_prefix(const void *image, int in_dtype, float *xs, int nxy, int nz, bool pairs, int xstride,
                          cudaStream_t st);

cudaError_t launch_proj(int method, int groups, int rows, bool pairs, const Geom &g, const View *views,
                        const float *xs, const float *ampv, const uint8_t *map, void *proj, int out_dtype,
                        int view_begin, int view_stride, int view_count, float margin, cudaStream_t st);
// The paired prefix layout when it is small enough to stay cache-resident (<= 160 MB).
inline bool forward_pairs(long long nxy, int nz) { return 8LL * nxy * (nz + 1) <= 160LL * 1024 * 1024; }
int proj_default_groups(int nv);
int proj_default_rows(int nv);
bool proj_groups_valid(int nv, int groups);
bool proj_shape_valid(int nv, int groups, int rows);
size_t proj_smem_bytes(int nv, int nx, int ny, int groups, int rows);
// The forward projector with the candidates' voxel columns staged in shared memory
// (proj_staged.cu): xs holds the image as columns (launch_columns; 16-byte aligned),
// up to `slots` of them per stage; candidate groups 1, 2, 4 or 8.  state: one byte per column,
// its place in the map and whether its voxels are finite.  A stage wait that runs out sets bit 4
// of *err.
cudaError_t launch_columns(const void *image, int in_dtype, const uint8_t *map, float *xs, uint8_t *state, int nxy,
                           int nz, int xpad, int xstride, cudaStream_t st);
cudaError_t launch_proj_staged(int method, int groups, int slots, const ColumnsGeom &g, const View *views,
                               const float *xs, const float *ampv, const uint8_t *state, void *proj, int out_dtype,
                               int view_begin, int view_stride, int view_count, float margin, int *err,
                               cudaStream_t st);
size_t proj_staged_smem_bytes(int nv, int nlines, int xstride, int groups, int slots);
bool proj_slots_valid(int xstride, int slots);
// Row pairs per consumer warp; consumer warps along the rows, the columns and the
// candidates; blocks along the rows.
struct StagedShape {
    int np, warps, parts, groups, split;
};
StagedShape staged_shape(int nv, int groups);
int staged_columns(const StagedShape &shape, int nu);

// The same with the candidates' prefix columns (launch_prefix, single sums) staged in two
// buffers of `slots` columns (proj_sums.cu); groups and rows as launch_proj.
cudaError_t launch_proj_sums(int method, int groups, int rows, int slots, const Geom &g, const View *views,
                             const float *xs, const float *ampv, const uint8_t *map, void *proj, int out_dtype,
                             int view_begin, int view_stride, int view_count, float margin, int *err, cudaStream_t st);
size_t proj_sums_smem_bytes(int nv, int nx, int ny, int xstride, int groups, int rows, int slots);

// voxel-driven bilinear modes: back,pd (v outside the detector skipped), back,hpd (v
// clamped), back,var (geom/cbct/cbct_back_var.c)
enum PdMode { kPdOff = 0, kPdClamp = 1, kPdVar = 2 };
// proj in storage type in_dtype (kF32, kBF16, kF16), read as it is; the image is
// (sum * scale) * scale2.
cudaError_t launch_pd(int mode, int mz, const Geom &g, const View *views, const void *proj,
                      const uint8_t *map, void *image, int out_dtype, int view_begin, int view_stride,
                      int view_count, float scale, cudaStream_t st, bool accumulate = false, int in_dtype = kF32,
                      float scale2 = 1.0f);

// ---------------------------------------------------------------------------
// Batched launches: the blocks of many plans' A (or A^T) in one persistent grid.
// ---------------------------------------------------------------------------
constexpr int kBatchMax = 64;  // tasks per launch (the task table travels as a kernel parameter)

struct ProjTask {
    ColumnsGeom g;
    const View *views;
    const float *xs;
    const float *ampv;
    const uint8_t *map, *state;  // state: the staged projector's columns
    void *proj;
    int out_dtype;
    int vb, vs, vc, gx, first;  // view selection, blocks along u, first flat block of the task
    float margin;
    int *err;               // the plan's error flag (staged projector: a stage wait that ran out)
};
struct ProjBatch {
    int n, total;  // tasks, flat blocks of all tasks
    ProjTask t[kBatchMax];
};

struct BackTask {
    Geom g;
    const View *views;
    const void *ps;         // the class's source form (BackSrc)
    const float *ampv;      // the plan's axial amplitudes (unscaled sources)
    const uint8_t *map;
    void *image;
    int out_dtype;
    int *err;
    int vb, vs, vc, qcap, first;
    float scale;
};
struct BackBatch {
    int n, total;
    BackTask t[kBatchMax];
};

// The flat blocks of an A^T task (rows x column tiles).
int back_task_blocks(const Geom &g);
int proj_row_threads_of(int nv);
// lowp: some task stores BF16/FP16 (each task's out_dtype); otherwise all store FP32
cudaError_t launch_proj_batch(int method, int groups, int row_threads, bool pairs, bool lowp, size_t smem,
                              const ProjBatch &b, cudaStream_t st);
cudaError_t launch_back_batch(int method, int mz, bool vec, bool lowp, size_t smem, const BackBatch &b,
                              cudaStream_t st, int src = kSrcScaled);
// The staged forward projector (launch_proj_staged) over a batch of plans of one shape (and, up to
// three, of one `taps`); xstride and nlines: the largest column stride and max(nx, ny).
size_t proj_staged_smem_bytes(const StagedShape &shape, int nlines, int xstride, int slots);
cudaError_t launch_proj_staged_batch(int method, const StagedShape &shape, int taps, int slots, int xstride, int nlines,
                                     size_t smem, const ProjBatch &b, cudaStream_t st);
// proj_sums.cu over a batch of plans of one group count, row threads and slots.
cudaError_t launch_proj_sums_batch(int method, int groups, int row_threads, int slots, bool lowp, size_t smem,
                                   const ProjBatch &b, cudaStream_t st);
// Blocks of a persistent launch: the resident blocks of the device, at most `total`.
int persistent_grid(const void *kernel, int threads, size_t smem, int total);

// Raises (never lowers) a kernel's dynamic shared-memory limit on the current device.
cudaError_t allow_dynamic_smem(const void *kfn, size_t bytes);

size_t proj_smem_bytes(int nv, int nx, int ny, int groups);
int proj_max_lines();

}  // namespace ctsim
