// Host-side launchers of the time-step kernels (internal to the library).
#pragma once
#include <cuda_runtime.h>

#include "mfdm_device.cuh"

namespace mfdm {

// Launches RK stage `stage` (0..3) with operator direction `dir` (0 = F, 1 = B).
// Stage 0 reads `in` == U^n; stages 1-2 read `in` and U^n (`un`); stage 3 writes
// U, filters its interface rows and samples the receivers.
cudaError_t launch_stage(const Coef& C, const Fields& in, const Fields& out, const Fields& un,
                         const Fields& acc, int stage, int dir, cudaStream_t st);
// Replaces each of rows x nx floats (row pitch P) by its reciprocal, computed in
// FP64 and rounded once.
cudaError_t launch_reciprocal(float* a, int rows, int nx, int P, cudaStream_t st);
// Sets the device step counter to `it`.
cudaError_t launch_set_step(const Coef& C, int it, cudaStream_t st);
// Adds n to the device step counter (the end of a captured run of n steps).
cudaError_t launch_advance_step(const Coef& C, int n, cudaStream_t st);
// Cells of one shot, and those one stage launch updates, every shot counted.
inline long long shot_cells(const Coef& C) { return (long long)C.nx * (C.nzf + C.nzs); }
inline long long launch_cells(const Coef& C) {
  return shot_cells(C) * (C.nshots > 0 ? C.nshots : 1);
}
// The stage build a launch uses: C.variant, or by one shot's size when 0.
int stage_blocks_per_sm(const Coef& C);
// Rows per interior tile of a stage launch: C.seg, or by size when 0.
int stage_seg_rows(const Coef& C);

// cudaMalloc for the library's own buffers: an allocation that does not fit is
// tried again once the idle memory of the dispersion image's pool has gone back
// (mfdm_dispersion.cu).
cudaError_t device_malloc(void** p, size_t bytes);
template <class T>
cudaError_t device_malloc(T** p, size_t bytes) {
  return device_malloc(reinterpret_cast<void**>(p), bytes);
}

// Library-internal host helpers (mfdm_host.cu): record a failure for
// mfdm_last_error() and return `code`.
int set_error(int code, const char* msg);
// Ricker value at `time` in the reference's host float arithmetic: the one
// source of every Ricker table the library uploads.
float ricker_ref(float fpeak, float time);
// CFS-PML factors (d/beta, alpha + d/beta, 1/beta, 0) of cell i of an axis of n
// cells, computed in FP64 on the host: the one source of every PML table.
float4 pml_cell(float fpeak, float beta0, int npd, int npow, float vp_max, float rc,
                float thickness, int i, int n, bool lo, bool hi);
}  // namespace mfdm
