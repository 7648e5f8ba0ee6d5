// Small kernels of the fluid-solid time step and the choice of the stage build.
// The stage kernels are in mfdm_stage.cu.
#include "mfdm_kernels.h"

namespace mfdm {

namespace b2 {
cudaError_t launch_stage(const Coef&, const Fields&, const Fields&, const Fields&, const Fields&, int, int, cudaStream_t);
}
namespace b3 {
cudaError_t launch_stage(const Coef&, const Fields&, const Fields&, const Fields&, const Fields&, int, int, cudaStream_t);
}
namespace b4 {
cudaError_t launch_stage(const Coef&, const Fields&, const Fields&, const Fields&, const Fields&, int, int, cudaStream_t);
}
namespace b4o {
cudaError_t launch_stage(const Coef&, const Fields&, const Fields&, const Fields&, const Fields&, int, int, cudaStream_t);
}

namespace {

__global__ void reciprocal_rows_kernel(float* a, int rows, int nx, int P) {
  const int ix = blockIdx.x * blockDim.x + threadIdx.x, iz = blockIdx.y;
  if (ix < nx && iz < rows) {
    float* p = a + (size_t)iz * P + ix;
    *p = float(1.0 / double(*p));
  }
}

__global__ void set_step_kernel(int* step, int it) { *step = it; }
__global__ void advance_step_kernel(int* step, int n) { *step += n; }

}  // namespace

// The builds contract the strips' and rows' arithmetic differently and their two
// accumulation forms round differently, so the choice among them follows the grid
// of one shot alone: a shot's bits do not depend on how many shots step with it,
// and a batch gives what its shots give alone. (Tile heights change no bits and
// follow the whole launch.)
// Up to half a million cells the launch is one wave or two and its time is the
// latency of a block: the build with the larger register budget (3) is faster;
// beyond, the throughput of the interior tiles decides and the build with more
// resident blocks (4) is. Measured before launches were chained (mfdm_stage.cu), us
// a step, build 3 / 4: 160x121 23.4 / 27.4; 400x400 30.5 / 40.2; 800x400 35.4 /
// 43.1; 700x700 44.6 / 46.9; 1200x800 98.5 / 83.6; 4096x2048 624 / 498. Batches by
// this rule / by the whole launch: 64 of 160x121 171 / 187, 8 of 400x400 141 / 135,
// 4 of 800x600 180 / 168.
int stage_blocks_per_sm(const Coef& C) {
  if (C.variant == 2 || C.variant == 3 || C.variant == 4) return C.variant;
  return shot_cells(C) < 500000 ? 3 : 4;
}

// Short tiles give a small grid enough blocks, tall ones stage fewer halo rows.
// Measured with the builds above (us a step at 8 / 16 / 24 / 32 rows): 400x400
// 28.1 / 28.4 / 29.8 / 29.9; 800x400 36.7 / 33.6 / 38.3 / 36.0; 1200x800 82.6 /
// 78.6 / 76.0 / 77.7; 2048x1024 166 / 156 / 154 / 154; 4096x2048 576 / 521 / 502 / 495.
int stage_seg_rows(const Coef& C) {
  if (C.seg > 0) return C.seg;
  const long long n = launch_cells(C);
  return n < 200000 ? 8 : n < 500000 ? 16 : n < 4000000 ? 24 : 32;
}

cudaError_t launch_stage(const Coef& C, const Fields& in, const Fields& out, const Fields& un,
                         const Fields& acc, int stage, int dir, cudaStream_t st) {
  switch (stage_blocks_per_sm(C)) {
    case 2: return b2::launch_stage(C, in, out, un, acc, stage, dir, st);
    case 3: return b3::launch_stage(C, in, out, un, acc, stage, dir, st);
    // Accumulating once a step saves 17 % of the traffic. Below 2.5 million cells
    // a shot is bound by latency and the L2 cache and gains less (us a step,
    // in every stage / once: 1200x800 80.2 / 77.1, 1600x1500 192 / 169), and the
    // reference's order of roundings stays; above, DRAM traffic decides
    // (4096x2048: 570 / 495). A batch of smaller grids keeps the order of its
    // shots alone and pays for it (64 shots of 1200x800: 4394 / 3721).
    default:
      return shot_cells(C) < 2500000 ? b4::launch_stage(C, in, out, un, acc, stage, dir, st)
                                       : b4o::launch_stage(C, in, out, un, acc, stage, dir, st);
  }
}

cudaError_t launch_reciprocal(float* a, int rows, int nx, int P, cudaStream_t st) {
  if (rows <= 0 || nx <= 0) return cudaSuccess;
  reciprocal_rows_kernel<<<dim3((nx + 255) / 256, rows), 256, 0, st>>>(a, rows, nx, P);
  return cudaGetLastError();
}

cudaError_t launch_set_step(const Coef& C, int it, cudaStream_t st) {
  set_step_kernel<<<1, 1, 0, st>>>(C.step, it);
  return cudaGetLastError();
}

cudaError_t launch_advance_step(const Coef& C, int n, cudaStream_t st) {
  advance_step_kernel<<<1, 1, 0, st>>>(C.step, n);
  return cudaGetLastError();
}

}  // namespace mfdm
