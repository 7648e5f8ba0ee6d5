// Tiles of the stage kernels (fluid-solid and solid only): a block of 256 threads
// stages the stage input of 32 columns x some rows and their halo in shared
// memory and computes one cell per thread and 8 rows.
#pragma once
#include "mfdm_async.cuh"

namespace mfdm {
namespace tiles {

constexpr int kThreads = 256;
constexpr int kTX = 32;                   // columns of a tile
constexpr int kW = kTX + 8;               // staged columns x0-4 .. x0+35
constexpr int kRowStep = kThreads / kTX;  // rows between a thread's cells (8)
constexpr int kTileRowsMax = 48;          // tallest interior tile
// Shared memory of an interior tile: tr + 6 rows of 5 fields, the columns and a
// 4-column halo each side (more than a PML tile or an interface block needs).
constexpr size_t tile_smem(int tr) { return size_t(tr + 6) * 5 * (kTX + 8) * sizeof(float); }

// Stage input staged as [row][field][column]: every neighbour of a cell is its
// base plus a compile-time offset.
template <int NST>
struct TileAcc {
  const float* base;
  __device__ __forceinline__ TileAcc(const float* tile, int lz, int c)
      : base(tile + lz * (NST * kW) + c) {}
  __device__ __forceinline__ float at(int f, int dz, int dx) const {
    return base[dz * (NST * kW) + f * kW + dx];
  }
};
// Stages rows z0-LO .. z0+tr+HI-1 of the NST fields at `f` (plane stride `plane`,
// `rows` rows of pitch P), columns x0-4 .. x0+35 (x0 a multiple of 4), with
// 16-byte asynchronous copies; zero outside the arrays. Every thread owns one
// float4 column of every kPass-th row.
template <int NST, int LO, int HI>
__device__ __forceinline__ void stage_tile(float* tile, const float* f, size_t plane, int x0, int z0,
                                           int tr, int rows, int P) {
  constexpr int kV = kW / 4, kPer = NST * kV, kPass = kThreads / kPer;
  const int rr = threadIdx.x / kPer, e = threadIdx.x - rr * kPer, q = e / kV, vc = (e - q * kV) * 4;
  const int col = x0 - 4 + vc;
  const bool in_x = col >= 0 && col < P;
  const float* src = f + q * plane + col;
  uint32_t dst = smem_addr(tile + ((3 - LO + rr) * NST + q) * kW + vc);
  if (rr < kPass)
    for (int r = z0 - LO + rr; r < z0 + tr + HI; r += kPass, dst += kPass * NST * kW * 4) {
      const bool ok = in_x && r >= 0 && r < rows;
      cp_async16(dst, ok ? src + (size_t)r * P : f, ok);
    }
  cp_async_commit();
}

// A rectangle of tiles: columns from x0 (`ntx` tiles a row) to below x1, rows
// z0..z1-1; its blocks are [first, next rectangle's first).
struct Band {
  int first, x0, x1, ntx, z0, z1;
};
struct Tile {
  int x0, x1, z0, z1;
};
__device__ __forceinline__ Tile tile_of(const Band& b, int blk, int tr) {
  const int k = blk - b.first, bz = k / b.ntx;
  Tile t;
  t.x0 = b.x0 + (k - bz * b.ntx) * kTX;
  t.x1 = b.x1;
  t.z0 = b.z0 + bz * tr;
  t.z1 = min(t.z0 + tr, b.z1);
  return t;
}

// Launches a stage kernel; chained: it may start while the stage launch before it
// on the stream ends (mfdm_async.cuh).
template <class Args>
cudaError_t launch_tiles(void (*kernel)(Args), const Args& a, int blocks, size_t smem, bool chained,
                         cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Columns [x0, x1) x rows [z0, z1) in tiles of tz rows, blocks from `first` on.
inline int make_band(Band& b, int x0, int x1, int z0, int z1, int tz, int first) {
  const bool empty = x1 <= x0 || z1 <= z0;
  b = {first, x0, x1, empty ? 1 : ceil_div(x1 - x0, kTX), z0, empty ? z0 : z1};
  return first + (empty ? 0 : b.ntx * ceil_div(z1 - z0, tz));
}

}  // namespace tiles
}  // namespace mfdm
