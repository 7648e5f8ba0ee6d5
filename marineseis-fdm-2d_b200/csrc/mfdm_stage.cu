// sm_100a stage kernels of the fluid-solid RK4 time step.
//
// One launch per RK stage does the whole stage: the stage right-hand side of
// every fluid and solid cell (the four reference RHS kernels), the mirrored
// ghost fluxes (built on the fly from the stage input instead of a separate
// build_ghost_flux launch), the source, the interface coupling and the RK4
// bookkeeping (the 48 matrix_add / matrix_self_add launches and the 48 reset
// copies of the reference). The last stage's interface blocks also filter the
// interface rows and sample the receivers. Reference: src/pml_fs_kernels.cu:428-868.
//
// Block roles inside one stage launch (the shot is the fastest block index, so
// the shots of one tile run side by side and all but the first read its
// coefficients from L2), in the order of the block index, the slow ones first:
//   interface columns (fluid row nz_f-1 and solid row 0, coupled);
//   the rows with conservative or one-sided operators (fluid rows 3..5 under
//     the free surface and nz_f-3, nz_f-2, solid rows 1, 2), whole rows;
//   PML tiles of 32 columns x 8 rows over the absorbing strips;
//   interior tiles of 32 columns x `tr` rows, which take a branch-free body.
#include <algorithm>

#include "mfdm_device.cuh"
#include "mfdm_kernels.h"
#include "mfdm_tile.cuh"

// This file is compiled four times: with a register budget for 3 (as it is), 2
// (mfdm_stage_b2.cu) and 5 (mfdm_stage_b4.cu, mfdm_stage_b4o.cu) resident blocks
// per SM; the last accumulates once a step (see rk_acc), the others in every
// stage, in the reference's order.
#ifndef MFDM_STAGE_NS
#define MFDM_STAGE_NS b3
#define MFDM_STAGE_BLOCKS 3
#define MFDM_STAGE_ONCE false
#endif

namespace mfdm {
namespace MFDM_STAGE_NS {
namespace {

using namespace tiles;

constexpr bool kOnce = MFDM_STAGE_ONCE;
// Launches of the other builds may start as the stage launch before them ends: the
// gap between dependent launches is 3 to 14 % of a step (us a step, plain /
// chained: 160x121 24.6 / 21.1, 400x400 30.1 / 28.0, 800x400 36.0 / 31.8,
// 1200x800 83.8 / 79.7, 2048x1024 177 / 172). A block lets the next grid start once
// its own operands have arrived, not at its start: the waiting blocks of two later
// grids would take the slots (160x121 26.4, 800x400 at 16 rows 32.0). Large grids gain nothing
// (4096x2048 499 / 505).
constexpr bool kChain = !kOnce;
struct FluidTile : TileAcc<3> {
  using TileAcc<3>::TileAcc;
  __device__ __forceinline__ float fvx(int dz, int dx) const { return at(0, dz, dx); }
  __device__ __forceinline__ float fvz(int dz, int dx) const { return at(1, dz, dx); }
  __device__ __forceinline__ float fp(int dz, int dx) const { return at(2, dz, dx); }
};
struct SolidTile : TileAcc<5> {
  using TileAcc<5>::TileAcc;
  __device__ __forceinline__ float svx(int dz, int dx) const { return at(0, dz, dx); }
  __device__ __forceinline__ float svz(int dz, int dx) const { return at(1, dz, dx); }
  __device__ __forceinline__ float ssx(int dz, int dx) const { return at(2, dz, dx); }
  __device__ __forceinline__ float ssz(int dz, int dx) const { return at(3, dz, dx); }
  __device__ __forceinline__ float ssxz(int dz, int dx) const { return at(4, dz, dx); }
};

// The shot's source cell.
__device__ __forceinline__ int2 source_of(const Coef& C, int shot) {
  return C.src_pos ? __ldg(C.src_pos + shot) : make_int2(C.srcx, C.srcz);
}
__device__ __forceinline__ float4 pml_at(const float4* t, size_t so, int i) {
  return __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(t) + so) + i);
}

// A value that the launch before may have written: not through the read-only
// cache where this launch may have started before that one's end.
__device__ __forceinline__ float ld(const float* p) { return kChain ? *p : __ldg(p); }
struct Ld {
  __device__ __forceinline__ float operator()(const float* p) const { return ld(p); }
};

// Point-wise operands of one cell: `u`, U^n (second and third stage) or the
// accumulator (last stage); `q`, the accumulator where these stages add to it;
// and the coefficient block's values.
template <int NST, int NCOEF>
struct Pt { float u[NST], q[NST], k[NCOEF]; };
// Stages that read the accumulator besides U^n.
template <int KIND>
constexpr bool kAdds = !kOnce && (KIND == kStageSecond || KIND == kStageThird);

// The coefficients, which no launch writes, and the rest, which the launch before
// may have written.
template <int NST, int NCOEF>
__device__ __forceinline__ void load_coef(Pt<NST, NCOEF>& p, const float* coef, size_t plane, size_t i) {
#pragma unroll
  for (int q = 0; q < NCOEF; ++q) p.k[q] = __ldg(coef + q * plane + i);
}
template <int KIND, int NST, int NCOEF>
__device__ __forceinline__ void load_pt(Pt<NST, NCOEF>& p, const float* u, const float* acc,
                                        size_t plane, size_t i) {
#pragma unroll
  for (int f = 0; f < NST; ++f) {
    if (KIND != kStageFirst) p.u[f] = ld(u + f * plane + i);
    if (kAdds<KIND>) p.q[f] = (acc + f * plane)[i];
  }
}

// The four ADE values of a strip cell: the stage input's (`y`) and the operands
// `u` and `q` as in Pt, loaded before any store of the cell.
template <int KIND>
__device__ __forceinline__ void load_ade(float* y, float* u, float* qa, float* const* in, float* const* un,
                                         float* const* acc, size_t i) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    y[q] = ld(in[q] + i);
    if (KIND == kStageSecond || KIND == kStageThird) u[q] = ld(un[q] + i);
    if (KIND == kStageLast) u[q] = acc[q][i];
    if (kAdds<KIND>) qa[q] = acc[q][i];
  }
}

// RK update of one value from loaded operands: stage input y, u and q as in Pt.
template <int KIND>
__device__ __forceinline__ void rk_store(float k, float y, float u, float q, float* out, float* acc,
                                         size_t i, float c, float w) {
  if (KIND == kStageFirst) {
    out[i] = fmaf(c, k, y);
    if (!kOnce) acc[i] = fmaf(w, k, y);
  } else if (KIND == kStageLast) {
    out[i] = kOnce ? rk_last(k, y, u, c) : fmaf(c, k, u);
  } else {
    out[i] = fmaf(c, k, u);
    if (kAdds<KIND>)
      acc[i] = fmaf(w, k, q);
    else if (KIND == kStageSecond)
      acc[i] = rk_acc(k, y, u, w);
  }
}

constexpr int kBands = 6;  // fluid: left, right, top (four-side CPML); solid: left, right, bottom

struct StageArgs {
  Coef C;
  Fields in, out, un, acc;
  int s, nshots;
  int nbi;               // interface blocks
  int nft, fb0, nfb, ns;  // row blocks: fluid rows 3..2+nft and fb0..fb0+nfb-1, solid rows 1..ns
  int ncol;              // column chunks of a row
  Band pml[kBands];      // PML tiles
  Band inner[2];         // interior tiles of the fluid and the solid, `tr` rows each
  int tr;
  float cc, w;
};

// One fluid (solid) tile: rows 6..nz_f-4 (3..nz_s-4; from row 3
// with four-side CPML), where the plain operators hold. PML: cells may lie in an
// absorbing strip (one row per thread); otherwise none does and a thread takes
// every kRowStep-th row.
template <int DIR, int KIND, bool CPML, bool PML>
__device__ __forceinline__ void fluid_tile(const StageArgs& a, int shot, const Tile& tl, float* tile) {
  const Coef& C = a.C;
  const int P = C.P, nx = C.nx, nzf = C.nzf, npd = C.npd;
  const size_t so = size_t(shot) * C.shot_stride, nf = size_t(nzf) * P;
  const int ty = threadIdx.x / kTX, tx = threadIdx.x % kTX, ix = tl.x0 + tx;
  const float* u = (KIND == kStageLast ? a.acc.fvx : a.un.fvx) + so;
  const float* coef = C.rhof - 4 * nf;  // the fluid coefficient block [6][nz_f][P]
  if (kChain) wait_previous();
  stage_tile<3, DIR == kDirF ? 1 : 3, DIR == kDirF ? 3 : 1>(
      tile, a.in.fvx + so, nf, tl.x0, tl.z0, PML ? kRowStep : a.tr, nzf, P);
  int iz = tl.z0 + ty;
  const bool active = ix < tl.x1 && (!PML || ix >= 3) && iz < tl.z1;
  Pt<3, 6> p;
  if (active) load_pt<KIND>(p, u, a.acc.fvx + so, nf, (size_t)iz * P + ix);
  if (active) load_coef(p, coef, nf, (size_t)iz * P + ix);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool side = PML && active && min(ix - 3, nx - 4 - ix) < npd;
  const bool top = PML && CPML && active && iz <= npd + 2;  // four-side CPML: rows 3..npd+2
  const size_t si = so + (size_t)iz * C.Ps + (side ? xstrip_col(ix, nx, npd) : 0);
  const size_t zi = so + (size_t)(iz - 3) * P + ix;
  float ade[4], ua[4], qa[4], zade[4], uz[4], qz[4];
  float4 px = zero, pmz = zero;
  const int2 src = source_of(C, shot);
  // the source's 5x5 cells touch this tile
  const bool near_src = src.x >= tl.x0 - 2 && src.x < tl.x0 + kTX + 2 && src.y >= tl.z0 - 2 && src.y < tl.z1 + 2;
  if (side) px = pml_at(C.pmlx, so, ix);
  if (top) pmz = pml_at(C.pmlzf, so, iz);
  if (side) load_ade<KIND>(ade, ua, qa, a.in.fx, a.un.fx, a.acc.fx, si);
  if (top) load_ade<KIND>(zade, uz, qz, a.in.fz, a.un.fz, a.acc.fz, zi);
  cp_async_wait_all();
  if (kChain) launch_dependents();
  __syncthreads();
  if (!active) return;
#pragma unroll 1
  for (;;) {
    const size_t i = (size_t)iz * P + ix;
    const FluidTile A(tile, 3 + iz - tl.z0, 4 + tx);
    const FluidCoefs cf{p.k[0], p.k[1], p.k[2], p.k[3], p.k[4], p.k[5]};
    FluidK k = fluid_rhs<DIR, true, CPML>(C, A, iz, ix, side, ade, cf, px, top, zade, pmz);
    if (near_src)
      k.p += source_term(C, src.x, src.y, C.src_amp + size_t(shot) * C.src_stride, iz, ix,
                         time_index(C), a.s);
    const float kv[3] = {k.vx, k.vz, k.p};
#pragma unroll
    for (int f = 0; f < 3; ++f)
      rk_store<KIND>(kv[f], A.at(f, 0, 0), p.u[f], p.q[f], a.out.fvx + f * nf, a.acc.fvx + f * nf, so + i,
                     a.cc, a.w);
    if (PML) {
      const float ka[4] = {k.V0, k.V1, k.E0, k.E1}, kz[4] = {k.ZV0, k.ZV1, k.ZE0, k.ZE1};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (side) rk_store<KIND>(ka[q], ade[q], ua[q], qa[q], a.out.fx[q], a.acc.fx[q], si, a.cc, a.w);
        if (top) rk_store<KIND>(kz[q], zade[q], uz[q], qz[q], a.out.fz[q], a.acc.fz[q], zi, a.cc, a.w);
      }
      return;
    }
    iz += kRowStep;
    if (iz >= tl.z1) return;
    load_pt<KIND>(p, u, a.acc.fvx + so, nf, (size_t)iz * P + ix);
    load_coef(p, coef, nf, (size_t)iz * P + ix);
  }
}

template <int DIR, int KIND, bool CPML, bool PML>
__device__ __forceinline__ void solid_tile(const StageArgs& a, int shot, const Tile& tl, float* tile) {
  const Coef& C = a.C;
  const int P = C.P, nx = C.nx, nzs = C.nzs, npd = C.npd, zb0 = nzs - 3 - npd;
  const size_t so = size_t(shot) * C.shot_stride, ns = size_t(nzs) * P;
  const int ty = threadIdx.x / kTX, tx = threadIdx.x % kTX, ix = tl.x0 + tx;
  const float* u = (KIND == kStageLast ? a.acc.svx : a.un.svx) + so;
  const float* coef = C.rhos - 4 * ns;  // the solid coefficient block [9][nz_s][P]
  if (kChain) wait_previous();
  stage_tile<5, DIR == kDirF ? 1 : 3, DIR == kDirF ? 3 : 1>(
      tile, a.in.svx + so, ns, tl.x0, tl.z0, PML ? kRowStep : a.tr, nzs, P);
  int iz = tl.z0 + ty;
  const bool active = ix < tl.x1 && (!PML || ix >= 3) && iz < tl.z1;
  Pt<5, 9> p;
  if (active) load_pt<KIND>(p, u, a.acc.svx + so, ns, (size_t)iz * P + ix);
  if (active) load_coef(p, coef, ns, (size_t)iz * P + ix);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool side = PML && active && min(ix - 3, nx - 4 - ix) < npd;
  const bool bottom = PML && active && iz >= zb0;
  const size_t sxi = so + (size_t)iz * C.Ps + (side ? xstrip_col(ix, nx, npd) : 0);
  const size_t szi = so + (size_t)(iz - zb0) * P + ix;
  float xade[4], ux[4], qx[4], zade[4], uz[4], qz[4];
  float4 px = zero, pz = zero;
  if (side) px = pml_at(C.pmlx, so, ix);
  if (bottom) pz = pml_at(C.pmlz, so, iz);
  if (side) load_ade<KIND>(xade, ux, qx, a.in.sx, a.un.sx, a.acc.sx, sxi);
  if (bottom) load_ade<KIND>(zade, uz, qz, a.in.sz, a.un.sz, a.acc.sz, szi);
  cp_async_wait_all();
  if (kChain) launch_dependents();
  __syncthreads();
  if (!active) return;
#pragma unroll 1
  for (;;) {
    const size_t i = (size_t)iz * P + ix;
    const SolidTile A(tile, 3 + iz - tl.z0, 4 + tx);
    const SolidCoefs cf{p.k[0], p.k[1], p.k[2], p.k[3], p.k[4], p.k[5], p.k[6], p.k[7], p.k[8]};
    const SolidK k = solid_rhs<DIR, true, CPML>(C, A, iz, ix, side, bottom, xade, zade, cf, px, pz);
    const float kv[5] = {k.vx, k.vz, k.sx, k.sz, k.sxz};
#pragma unroll
    for (int f = 0; f < 5; ++f)
      rk_store<KIND>(kv[f], A.at(f, 0, 0), p.u[f], p.q[f], a.out.svx + f * ns, a.acc.svx + f * ns, so + i,
                     a.cc, a.w);
    if (PML) {
      const float kx[4] = {k.XV0, k.XV1, k.XE0, k.XE1}, kz[4] = {k.ZV0, k.ZV1, k.ZE0, k.ZE1};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (side) rk_store<KIND>(kx[q], xade[q], ux[q], qx[q], a.out.sx[q], a.acc.sx[q], sxi, a.cc, a.w);
        if (bottom) rk_store<KIND>(kz[q], zade[q], uz[q], qz[q], a.out.sz[q], a.acc.sz[q], szi, a.cc, a.w);
      }
      return;
    }
    iz += kRowStep;
    if (iz >= tl.z1) return;
    load_pt<KIND>(p, u, a.acc.svx + so, ns, (size_t)iz * P + ix);
    load_coef(p, coef, ns, (size_t)iz * P + ix);
  }
}

// Whole rows by direct loads: each half of the block takes kIfCols columns of
// one row with the fully general right-hand side. An interface block's halves
// take fluid row nz_f-1 and solid row 0 of the same columns; their RHS meet in shared memory for the
// normal/tangential coupling (pml_fs_kernels.cuh:754-827) and each half updates
// its own medium. In the last stage a block owns kIfCols - 6 columns and
// recomputes the three on either side, so that it can filter its rows (7-point
// Gaussian along x, renormalised at the clamped ends, and the continuity
// average, src/pml_fs_kernels.cu:428-525, out of place) and sample the
// receivers (src/main.cu:195-211) in the same launch.
constexpr int kIfCols = kThreads / 2;
__host__ __device__ constexpr int interface_cols(int kind) { return kind == kStageLast ? kIfCols - 6 : kIfCols; }

template <int DIR, int KIND, bool CPML>
__device__ __forceinline__ void row_block(const StageArgs& a, int shot, int blk, float* smem) {
  const Coef& C = a.C;
  const int nx = C.nx, P = C.P, nzf = C.nzf, nzs = C.nzs, npd = C.npd;
  const size_t so = size_t(shot) * C.shot_stride, nf = size_t(nzf) * P, ns = size_t(nzs) * P;
  const int t = threadIdx.x % kIfCols, half = threadIdx.x / kIfCols;
  const bool iface = blk < a.nbi;
  const int H = iface && KIND == kStageLast ? 3 : 0;
  bool solid = half == 1;
  int iz = solid ? 0 : nzf - 1, ix = blk * interface_cols(KIND) + t - H;
  bool valid = true;
  if (!iface) {
    const int pair = (blk - a.nbi) / a.ncol, q = 2 * pair + half;
    ix = (blk - a.nbi - pair * a.ncol) * kIfCols + t;
    solid = q >= a.nft + a.nfb;
    iz = q < a.nft ? 3 + q : (solid ? 1 + q - a.nft - a.nfb : a.fb0 + q - a.nft);
    valid = q < a.nft + a.nfb + a.ns;
  }
  valid = valid && ix >= 3 && ix <= nx - 4;
  const bool side = valid && min(ix - 3, nx - 4 - ix) < npd;
  const int scol = side ? xstrip_col(ix, nx, npd) : 0;
  const int zb0 = nzs - 3 - npd;
  const bool bottom = iz >= zb0;             // a solid row the bottom band reaches
  const bool ftop = CPML && iz <= npd + 2;   // a fluid row the top band reaches
  const size_t fi = (size_t)iz * P + ix, si = fi;  // the fluid or solid cell
  float(*kk)[kIfCols] = reinterpret_cast<float(*)[kIfCols]>(smem);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float y[5], u[5], q[5], kv[5], xa[4], ux[4], qx[4], za[4], uz[4], qz[4], kx[4], kz[4];
  bool has_E = true;
  size_t xi = 0, zi = 0;
  if (kChain) wait_previous();
  if (valid) {
    const float4 px = side ? pml_at(C.pmlx, so, ix) : zero;
    if (!solid) {
      const FluidAt<Ld> A{a.in.fvx + so, a.in.fvz + so, a.in.fp + so, fi, P};
      xi = so + (size_t)iz * C.Ps + scol;
      zi = so + (size_t)(iz - 3) * P + ix;
      const float* ub = (KIND == kStageLast ? a.acc.fvx : a.un.fvx) + so;
#pragma unroll
      for (int f = 0; f < 3; ++f) {
        y[f] = ld(a.in.fvx + so + f * nf + fi);
        u[f] = KIND == kStageFirst ? 0.f : ub[f * nf + fi];
        if (kAdds<KIND>) q[f] = (a.acc.fvx + so)[f * nf + fi];
      }
      if (side) load_ade<KIND>(xa, ux, qx, a.in.fx, a.un.fx, a.acc.fx, xi);
      if (ftop) load_ade<KIND>(za, uz, qz, a.in.fz, a.un.fz, a.acc.fz, zi);
      FluidK k = fluid_rhs<DIR, false, CPML>(C, A, iz, ix, side, xa, fluid_coefs_global(C, fi), px,
                                             ftop, za, ftop ? pml_at(C.pmlzf, so, iz) : zero);
      const int2 src = source_of(C, shot);
      k.p += source_term(C, src.x, src.y, C.src_amp + size_t(shot) * C.src_stride, iz, ix,
                         time_index(C), a.s);
      has_E = k.has_E;
      kv[0] = k.vx; kv[1] = k.vz; kv[2] = k.p;
      kx[0] = k.V0; kx[1] = k.V1; kx[2] = k.E0; kx[3] = k.E1;
      kz[0] = k.ZV0; kz[1] = k.ZV1; kz[2] = k.ZE0; kz[3] = k.ZE1;
    } else {
      const SolidAt<Ld> A{a.in.svx + so, a.in.svz + so, a.in.ssx + so, a.in.ssz + so, a.in.ssxz + so, si, P};
      xi = so + (size_t)iz * C.Ps + scol;
      zi = so + (size_t)(iz - zb0) * P + ix;
      const float* ub = (KIND == kStageLast ? a.acc.svx : a.un.svx) + so;
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        y[f] = ld(a.in.svx + so + f * ns + si);
        u[f] = KIND == kStageFirst ? 0.f : ub[f * ns + si];
        if (kAdds<KIND>) q[f] = (a.acc.svx + so)[f * ns + si];
      }
      if (side) load_ade<KIND>(xa, ux, qx, a.in.sx, a.un.sx, a.acc.sx, xi);
      if (bottom) load_ade<KIND>(za, uz, qz, a.in.sz, a.un.sz, a.acc.sz, zi);
      const SolidK k = solid_rhs<DIR, false, CPML>(C, A, iz, ix, side, bottom, xa, za,
                                                   solid_coefs_global(C, si, si + (size_t)(nzf - 1) * P),
                                                   px, bottom ? pml_at(C.pmlz, so, iz) : zero);
      kv[0] = k.vx; kv[1] = k.vz; kv[2] = k.sx; kv[3] = k.sz; kv[4] = k.sxz;
      kx[0] = k.XV0; kx[1] = k.XV1; kx[2] = k.XE0; kx[3] = k.XE1;
      kz[0] = k.ZV0; kz[1] = k.ZV1; kz[2] = k.ZE0; kz[3] = k.ZE1;
    }
  }
  const bool owner = valid && t >= H && t < kIfCols - H;
  if (owner) {
    if (side) {
      float* const* ox = solid ? a.out.sx : a.out.fx;
      float* const* ax = solid ? a.acc.sx : a.acc.fx;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q < 2 || has_E) rk_store<KIND>(kx[q], xa[q], ux[q], qx[q], ox[q], ax[q], xi, a.cc, a.w);
    }
    if (solid ? bottom : ftop) {
      float* const* oz = solid ? a.out.sz : a.out.fz;
      float* const* az = solid ? a.acc.sz : a.acc.fz;
#pragma unroll
      for (int q = 0; q < 4; ++q) rk_store<KIND>(kz[q], za[q], uz[q], qz[q], oz[q], az[q], zi, a.cc, a.w);
    }
  }
  if (kChain) launch_dependents();
  float2 n = make_float2(0.f, 0.f);
  if (iface) {  // the whole block is one or is not
    if (valid) {
      n = __ldg(C.nrm + ix);
#pragma unroll
      for (int f = 0; f < 5; ++f)
        if (solid || f < 3) kk[(solid ? 3 : 0) + f][t] = kv[f];
    }
    __syncthreads();
    if (valid) {
      const float kf[3] = {kk[0][t], kk[1][t], kk[2][t]};
      const float ks[5] = {kk[3][t], kk[4][t], kk[5][t], kk[6][t], kk[7][t]};
      float kc[8];
      couple_rhs<DIR>(n, kf, ks, kc);
#pragma unroll
      for (int f = 0; f < 5; ++f) kv[f] = solid ? kc[3 + f] : (f < 3 ? kc[f] : 0.f);
    }
  }
  if (KIND != kStageLast || !iface) {
    if (!owner) return;
    if (!solid) {
#pragma unroll
      for (int f = 0; f < 3; ++f)
        rk_store<KIND>(kv[f], y[f], u[f], q[f], a.out.fvx + f * nf, a.acc.fvx + f * nf, so + fi, a.cc, a.w);
    } else {
#pragma unroll
      for (int f = 0; f < 5; ++f)
        rk_store<KIND>(kv[f], y[f], u[f], q[f], a.out.svx + f * ns, a.acc.svx + f * ns, so + si, a.cc, a.w);
    }
    return;
  }
  // the coupled state before the filter, then the filter
  __syncthreads();  // every read of kk is done
  if (valid) {
    if (!solid) {
#pragma unroll
      for (int f = 0; f < 3; ++f) kk[f][t] = kOnce ? rk_last(kv[f], y[f], u[f], a.cc) : fmaf(a.cc, kv[f], u[f]);
    } else {
#pragma unroll
      for (int f = 0; f < 5; ++f) kk[3 + f][t] = kOnce ? rk_last(kv[f], y[f], u[f], a.cc) : fmaf(a.cc, kv[f], u[f]);
    }
  }
  __syncthreads();
  if (!owner) return;
  const int klo = max(-3, 3 - ix), khi = min(3, nx - 4 - ix);
  // taps k = klo..khi in ascending order (the reference's summation order)
  float wsum = 0.0f;
#pragma unroll
  for (int k = -3; k <= 3; ++k)
    if (k >= klo && k <= khi) wsum += c_w7[k + 3];
  float v[8], un[8];
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    float sum = 0.0f;
#pragma unroll
    for (int k = -3; k <= 3; ++k)
      if (k >= klo && k <= khi) sum += c_w7[k + 3] * kk[f][t + k];
    v[f] = sum / wsum;
  }
  interface_average(n, v, un);
  const int it = time_index(C), j = C.gap > 0 ? it / C.gap : 0;
  const bool sample = C.rec != nullptr && C.gap > 0 && j * C.gap == it && j < C.rec_cap;
  float* row = C.rec + (sample ? size_t(shot) * C.rec_stride + (size_t)j * 3 * nx : 0);
  if (!solid) {
#pragma unroll
    for (int f = 0; f < 3; ++f) a.out.fvx[so + f * nf + fi] = un[f];
    if (sample) row[2 * nx + ix] = un[2];
    if (!isfinite(un[2])) atomicOr(C.status, 1);
  } else {
#pragma unroll
    for (int f = 0; f < 5; ++f) a.out.svx[so + f * ns + si] = un[3 + f];
    if (sample) {
      row[ix] = un[3];
      row[nx + ix] = un[4];
    }
    if (!(isfinite(un[3]) && isfinite(un[4]))) atomicOr(C.status, 1);
  }
}

template <int DIR, int KIND, bool CPML>
__global__ void __launch_bounds__(kThreads, MFDM_STAGE_BLOCKS)
    stage_kernel(const __grid_constant__ StageArgs a) {
  extern __shared__ __align__(16) float tile[];
  const int shot = a.nshots > 1 ? int(blockIdx.x % unsigned(a.nshots)) : 0;
  const int b = a.nshots > 1 ? int(blockIdx.x / unsigned(a.nshots)) : int(blockIdx.x);
  if (b < a.pml[0].first) {
    row_block<DIR, KIND, CPML>(a, shot, b, tile);
  } else if (b < a.inner[0].first) {
    int k = 0;
#pragma unroll
    for (int q = 1; q < kBands; ++q)
      if (b >= a.pml[q].first) k = q;
    const Tile t = tile_of(a.pml[k], b, kRowStep);
    if (k < 3)
      fluid_tile<DIR, KIND, CPML, true>(a, shot, t, tile);
    else
      solid_tile<DIR, KIND, CPML, true>(a, shot, t, tile);
  } else if (b < a.inner[1].first) {
    fluid_tile<DIR, KIND, CPML, false>(a, shot, tile_of(a.inner[0], b, a.tr), tile);
  } else {
    solid_tile<DIR, KIND, CPML, false>(a, shot, tile_of(a.inner[1], b, a.tr), tile);
  }
}

// Rows of an interior tile: the height set or chosen, rounded up to a multiple of 8, at most 48.
int tile_rows_of(const Coef& C) {
  const int tr = (stage_seg_rows(C) + kRowStep - 1) / kRowStep * kRowStep;
  return tr < kTileRowsMax ? tr : kTileRowsMax;
}

template <int DIR, int KIND, bool CPML>
cudaError_t launch_one(const Coef& C, const Fields& in, const Fields& out, const Fields& un,
                       const Fields& acc, cudaStream_t st) {
  StageArgs a;
  a.C = C; a.in = in; a.out = out; a.un = un; a.acc = acc;
  a.nshots = C.nshots > 0 ? C.nshots : 1;
  a.tr = tile_rows_of(C);
  a.s = KIND;
  a.nbi = ceil_div(C.nx, interface_cols(KIND));
  const int nx = C.nx, nzf = C.nzf, nzs = C.nzs, npd = C.npd;
  // fluid rows 3..nz_f-2: conservative rows above and below the tiles' rows
  const int f0 = CPML ? 3 : std::min(6, nzf - 1), f1 = std::max(nzf - 3, f0);
  a.nft = f0 - 3; a.fb0 = f1; a.nfb = nzf - 1 - f1;
  // solid rows 1..nz_s-4
  const int s0 = std::min(3, nzs - 3), s1 = nzs - 3;
  a.ns = s0 - 1;
  a.ncol = ceil_div(nx, kIfCols);
  int n = a.nbi + a.ncol * ceil_div(a.nft + a.nfb + a.ns, 2);
  // Tiles: the side strips in whole tile columns, the top band (four-side
  // CPML) and the bottom band between them, and the interior.
  int xl = std::min(ceil_div(3 + npd, kTX) * kTX, nx - 3), xr = std::max((nx - 3 - npd) / kTX * kTX, xl);
  if (xr - xl < 4) xl = xr = nx - 3;  // no interior columns: all in the left band
  const int ft = CPML ? std::min(std::max(npd + 3, f0), f1) : f0;
  const int sb = std::min(std::max(nzs - 3 - npd, s0), s1);
  n = make_band(a.pml[0], 0, xl, f0, f1, kRowStep, n);
  n = make_band(a.pml[1], xr, nx - 3, f0, f1, kRowStep, n);
  n = make_band(a.pml[2], xl, xr, f0, ft, kRowStep, n);
  n = make_band(a.pml[3], 0, xl, s0, s1, kRowStep, n);
  n = make_band(a.pml[4], xr, nx - 3, s0, s1, kRowStep, n);
  n = make_band(a.pml[5], xl, xr, sb, s1, kRowStep, n);
  n = make_band(a.inner[0], xl, xr, ft, f1, a.tr, n);
  n = make_band(a.inner[1], xl, xr, s0, sb, a.tr, n);
  a.cc = C.rk_c[KIND];
  a.w = KIND < kStageLast ? C.rk_w[KIND] : 0.f;
  if (kOnce) {
    const RkOnce once = rk_once(C.rk_c[2]);
    if (KIND == kStageSecond) a.w = once.w;
    if (KIND == kStageLast) a.cc = once.c;
  }
  return launch_tiles(stage_kernel<DIR, KIND, CPML>, a, n * a.nshots, tile_smem(a.tr),
                      kChain && C.chain != 0, st);
}

template <int DIR, bool CPML>
cudaError_t launch_kind(const Coef& C, const Fields& in, const Fields& out, const Fields& un,
                        const Fields& acc, int stage, cudaStream_t st) {
  switch (stage) {
    case 0: return launch_one<DIR, kStageFirst, CPML>(C, in, out, un, acc, st);
    case 1: return launch_one<DIR, kStageSecond, CPML>(C, in, out, un, acc, st);
    case 2: return launch_one<DIR, kStageThird, CPML>(C, in, out, un, acc, st);
    default: return launch_one<DIR, kStageLast, CPML>(C, in, out, un, acc, st);
  }
}

}  // namespace

cudaError_t launch_stage(const Coef& C, const Fields& in, const Fields& out, const Fields& un,
                         const Fields& acc, int stage, int dir, cudaStream_t st) {
  // the four-side CPML variant runs its own kernel instantiations
  if (dir == kDirF)
    return C.cpml ? launch_kind<kDirF, true>(C, in, out, un, acc, stage, st)
                  : launch_kind<kDirF, false>(C, in, out, un, acc, stage, st);
  return C.cpml ? launch_kind<kDirB, true>(C, in, out, un, acc, stage, st)
                : launch_kind<kDirB, false>(C, in, out, un, acc, stage, st);
}

}  // namespace MFDM_STAGE_NS
}  // namespace mfdm
