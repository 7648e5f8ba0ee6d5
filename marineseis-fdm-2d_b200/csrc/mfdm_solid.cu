// sm_100a kernels of the solid-only time step with a free surface (see mfdm_solid.h),
// and of its four-side CFS-PML variant (the CPML instantiations below).
//
// One launch per RK stage does the whole stage: velocity and stress
// right-hand sides of every cell (the reference's update_velocity and
// update_stress, which run as two kernels on two streams), the free-surface
// ghost fluxes (built on the fly from the stage input instead of a separate
// build_ghost_flux launch), the explosive source and the fused RK4 update
// (the reference's vector_add / vector_self_add launches over full grids); the
// last stage also samples the receiver row. Blocks are tiles of 32 columns (as
// the fluid-solid kernels', mfdm_stage.cu), the slow ones first: 8 rows from the
// free surface down with the general right-hand side, 8 rows of an absorbing
// strip, or `tr` interior rows with a branch-free body. Every operand of a cell
// is loaded before its arithmetic and its stores.
//
// Bound: HBM. A step moves 96 floats a cell (inputs 4 x 5, U^n 2 x 5, the
// accumulator 2 x 5, coefficients 4 x 9, outputs 4 x 5), 250 us of 2048x2048 at
// the measured copy rate. Measured, us a step, against tiles of 32 x 16 that loaded
// operand by operand and sampled the receivers in a fifth launch: 400x400 50 -> 20,
// 1000x1000 122 -> 87, 2048x2048 338 -> 292, 4096x4096 1146 -> 1057. A launch may
// start as the one before it ends (mfdm_stage.cu); without: 23, 92, 300, 1058.
#include <algorithm>

#include "mfdm_device.cuh"
#include "mfdm_solid.h"
#include "mfdm_tile.cuh"

namespace mfdm {
namespace solid {
namespace {

using namespace tiles;

enum { kVX = 0, kVZ, kSX, kSZ, kSXZ };

// Point-wise coefficients of a cell, in this order.
enum { kCXIX = 0, kCXIZ, kCZEX, kCZEZ, kCRR, kC11, kC13, kC33, kC55, kNCoef };

struct Out {
  float vx, vz, sx, sz, sxz;
  float XV0, XV1, XE0, XE1, ZV0, ZV1, ZE0, ZE1;
};

// Zeta-ADE row of a cell in a zeta-PML band: the bottom band (rows
// nz-3-npd..nz-4) at 0..npd-1; with CPML the top band (rows 3..npd+2) after it.
template <bool CPML>
__device__ __forceinline__ int zeta_row(int iz, int nz, int npd) {
  if (CPML && iz <= npd + 2) return npd + iz - 3;
  return iz - (nz - 3 - npd);
}

// Right-hand side of cell (iz, ix), 3 <= iz <= nz-4 (include/pml_fs_kernels.cuh:10-307).
// CPML: the four-side variant Cpml::SolidOnly (include/cpml_kernels.cuh:8-217):
// no free surface, so every row takes the plain biased operators (rows 0..2
// are zero), and the zeta-PML also covers the top band (rows 3..npd+2).
// `A(q, dz, dx)` returns stage-input field q (kVX..kSXZ) dz rows and dx columns
// away, |dz|, |dx| <= 3; `K(c)` point-wise coefficient c (kCXIX..kC55).
// SURF: the cell may be one of the three rows under the free surface. PML: it may
// lie in the xi strips (`side`, ADE memory xa, factors px) or in a zeta band
// (`bottom`, za, pz).
template <int DIR, bool SURF, bool PML, bool CPML, class Acc, class Kc>
__device__ __forceinline__ Out rhs(const SCoef& C, const Acc& A, const Kc& K, int iz, int ix,
                                   bool side, bool bottom, const float* xa, const float* za,
                                   float4 px, float4 pz) {
  Out o;
  const int P = C.P;
  const size_t i = (size_t)iz * P + ix;
  const int dist = SURF && !CPML ? iz - 3 : 3;
  constexpr bool IN = !SURF;
  side = PML && side;
  bottom = PML && bottom;
  const float xix = K(kCXIX), xiz = K(kCXIZ), zex = K(kCZEX), zez = K(kCZEZ);
  const float gxixi = xix * xix + xiz * xiz, gzeze = zex * zex + zez * zez;
  const float gxize = xix * zex + xiz * zez;
  auto dx5 = [&](int q) {
    return d5<DIR>(A(q, 0, -3), A(q, 0, -2), A(q, 0, -1), A(q, 0, 0), A(q, 0, 1), A(q, 0, 2),
                   A(q, 0, 3));
  };
  auto dzn = [&](int q, int d) {
    auto col = [&](int j) { return A(q, j, 0); };
    return dz_near<DIR>(col, d, true);
  };
  o.XV0 = o.XV1 = o.XE0 = o.XE1 = o.ZV0 = o.ZV1 = o.ZE0 = o.ZE1 = 0.f;

  // ---- momentum: rho dv/dt = div sigma ----
  {
    float rvx, rvz, dxx = 0.f, dxz = 0.f, dzx = 0.f, dzz = 0.f;
    if (!IN && dist < 3) {
      // conservative rows under the free surface; above it the image G = -F of
      // the rows below (src/pml_fs_kernels.cu:7-19)
      auto Fs = [&](int r) -> float2 {
        const size_t k = (size_t)r * P + ix;
        const float Jk = __ldg(C.J + k), ax = __ldg(C.zex + k), az = __ldg(C.zez + k);
        const float sx = A(kSX, r - iz, 0), sz = A(kSZ, r - iz, 0), sxz = A(kSXZ, r - iz, 0);
        return make_float2(Jk * (ax * sx + az * sxz), Jk * (ax * sxz + az * sz));
      };
      auto Fxi = [&](int j) -> float2 {
        const size_t k = i + j;
        const float Jk = __ldg(C.J + k), ax = __ldg(C.xix + k), az = __ldg(C.xiz + k);
        const float sx = A(kSX, 0, j), sz = A(kSZ, 0, j), sxz = A(kSXZ, 0, j);
        return make_float2(Jk * (ax * sx + az * sxz), Jk * (ax * sxz + az * sz));
      };
      auto Fze = [&](int j) -> float2 {
        const int r = iz + j;
        if (r >= 3) return Fs(r);
        const float2 b = Fs(6 - r);
        return make_float2(-b.x, -b.y);
      };
      const float2 a = dflux<DIR>(Fxi), b = dflux<DIR>(Fze);
      const float Jc = __ldg(C.J + i);
      rvx = (a.x + b.x) / Jc;
      rvz = (a.y + b.y) / Jc;
      const float dxsx = dx5(kSX), dxsz = dx5(kSZ), dxsxz = dx5(kSXZ);
      const float dzsx = dzn(kSX, dist), dzsz = dzn(kSZ, dist), dzsxz = dzn(kSXZ, dist);
      dxx = xix * (dxsx + gxize / gxixi * dzsx) + xiz * (dxsxz + gxize / gxixi * dzsxz);
      dxz = xix * (dxsxz + gxize / gxixi * dzsxz) + xiz * (dxsz + gxize / gxixi * dzsz);
    } else {
      const float sxdx = dx5(kSX), sxdz = dzn(kSX, 3), szdx = dx5(kSZ), szdz = dzn(kSZ, 3);
      const float tdx = dx5(kSXZ), tdz = dzn(kSXZ, 3);
      rvx = xix * sxdx + zex * sxdz + xiz * tdx + zez * tdz;
      rvz = xix * tdx + zex * tdz + xiz * szdx + zez * szdz;
      if (side || bottom) {
        dxx = xix * (sxdx + gxize / gxixi * sxdz) + xiz * (tdx + gxize / gxixi * tdz);
        dxz = xix * (tdx + gxize / gxixi * tdz) + xiz * (szdx + gxize / gxixi * szdz);
        dzx = zex * (sxdz + gxize / gzeze * sxdx) + zez * (gxize / gzeze * tdx + tdz);
        dzz = zex * (gxize / gzeze * tdx + tdz) + zez * (gxize / gzeze * szdx + szdz);
      }
    }
    const float ir = K(kCRR);
    o.vx = rvx * ir;
    o.vz = rvz * ir;
    if (side) {
      const float4 p = px;
      const float V0 = xa[0], V1 = xa[1];
      o.XV0 = -p.y * V0 + p.x * dxx;
      o.XV1 = -p.y * V1 + p.x * dxz;
      o.vx += ((p.z - 1.0f) * dxx - p.z * V0) * ir;
      o.vz += ((p.z - 1.0f) * dxz - p.z * V1) * ir;
    }
    if (bottom) {
      const float4 p = pz;
      const float V0 = za[0], V1 = za[1];
      o.ZV0 = -p.y * V0 + p.x * dzx;
      o.ZV1 = -p.y * V1 + p.x * dzz;
      o.vx += ((p.z - 1.0f) * dzx - p.z * V0) * ir;
      o.vz += ((p.z - 1.0f) * dzz - p.z * V1) * ir;
    }
  }
  // ---- stress ----
  {
    const float c11 = K(kC11), c13 = K(kC13), c33 = K(kC33), c55 = K(kC55);
    const float dvx_dxi = dx5(kVX), dvz_dxi = dx5(kVZ);
    if (!IN && dist == 0) {
      // traction-free row: the zeta derivatives eliminated through the ALM
      // coefficients (src/elements.cu:907-977)
      const float a0 = __ldg(C.alm + ix), a1 = __ldg(C.alm + P + ix), a2 = __ldg(C.alm + 2 * P + ix),
                  a3 = __ldg(C.alm + 3 * P + ix), a4 = __ldg(C.alm + 4 * P + ix),
                  a5 = __ldg(C.alm + 5 * P + ix);
      o.sx = (c11 * a0 + c13 * a1) * dvx_dxi + (c11 * a3 + c13 * a4) * dvz_dxi;
      o.sz = (c13 * a0 + c33 * a1) * dvx_dxi + (c13 * a3 + c33 * a4) * dvz_dxi;
      o.sxz = c55 * (a2 * dvx_dxi + a5 * dvz_dxi);
      if (side) {
        const float4 p = px;
        const float E0 = xa[2], E1 = xa[3];
        o.XE0 = -p.y * E0 + p.x * dvx_dxi;
        o.XE1 = -p.y * E1 + p.x * dvz_dxi;
        const float cxx_x = c11 * a0 + c13 * a1, cxx_z = c11 * a3 + c13 * a4;
        o.sx += (p.z - 1.0f) * (cxx_x * dvx_dxi + cxx_z * dvz_dxi) - p.z * (cxx_x * E0 + cxx_z * E1);
        const float czz_x = c13 * a0 + c33 * a1, czz_z = c13 * a3 + c33 * a4;
        o.sz += (p.z - 1.0f) * (czz_x * dvx_dxi + czz_z * dvz_dxi) - p.z * (czz_x * E0 + czz_z * E1);
        o.sxz += c55 * ((p.z - 1.0f) * (a2 * dvx_dxi + a5 * dvz_dxi) - p.z * (a2 * E0 + a5 * E1));
      }
      return o;
    }
    const float dvx_dze = dzn(kVX, dist), dvz_dze = dzn(kVZ, dist);
    o.sx = c11 * (xix * dvx_dxi + zex * dvx_dze) + c13 * (xiz * dvz_dxi + zez * dvz_dze);
    o.sz = c13 * (xix * dvx_dxi + zex * dvx_dze) + c33 * (xiz * dvz_dxi + zez * dvz_dze);
    o.sxz = c55 * (xiz * dvx_dxi + zez * dvx_dze + xix * dvz_dxi + zex * dvz_dze);
    if (side) {
      const float Dvx = dvx_dxi + (gxize / gxixi) * dvx_dze, Dvz = dvz_dxi + (gxize / gxixi) * dvz_dze;
      const float4 p = px;
      const float E0 = xa[2], E1 = xa[3], invb = p.z;
      o.XE0 = -p.y * E0 + p.x * Dvx;
      o.XE1 = -p.y * E1 + p.x * Dvz;
      o.sx += c11 * (invb - 1.0f) * xix * Dvx + c13 * (invb - 1.0f) * xiz * Dvz -
              invb * c11 * xix * E0 - invb * c13 * xiz * E1;
      o.sz += c13 * (invb - 1.0f) * xix * Dvx + c33 * (invb - 1.0f) * xiz * Dvz -
              invb * c13 * xix * E0 - invb * c33 * xiz * E1;
      o.sxz += c55 * (invb - 1.0f) * (xiz * Dvx + xix * Dvz) - invb * c55 * xiz * E0 -
               invb * c55 * xix * E1;
    }
    if (bottom) {
      const float Dvx = dvx_dze + (gxize / gzeze) * dvx_dxi, Dvz = dvz_dze + (gxize / gzeze) * dvz_dxi;
      const float4 p = pz;
      const float E0 = za[2], E1 = za[3], invb = p.z;
      o.ZE0 = -p.y * E0 + p.x * Dvx;
      o.ZE1 = -p.y * E1 + p.x * Dvz;
      o.sx += c11 * (invb - 1.0f) * zex * Dvx + c13 * (invb - 1.0f) * zez * Dvz -
              invb * c11 * zex * E0 - invb * c13 * zez * E1;
      o.sz += c13 * (invb - 1.0f) * zex * Dvx + c33 * (invb - 1.0f) * zez * Dvz -
              invb * c13 * zex * E0 - invb * c33 * zez * E1;
      o.sxz += c55 * (invb - 1.0f) * (zez * Dvx + zex * Dvz) - invb * c55 * zez * E0 -
               invb * c55 * zex * E1;
    }
  }
  return o;
}

// The point-wise operands of one cell: U^n or, in the last stage, the
// accumulator (`u`) and the coefficients (`k`).
struct Pt { float u[5], k[kNCoef]; };

template <int KIND>
__device__ __forceinline__ void load_pt(Pt& p, const SCoef& C, const SFields& un,
                                        const SFields& acc, size_t i) {
  const float* const pu = KIND == kStageLast ? acc.vx : un.vx;
  const size_t n = (size_t)C.nz * C.P;  // the five fields lie one after another
#pragma unroll
  for (int q = 0; q < 5; ++q)
    if (KIND != kStageFirst) p.u[q] = (pu + q * n)[i];
}
// The coefficients, which no launch writes.
__device__ __forceinline__ void load_coef(Pt& p, const SCoef& C, size_t i) {
  p.k[kCXIX] = __ldg(C.xix + i);
  p.k[kCXIZ] = __ldg(C.xiz + i);
  p.k[kCZEX] = __ldg(C.zex + i);
  p.k[kCZEZ] = __ldg(C.zez + i);
  p.k[kCRR] = __ldg(C.rcp_rho + i);
  p.k[kC11] = __ldg(C.C11 + i);
  p.k[kC13] = __ldg(C.C13 + i);
  p.k[kC33] = __ldg(C.C33 + i);
  p.k[kC55] = __ldg(C.C55 + i);
}

// The four ADE values of a strip cell: the stage input's (`y`) and U^n's or the
// accumulator's (`u`).
template <int KIND>
__device__ __forceinline__ void load_ade(float* y, float* u, float* const* in, float* const* un,
                                         float* const* acc, size_t i) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    y[q] = in[q][i];
    if (KIND == kStageSecond || KIND == kStageThird) u[q] = un[q][i];
    if (KIND == kStageLast) u[q] = acc[q][i];
  }
}

// RK update of one value from loaded operands.
template <int KIND>
__device__ __forceinline__ void put(float k, float y, float u, float* out, float* acc, size_t i,
                                    float c, float w) {
  if (KIND == kStageFirst) {
    out[i] = fmaf(c, k, y);
  } else if (KIND == kStageLast) {
    out[i] = rk_last(k, y, u, c);
  } else {
    out[i] = fmaf(c, k, u);
    if (KIND == kStageSecond) acc[i] = rk_acc(k, y, u, w);
  }
}

constexpr int kBands = 5;  // free surface, left, right, top (CPML), bottom

struct Args {
  SCoef C;
  SFields in, out, un, acc;
  int s;
  Band edge[kBands];  // 8 rows each
  Band inner;         // `tr` rows
  int tr;
  float c, w;
};

// One tile. SURF, PML as in rhs(); neither: an interior tile, a thread takes
// every kRowStep-th row of its column.
template <int DIR, int KIND, bool SURF, bool PML, bool CPML>
__device__ __forceinline__ void run_tile(const Args& a, const Tile& tl, float* tile) {
  const SCoef& C = a.C;
  const int nx = C.nx, nz = C.nz, npd = C.npd, P = C.P;
  const size_t n = (size_t)nz * P;
  const int ty = threadIdx.x / kTX, tx = threadIdx.x % kTX, ix = tl.x0 + tx;
  constexpr int LO = !SURF && DIR == kDirF ? 1 : 3, HI = !SURF && DIR == kDirB ? 1 : 3;
  int iz = tl.z0 + ty;
  const bool active = ix < tl.x1 && (!PML || ix >= 3) && iz < tl.z1;
  Pt p;
  if (active) load_coef(p, C, (size_t)iz * P + ix);
  const bool side = PML && active && min(ix - 3, nx - 4 - ix) < npd;
  const bool band = PML && active && (iz >= nz - 3 - npd || (CPML && iz <= npd + 2));
  const size_t si = (size_t)iz * C.Ps + (side ? xstrip_col(ix, nx, npd) : 0);
  const size_t zi = (size_t)zeta_row<CPML>(iz, nz, npd) * P + ix;
  float xa[4], ux[4], za[4], uz[4];
  float4 px = make_float4(0.f, 0.f, 0.f, 0.f), pz = px;
  const int2 src = __ldg(C.src_pos);
  // the source's 5x5 cells touch this tile
  const bool near_src = src.x >= 0 && src.x >= tl.x0 - 2 && src.x < tl.x0 + kTX + 2 &&
                        src.y >= tl.z0 - 2 && src.y < tl.z1 + 2;
  if (side) px = __ldg(C.pmlx + ix);
  if (band) pz = __ldg(C.pmlz + iz);
  wait_previous();
  stage_tile<5, LO, HI>(tile, a.in.vx, n, tl.x0, tl.z0, PML ? kRowStep : a.tr, nz, P);
  if (active) load_pt<KIND>(p, C, a.un, a.acc, (size_t)iz * P + ix);
  if (side) load_ade<KIND>(xa, ux, a.in.x, a.un.x, a.acc.x, si);
  if (band) load_ade<KIND>(za, uz, a.in.z, a.un.z, a.acc.z, zi);
  cp_async_wait_all();
  launch_dependents();
  __syncthreads();
  if (!active) return;
#pragma unroll 1
  for (;;) {
    const size_t i = (size_t)iz * P + ix;
    const TileAcc<5> T(tile, 3 + iz - tl.z0, 4 + tx);
    auto A = [&](int q, int dz, int dx) { return T.at(q, dz, dx); };
    auto K = [&](int cf) { return p.k[cf]; };
    Out o = rhs<DIR, SURF, PML, CPML>(C, A, K, iz, ix, side, band, xa, za, px, pz);
    if (near_src) {
      // explosive source on both normal stresses (src/pml_fs_kernels.cu:22-26)
      const int it = (C.step ? __ldg(C.step) : 0) + C.it_off, sx = ix - src.x, sz = iz - src.y;
      if (sx >= -2 && sx <= 2 && sz >= -2 && sz <= 2 && it >= 0 && it < C.src_steps) {
        const float q = __ldg(C.src_amp + (size_t)it * 4 + a.s) * c_srcw[(sz + 2) * 5 + (sx + 2)];
        o.sx += q;
        o.sz += q;
      }
    }
    const float k[5] = {o.vx, o.vz, o.sx, o.sz, o.sxz};
#pragma unroll
    for (int q = 0; q < 5; ++q)
      put<KIND>(k[q], T.at(q, 0, 0), p.u[q], a.out.vx + q * n, a.acc.vx + q * n, i, a.c, a.w);
    if (PML) {
      const float kx[4] = {o.XV0, o.XV1, o.XE0, o.XE1}, kz[4] = {o.ZV0, o.ZV1, o.ZE0, o.ZE1};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (side) put<KIND>(kx[q], xa[q], ux[q], a.out.x[q], a.acc.x[q], si, a.c, a.w);
        if (band) put<KIND>(kz[q], za[q], uz[q], a.out.z[q], a.acc.z[q], zi, a.c, a.w);
      }
    }
    if (KIND == kStageLast && iz == C.rec_row) {  // the receiver row (src/main.cu:284-311)
      const float v = rk_last(k[kVZ], T.at(kVZ, 0, 0), p.u[kVZ], a.c);
      const int it = (C.step ? __ldg(C.step) : 0) + C.it_off, j = C.gap > 0 ? it / C.gap : 0;
      if (!isfinite(v)) atomicOr(C.status, 1);
      if (C.rec != nullptr && C.gap > 0 && j * C.gap == it && j < C.rec_cap)
        C.rec[(size_t)j * nx + ix] = v;
    }
    if (PML) return;
    iz += kRowStep;
    if (iz >= tl.z1) return;
    load_coef(p, C, (size_t)iz * P + ix);
    load_pt<KIND>(p, C, a.un, a.acc, (size_t)iz * P + ix);
  }
}

template <int MINB, int DIR, int KIND, bool CPML>
__global__ void __launch_bounds__(kThreads, MINB) k_stage(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) float tile[];
  const int b = blockIdx.x;
  if (b >= a.inner.first) {
    run_tile<DIR, KIND, false, false, CPML>(a, tile_of(a.inner, b, a.tr), tile);
  } else if (!CPML && b < a.edge[1].first) {
    run_tile<DIR, KIND, true, true, CPML>(a, tile_of(a.edge[0], b, kRowStep), tile);
  } else {
    int k = 1;
#pragma unroll
    for (int q = 2; q < kBands; ++q)
      if (b >= a.edge[q].first) k = q;
    run_tile<DIR, KIND, false, true, CPML>(a, tile_of(a.edge[k], b, kRowStep), tile);
  }
}

__global__ void k_set_step(int* step, int it) { *step = it; }
__global__ void k_advance_step(int* step, int n) { *step += n; }

template <int MINB, int DIR, int KIND>
cudaError_t launch_t(const SCoef& C, const SFields& in, const SFields& out, const SFields& un,
                     const SFields& acc, cudaStream_t st) {
  Args a;
  a.C = C; a.in = in; a.out = out; a.un = un; a.acc = acc;
  a.s = KIND;
  a.c = C.rk_c[KIND];
  a.w = KIND == kStageSecond ? C.rk_w : 0.f;
  const int nx = C.nx, nz = C.nz, npd = C.npd;
  // tall tiles stage fewer halo rows, short ones give a small grid enough blocks
  // (us a step at 8 / 16 / 24 / 32 rows: 200x200 19.2 / 19.6 / 19.6 / 19.7, 600x600
  // 37.2 / 35.1 / 37.2 / 37.7, 2048x2048 328 / 314 / 307 / 312)
  a.tr = MINB == 5 ? 3 * kRowStep : (long long)nx * nz < 100000 ? kRowStep : 2 * kRowStep;
  // rows 3..nz-4: 8 rows under the free surface, the bottom band (and the top
  // band with CPML); columns 3..nx-4: the side strips in whole tile columns
  const int z0 = C.cpml ? 3 : std::min(3 + kRowStep, nz - 3), z1 = nz - 3;
  int xl = std::min(ceil_div(3 + npd, kTX) * kTX, nx - 3), xr = std::max((nx - 3 - npd) / kTX * kTX, xl);
  if (xr - xl < 4) xl = xr = nx - 3;  // no interior columns: all in the left band
  const int zt = C.cpml ? std::min(std::max(npd + 3, z0), z1) : z0;
  const int zb = std::min(std::max(nz - 3 - npd, zt), z1);
  int n = make_band(a.edge[0], 0, nx - 3, 3, z0, kRowStep, 0);
  n = make_band(a.edge[1], 0, xl, z0, z1, kRowStep, n);
  n = make_band(a.edge[2], xr, nx - 3, z0, z1, kRowStep, n);
  n = make_band(a.edge[3], xl, xr, z0, zt, kRowStep, n);
  n = make_band(a.edge[4], xl, xr, zb, z1, kRowStep, n);
  n = make_band(a.inner, xl, xr, zt, zb, a.tr, n);
  return C.cpml ? launch_tiles(k_stage<MINB, DIR, KIND, true>, a, n, tile_smem(a.tr), C.chain != 0, st)
                : launch_tiles(k_stage<MINB, DIR, KIND, false>, a, n, tile_smem(a.tr), C.chain != 0, st);
}

template <int MINB, int DIR>
cudaError_t launch_d(const SCoef& C, const SFields& in, const SFields& out, const SFields& un,
                     const SFields& acc, int stage, cudaStream_t st) {
  switch (stage) {
    case 0: return launch_t<MINB, DIR, kStageFirst>(C, in, out, un, acc, st);
    case 1: return launch_t<MINB, DIR, kStageSecond>(C, in, out, un, acc, st);
    case 2: return launch_t<MINB, DIR, kStageThird>(C, in, out, un, acc, st);
    default: return launch_t<MINB, DIR, kStageLast>(C, in, out, un, acc, st);
  }
}

}  // namespace

cudaError_t launch_stage(const SCoef& C, const SFields& in, const SFields& out, const SFields& un,
                         const SFields& acc, int stage, int dir, cudaStream_t st) {
  // Small grids are one wave or two, bound by the latency of a block, and take the
  // larger register budget; large ones are bound by memory and take more blocks
  // per SM (us a step, 3 / 5 blocks: 400x400 23.0 / 30.0, 600x600 35.1 / 40.8,
  // 800x800 56.6 / 54.6, 1000x1000 104 / 100, 2048x2048 343 / 307, 4096x4096
  // 1253 / 1068).
  if ((long long)C.nx * C.nz < 600000)
    return dir == kDirF ? launch_d<3, kDirF>(C, in, out, un, acc, stage, st)
                        : launch_d<3, kDirB>(C, in, out, un, acc, stage, st);
  return dir == kDirF ? launch_d<5, kDirF>(C, in, out, un, acc, stage, st)
                      : launch_d<5, kDirB>(C, in, out, un, acc, stage, st);
}

cudaError_t launch_set_step(const SCoef& C, int it, cudaStream_t st) {
  k_set_step<<<1, 1, 0, st>>>(C.step, it);
  return cudaGetLastError();
}

cudaError_t launch_advance_step(const SCoef& C, int n, cudaStream_t st) {
  k_advance_step<<<1, 1, 0, st>>>(C.step, n);
  return cudaGetLastError();
}

}  // namespace solid
}  // namespace mfdm
