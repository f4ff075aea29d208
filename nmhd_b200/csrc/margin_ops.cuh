// Margin fill and CFL-time operations shared by the single-box kernels
// (step.cu) and the batched-ensemble kernels (batch.cu).
#pragma once
#include <cuda_runtime.h>

#include "step.cuh"

namespace nmhd {
namespace margin {

__device__ __forceinline__ int wrap(int v, int s) {
  while (v < 0) v += s;
  while (v >= s) v -= s;
  return v;
}

// CFL time of a cell (cfl_condition_inner/kernel,
// src/library/mhd_solver.inlrb:496-521): min over axes of
// cfl*d / |v_d + sqrt((gamma p + b2)/rho)|, b2 = sum of max(B_lo^2, B_hi^2),
// from its 8 fields and the B of its upper faces.
__device__ __forceinline__ float cfl_time(const GridParams &g, const float u[8], float bxh, float byh, float bzh) {
  const float b2 = fmaxf(u[5] * u[5], bxh * bxh) + fmaxf(u[6] * u[6], byh * byh) + fmaxf(u[7] * u[7], bzh * bzh);
  const float c = sqrtf((g.gamma * u[4] + b2) / u[0]);
  const float tx = g.cfl * g.dx / fabsf(u[1] + c);
  const float ty = g.cfl * g.dy / fabsf(u[2] + c);
  const float tz = g.cfl * g.dz / fabsf(u[3] + c);
  return fminf(fminf(tx, ty), tz);
}

__device__ __forceinline__ float cfl_of_cell(const GridParams &g, const float *w, int x, int y, int z) {
  const size_t N = (size_t)g.n;
  const int o = (z * g.sy + y) * g.sx + x;
  const int oxp = (z * g.sy + y) * g.sx + wrap(x + 1, g.sx);
  const int oyp = (z * g.sy + wrap(y + 1, g.sy)) * g.sx + x;
  const int ozp = (wrap(z + 1, g.sz) * g.sy + y) * g.sx + x;
  float u[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) u[v] = w[v * N + o];
  return cfl_time(g, u, w[5 * N + oxp], w[6 * N + oyp], w[7 * N + ozp]);
}

// Number of cells whose CFL time the margin pass covers: the Y-margin rows, and
// with Z margins the Z-margin planes plus the last interior plane (its upper
// z-face is rewritten by the Z copy).  The final stage covers all other cells.
__device__ __host__ __forceinline__ long long margin_cfl_cells(const GridParams &g) {
  return 2LL * g.my * g.sx * g.sz + (g.mz > 0 ? (2LL * g.mz + 1) * g.sx * g.sy : 0);
}

__device__ __forceinline__ void margin_cfl_cell(const GridParams &g, int idx, int *x, int *y, int *z) {
  const int part_a = 2 * g.my * g.sx * g.sz;
  if (idx < part_a) {
    *x = idx % g.sx;
    const int r = (idx / g.sx) % (2 * g.my);
    *z = idx / (g.sx * 2 * g.my);
    *y = r < g.my ? r : g.sy - 2 * g.my + r;
  } else {
    const int j = idx - part_a;
    *x = j % g.sx;
    *y = (j / g.sx) % g.sy;
    const int p = j / (g.sx * g.sy);
    *z = p < g.mz ? p : g.sz - g.mz - 1 + (p - g.mz);
  }
}

// Integer and fractional shear displacement of the Y-margin exchange at time t
// (relative_displacement, src/library/mhd_solver.inlrb:244-259): all double
// except the float product fold * kExtentX.
struct ShearShift {
  int dint;
  float f;
};
__device__ __forceinline__ ShearShift shear_shift(const GridParams &g, double time) {
  const double d0 = 0.0 + time * g.rel_vel;
  const int fold = (int)floor(d0 / (double)g.extent_x);
  const double d1 = d0 - (double)((float)fold * g.extent_x);
  ShearShift s;
  s.dint = (int)floor(d1 / (double)g.dx);
  s.f = (float)(d1 / (double)g.dx - s.dint);
  return s;
}

// Gather half of the Y-margin exchange for item idx = (sz*M + sy)*Sx + sx,
// sy < M (communicate_gather_kernel_y, mhd_solver.inlrb:184-222): field v of
// the top interior row Sy-2M+sy shifted by +d_int in x with vx -
// relative_velocity (`inc`, sent to the rank above) and of the bottom interior
// row M+sy shifted by -d_int-1 with vx + relative_velocity (`dec`, sent to the
// rank below).  The reference's two-point interpolation weights both multiply
// the same sample; that arithmetic is kept.
__device__ __forceinline__ void gather_y_item(const GridParams &g, const ShearShift &sh, const float *w,
                                              int idx, float inc[8], float dec[8]) {
  const int M = g.my;
  const int sx = idx % g.sx;
  const int sy = (idx / g.sx) % M;
  const int sz = idx / (g.sx * M);
  const float rv = (float)g.rel_vel;
  const int inc_x = wrap((sx + sh.dint) % g.sx, g.sx);
  const int dec_x = wrap((sx - sh.dint - 1) % g.sx, g.sx);
  const size_t N = (size_t)g.n;
  const int src_inc = (sz * g.sy + (g.sy - 2 * M + sy)) * g.sx + inc_x;
  const int src_dec = (sz * g.sy + (M + sy)) * g.sx + dec_x;
  const float omf = 1.0f - sh.f;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const float vi = w[v * N + src_inc];
    const float vd = w[v * N + src_dec];
    float bi = omf * vi + sh.f * vi;
    float bd = sh.f * vd + omf * vd;
    if (v == 1) {
      bi = bi - rv;
      bd = bd + rv;
    }
    inc[v] = bi;
    dec[v] = bd;
  }
}

// Scatter half (communicate_scatter_kernel_y, mhd_solver.inlrb:224-242): the
// bottom margin row sy takes `inc` (from the rank below), the top margin row
// Sy-M+sy takes `dec` (from the rank above); By of row Sy-M (the interior's
// upper face) is kept.
__device__ __forceinline__ void scatter_y_item(const GridParams &g, float *w, int idx, const float inc[8],
                                               const float dec[8]) {
  const int M = g.my;
  const int sx = idx % g.sx;
  const int sy = (idx / g.sx) % M;
  const int sz = idx / (g.sx * M);
  const size_t N = (size_t)g.n;
  const int dst_lo = (sz * g.sy + sy) * g.sx + sx;
  const int dst_hi = (sz * g.sy + (g.sy - M + sy)) * g.sx + sx;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    w[v * N + dst_lo] = inc[v];
    if (!(v == 6 && sy == 0)) w[v * N + dst_hi] = dec[v];
  }
}

// One item of the shearing-periodic Y-margin fill of a single box (one rank:
// every message of the exchange goes to itself).  Reads only interior rows and
// writes only margin rows, so it runs in place.
__device__ __forceinline__ void fill_y_item(const GridParams &g, double time, float *w, int idx) {
  float inc[8], dec[8];
  gather_y_item(g, shear_shift(g, time), w, idx, inc, dec);
  scatter_y_item(g, w, idx, inc, dec);
}

// A box's fields as the margin fill leaves them, read from the state before
// it: the Z copy of the Y-filled planes, each margin cell the image of one
// interior cell.  The values are fill_y_item()'s and the Z copy's; only cells
// that the fill does not write are read.
struct Filled {
  const GridParams &g;
  const float *w;
  ShearShift sh;
  float omf, rv;
  __device__ __forceinline__ Filled(const GridParams &g_, const float *w_, const ShearShift &sh_)
      : g(g_), w(w_), sh(sh_), omf(1.0f - sh_.f), rv((float)g_.rel_vel) {}
  // Source cell of (x, y, z) as the Z copy and the shear shift map it; `row`
  // is -1, 0 or 1 for a bottom margin row, an interior row or a top margin row.
  __device__ __forceinline__ int source(int x, int y, int z, int *row) const {
    if (z < g.mz) z += g.sz - 2 * g.mz;
    else if (z >= g.sz - g.mz) z -= g.sz - 2 * g.mz;
    *row = y < g.my ? -1 : y >= g.sy - g.my ? 1 : 0;
    if (*row < 0) {
      x = wrap((x + sh.dint) % g.sx, g.sx);
      y += g.sy - 2 * g.my;
    } else if (*row > 0) {
      x = wrap((x - sh.dint - 1) % g.sx, g.sx);
      y -= g.sy - 2 * g.my;
    }
    return (z * g.sy + y) * g.sx + x;
  }
  __device__ __forceinline__ float value(int v, int src, int row) const {
    const float u = w[(size_t)v * g.n + src];
    if (row == 0) return u;
    float b = row < 0 ? omf * u + sh.f * u : sh.f * u + omf * u;
    if (v == 1) b = row < 0 ? b - rv : b + rv;
    return b;
  }
  // By of row Sy-M, the upper face of the interior, is kept by the fill.
  __device__ __forceinline__ float by(int x, int y, int z) const {
    int row, src = source(x, y, z, &row);
    if (y == g.sy - g.my && row > 0) {
      int zs = z < g.mz ? z + g.sz - 2 * g.mz : z >= g.sz - g.mz ? z - (g.sz - 2 * g.mz) : z;
      return w[(size_t)6 * g.n + (zs * g.sy + y) * g.sx + x];
    }
    return value(6, src, row);
  }
  __device__ __forceinline__ float at(int v, int x, int y, int z) const {
    int row, src = source(x, y, z, &row);
    return value(v, src, row);
  }
};

// Fills cell idx of the margin CFL set (margin_cfl_cell()) and returns its CFL
// time: the fill and margin CFL passes in one.  Y-margin rows come first in
// the set, so a cell of a Z-margin plane that lies in one is left to them.
__device__ __forceinline__ float fill_cfl_item(const GridParams &g, const ShearShift &sh, float *w, int idx) {
  int x, y, z;
  margin_cfl_cell(g, idx, &x, &y, &z);
  const bool yrow = y < g.my || y >= g.sy - g.my;
  if (yrow && idx >= 2 * g.my * g.sx * g.sz) return __uint_as_float(0x7f800000u);
  const Filled F(g, w, sh);
  const size_t N = (size_t)g.n;
  const int xp = x + 1 < g.sx ? x + 1 : 0, yp = y + 1 < g.sy ? y + 1 : 0, zp = z + 1 < g.sz ? z + 1 : 0;
  int row;
  const int src = F.source(x, y, z, &row);
  float u[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) u[v] = v == 6 ? F.by(x, y, z) : F.value(v, src, row);
  const float bxh = F.at(5, xp, y, z), byh = F.by(x, yp, z), bzh = F.at(7, x, y, zp);
  if (yrow || z < g.mz || z >= g.sz - g.mz) {
    float *dst = w + (z * g.sy + y) * g.sx + x;
    const bool kept = y == g.sy - g.my && z >= g.mz && z < g.sz - g.mz;  // By of the interior's upper face
#pragma unroll
    for (int v = 0; v < 8; ++v)
      if (!(v == 6 && kept)) dst[v * N] = u[v];
  }
  return cfl_time(g, u, bxh, byh, bzh);
}

}  // namespace margin
}  // namespace nmhd
