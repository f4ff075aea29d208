// Face fluxes of a 32 x 4 x 2-cell tile from a shared-memory copy of the
// stage input (kernel variant 5's flux kernel).
//
// The per-cell flux kernel reads its 40-odd stencil values per face from
// global memory, and each read costs a 64-bit address computed from the
// cell's wrapped neighbour offsets: on the 128x256x64 shearing box a fifth of
// its instructions are integer address arithmetic.  Here the tile first
// copies all 8 fields of the cells x0-2..x0+32, y0-2..y0+4, z0-2..z0+2 (the
// union of the three axes' 4-cell stencils and the +1 transverse neighbours
// of the face-centred B) into shared memory, with one tensor copy for tiles
// away from the box's y and z edges; every stencil read is then a shared load
// at a constant offset.  The fluxes are bitwise face_flux()'s: the quotients
// and roots are correctly rounded in both, here by shared reciprocals where the
// operands are in their range (rounded.cuh), else by the plain operations.
#pragma once
#include "cell_epilogue.cuh"

namespace nmhd {
namespace cell {
namespace sfx {

// Staged box: rows of P = 40 floats starting at the 16-byte aligned x0 - 4
// (x0 at row position 4), NJ = 7 rows (y0-2..y0+4) per plane, NK = 5 planes
// (z0-2..z0+2), the 8 fields FS floats apart.
constexpr int P = 40, NJ = 7, NK = 5, XO = 4;
constexpr int kReadBegin = XO - 2, kReadEnd = XO + BX + 1;  // row positions that are read (x0-2..x0+32)
constexpr int DY = P, DZ = P * NJ, FS = P * NJ * NK;
constexpr unsigned kTxBytes = 4u * 8u * FS;

struct __align__(128) Smem {
  float w[8 * FS];
  int gy[NJ], gz[NK];  // wrapped global offsets of (y0-2+j)*Sx, (z0-2+k)*Sx*Sy
  unsigned long long mbar;
};

// Tensor maps (4-D: x, y, z, field) of the staged box over each state buffer
// (0 w0, 1 w1, 2 predictor); `enabled` 0 where they cannot be made.
struct FluxMaps {
  CUtensorMap w[3];
  int enabled;
};

// Shared index of tile-local cell (a, b, c).
__device__ __forceinline__ int at(int a, int b, int c) { return ((c + 2) * NJ + (b + 2)) * P + XO + a; }

// The staged rows by W-float asynchronous copies (Sx % W == 0), the tile's
// threads over all (row, chunk) pairs of the positions that are read
// (x0-2..x0+32); a chunk beyond an x edge of the box is the (still aligned)
// chunk Sx away.  A flux launch of a 250x97x61 box took 169 us with 4-byte
// copies a row to a warp, 142 us so; of a 251x97x61 box 156 us.
template <int W>
__device__ __forceinline__ void copy_rows(const Smem &s, int nx, const float *__restrict__ w, size_t N, unsigned ds,
                                          int x0, int tid) {
  using Chunks = RowChunks<kReadBegin, kReadEnd, W>;
  static_assert(Chunks::first + W * Chunks::count <= P, "row length");
  for (int e = tid; e < NJ * NK * Chunks::count; e += kThreads) {
    const int r = e / Chunks::count, pos = Chunks::first + W * (e - r * Chunks::count);
    const float *src = w + (s.gz[r / NJ] + s.gy[r % NJ] + row_column<W>(x0 - XO + pos, nx));
    const unsigned d = ds + 4u * (r * P + pos);
#pragma unroll
    for (int f = 0; f < 8; ++f) epi::cp_async<W>(d + 4u * (f * FS), src + f * N);
  }
}

// What staged row e (field, z, y) holds beyond the x edges of the box: cells
// Sx-2 and Sx-1 before the first column, cell 0 after the last.  Of tiles whose
// rows and planes lie inside the box.
constexpr int kRows = 8 * NJ * NK;
static_assert(kRows <= 2 * kThreads, "two rows a thread");
struct Wrapped {
  float l2, l1, h;
};
__device__ __forceinline__ Wrapped wrapped_columns(const GridParams &g, const float *__restrict__ w, bool low,
                                                   bool high, int y0, int z0, int e) {
  const int f = e / (NJ * NK), r = e - f * (NJ * NK);
  const float *row = w + f * (size_t)g.n + ((z0 - 2 + r / NJ) * g.sy + (y0 - 2 + r % NJ)) * g.sx;
  Wrapped v = {};
  if (low) v.l2 = __ldg(row + g.sx - 2), v.l1 = __ldg(row + g.sx - 1);
  if (high) v.h = __ldg(row);
  return v;
}

// Copies the stage input w around tile (x0, y0, z0) into s.w.  Tiles whose rows
// and planes lie inside the box: one tensor copy issued by thread 0, completing
// on the mbarrier (bounded wait; false if it timed out); beyond an x edge it
// leaves zeros, and the columns there that are read are put in by single loads
// (tiles at x edges by 16-byte copies: 162 us a launch on the 256x128x64 box, so
// 156; 31.2 -> 29.2 us on 64^3, where every tile is at one).  Others: cp.async through
// the wrapped offset tables, in the widest row chunks that Sx is a multiple of
// (16, 8 or 4 bytes).  Every thread of the CTA calls it.  kOnce: the CTA stages no other
// tile, so a thread goes on when it has seen the copy land (and the answer is
// the thread's own).
template <bool kOnce = false>
__device__ __forceinline__ bool stage(Smem &s, const GridParams &g, const FluxMaps *maps, int buf,
                                      const float *__restrict__ w, int x0, int y0, int z0, int tid) {
  const size_t N = (size_t)g.n;
  const unsigned ds = (unsigned)__cvta_generic_to_shared(s.w), mb = (unsigned)__cvta_generic_to_shared(&s.mbar);
  const bool tma = maps && maps->enabled && y0 >= 2 && y0 + 5 <= g.sy && z0 >= 2 && z0 + 3 <= g.sz;
  if (tma) {
    const bool low = x0 == 0, high = x0 + BX >= g.sx;
    Wrapped wr[2];
    if (low || high) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (tid + i * kThreads < kRows) wr[i] = wrapped_columns(g, w, low, high, y0, z0, tid + i * kThreads);
    }
    auto patch = [&] {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int e = tid + i * kThreads;
        if (e >= kRows) break;
        float *row = s.w + e * P + XO;
        if (low) row[-2] = wr[i].l2, row[-1] = wr[i].l1;
        if (high) row[g.sx - x0] = wr[i].h;
      }
      __syncthreads();
    };
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(kTxBytes) : "memory");
      asm volatile(
          "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
          "%4, %5}], [%6];" ::"r"(ds),
          "l"(reinterpret_cast<unsigned long long>(&maps->w[buf])), "r"(x0 - XO), "r"(y0 - 2), "r"(z0 - 2), "r"(0),
          "r"(mb)
          : "memory");
    }
    __syncthreads();
    // (a second bounded wait where the first gives up: no copy may still be
    // writing when the CTA exits)
    if (kOnce) {
      const bool ok = epi::mbar_wait_bounded(mb) || (epi::mbar_wait_bounded(mb), false);
      if (low || high) patch();
      return ok;
    }
    const bool ok = __syncthreads_and(epi::mbar_wait_bounded(mb));
    if (!ok) {
      // flag it and wait once more (bounded) so that no copy is still
      // writing when the CTA exits
      epi::mbar_wait_bounded(mb);
      __syncthreads();
      if (tid == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(mb) : "memory");
      return false;
    }
    if (tid == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(mb) : "memory");
    if (low || high) patch();
    return true;
  }
  if (tid < NJ) s.gy[tid] = wrap_any(y0 - 2 + tid, g.sy) * g.sx;
  else if (tid < NJ + NK) s.gz[tid - NJ] = wrap_any(z0 - 2 + (tid - NJ), g.sz) * g.sx * g.sy;
  __syncthreads();
  if ((g.sx & 3) == 0) copy_rows<4>(s, g.sx, w, N, ds, x0, tid);
  else if ((g.sx & 1) == 0) copy_rows<2>(s, g.sx, w, N, ds, x0, tid);
  else copy_rows<1>(s, g.sx, w, N, ds, x0, tid);
  epi::cp_async_wait_all();
  __syncthreads();
  return true;
}

// The states on either side of a face from the cells' values x0..x3, and from
// sums of two values, which halve exactly where q.slope() holds.
template <class Q>
__host__ __device__ __forceinline__ void face_states(Q &q, const float x[4], float &l, float &r) {
  reconstruct4_with(q, x[0], x[1], x[2], x[3], l, r);
}
template <class Q>
__host__ __device__ __forceinline__ void face_means(Q &q, const float s[4], float &l, float &r) {
  reconstruct4_with(q, s[0], s[1], s[2], s[3], l, r);
  l *= 0.5f;
  r *= 0.5f;
}
#if NMHD_FAST_ARITH
// The fast-arithmetic kernel keeps face_input()'s and hlld_flux_plain()'s
// operations as they stand, so that runs of that mode keep their bits.  With
// products by shared approximate reciprocals and the three-instruction limiter a
// launch took 122 us instead of 141 (256x128x64 box): as near to an FP64 run (one
// step of six boxes, five seeds each: the same error to three digits), but another
// result, 4.7e-4 away after 16 steps.
struct AsCompiled {};
__device__ __forceinline__ void face_states(AsCompiled, const float x[4], float &l, float &r) {
  reconstruct4(x[0], x[1], x[2], x[3], l, r);
}
__device__ __forceinline__ void face_means(AsCompiled, const float s[4], float &l, float &r) {
  reconstruct4(0.5f * s[0], 0.5f * s[1], 0.5f * s[2], 0.5f * s[3], l, r);
}
#endif

// face_input() from the shared copy for the lower AX-face of cell index ci, in
// the arithmetic Q.  With the axis a constant every shared read is at a
// constant offset from the cell's address.
template <int AX, class Q>
__device__ __forceinline__ HlldIn staged_input(Q &q, const GridParams &g, bool order2, const float *w, int ci,
                                               int yidx, float half_dt) {
  constexpr int E1 = (AX + 1) % 3, E2 = (AX + 2) % 3;
  constexpr int stride[3] = {1, DY, DZ};
  constexpr int sa = stride[AX], t1 = stride[E1], t2 = stride[E2];
  const float *c = w + ci;
  HlldIn in;
  // density and pressure are checked to be at least 2^-40, so their slopes are
  // 0 or far above the least and need no check
  auto pair = [&](int f, auto &&checks, float &l, float &r) {
    const float *p = c + f * FS;
    const float x[4] = {p[-2 * sa], p[-sa], p[0], p[sa]};
    if (order2) face_states(checks, x, l, r);
    else l = x[1], r = x[2];
  };
  auto field = [&](int f, int t, float &l, float &r) {
    const float *p = c + f * FS;
    const float s[4] = {p[-2 * sa] + p[t - 2 * sa], p[-sa] + p[t - sa], p[0] + p[t], p[sa] + p[t + sa]};
    if (order2) face_means(q, s, l, r);
    else l = 0.5f * s[1], r = 0.5f * s[2];
  };
#if NMHD_FAST_ARITH
  Q &unchecked = q;
#else
  Ieee unchecked;
#endif
  pair(0, unchecked, in.dl, in.dr);
  pair(1 + AX, q, in.ul, in.ur);
  pair(1 + E1, q, in.vl, in.vr);
  pair(1 + E2, q, in.wl, in.wr);
  pair(4, unchecked, in.pl, in.pr);
  field(5 + E1, t1, in.byl, in.byr);
  field(5 + E2, t2, in.bzl, in.bzr);
  if (AX < 2 && g.shear) {
    // face-centred Kepler acceleration (from v_y at x-faces, v_x at y-faces),
    // half a stage kick on the normal velocity
    const float *p = c + (AX == 0 ? 2 : 1) * FS;
    const float v = 0.5f * (p[-sa] + p[0]);
    float acc;
    if (AX == 0) {
      acc = -2.0f * g.omega * v;
    } else {
      const float tide = 2.0f * g.q * (g.omega * g.omega), at = g.corner_y + g.dy * ((float)yidx + 0.5f);
#if NMHD_FAST_ARITH
      acc = fmaf(tide, at, 2.0f * g.omega * v);  // contracted so, whatever the compiler would choose
#else
      acc = 2.0f * g.omega * v + tide * at;
#endif
    }
    const float mbv = half_dt * acc;
    in.ul += mbv;
    in.ur += mbv;
  }
  return in;
}

// The lower faces along axes ax0..ax1-1 of cell ci in the plain arithmetic: a call,
// so that its registers and code stay out of the loop that seldom needs it.
static __device__ __noinline__ void plain_faces(const GridParams &g, const float *w, float *flux, int ci, int ax0,
                                                int ax1, int o, int yidx, float half_dt) {
#pragma unroll 1
  for (int ax = ax0; ax < ax1; ++ax) {
    const int sa = ax == 0 ? 1 : ax == 1 ? DY : DZ;
    const int t1 = ax == 0 ? DY : ax == 1 ? DZ : 1, t2 = ax == 0 ? DZ : ax == 1 ? 1 : DY;
    float f[7];
    hlld_flux_plain(g.gamma, w[(5 + ax) * FS + ci],
                    face_input<SharedLd>(g, w, FS, ci, ax, -2 * sa, -sa, sa, t1, t2, yidx, 2.0f * half_dt), f);
    float *out = flux + (size_t)(7 * ax) * g.n + o;
#pragma unroll
    for (int k = 0; k < 7; ++k) out[(size_t)k * g.n] = f[k];
  }
}

// The lower-face fluxes along axes ax0..ax1-1 of tile-local cell (a, b, c) at
// global (x, y, z), from the staged copy: flux_cell()'s values.  The loop over the axes holds
// one Riemann solver (three overflow the instruction caches) and a branch per
// axis that reads its input: with the axis a run-time number in the input too,
// a tenth of the instructions made addresses.  256x128x64 box: 1,912 warp
// instructions for a warp's three faces (2,293 before), 162 us a launch (181; 154
// now that the tiles at x edges are staged by tensor copies too),
// 72 % of the issue slots filled.  Four CTAs/SM hide the start and the staging
// of a tile better than one persistent CTA of 1,024 threads with a ring of five
// copies (201 us: its spills miss the small L1 that is left) or a stagger of
// the first CTAs (172 us).
__device__ __forceinline__ void flux_cell_order(const GridParams &g, bool order2, const float *w,
                                                float *__restrict__ flux, int ci, unsigned o, int y, float dt, int ax0,
                                                int ax1) {
  const size_t N = (size_t)g.n;
  const float half_dt = 0.5f * dt;
#if !NMHD_FAST_ARITH
  const bool ranged = g.gm1_ranged &&
                      likely_in_range(w[ci], w[4 * FS + ci], w[5 * FS + ci], w[6 * FS + ci], w[7 * FS + ci]);
#endif
#pragma unroll 1
  for (int ax = ax0; ax < ax1; ++ax) {
    // field k: uniform base, 32-bit byte offset of the cell (at most 2^28 cells)
    char *base = reinterpret_cast<char *>(flux + (size_t)(7 * ax) * N);
    auto out = [&](int k, float v) { *reinterpret_cast<float *>(base + k * (4 * N) + 4u * o) = v; };
    const float bn = w[(5 + ax) * FS + ci];
    auto input = [&](auto &q) {
      return ax == 0   ? staged_input<0>(q, g, order2, w, ci, y, half_dt)
             : ax == 1 ? staged_input<1>(q, g, order2, w, ci, y, half_dt)
                       : staged_input<2>(q, g, order2, w, ci, y, half_dt);
    };
#if NMHD_FAST_ARITH
    AsCompiled q;
    float f[7];
    hlld_flux_plain(g.gamma, bn, input(q), f);
#pragma unroll
    for (int k = 0; k < 7; ++k) out(k, f[k]);
#else
    bool ok = false;
    if (ranged) {
      Ranged q;
      const HlldIn in = input(q);
      ok = hlld_flux_with(q, g.gamma, g.gm1, bn, in, out);
    }
    if (!ok) {
      // the cell's other faces too: where one is out of range they mostly are
      plain_faces(g, w, flux, ci, ax, ax1, (int)o, y, half_dt);
      return;
    }
#endif
  }
}

__device__ __forceinline__ void flux_cell_staged(const GridParams &g, const float *w, float *__restrict__ flux,
                                                 int a, int b, int c, int x, int y, int z, float dt, int ax0 = 0,
                                                 int ax1 = 3) {
  const unsigned o = (unsigned)((z * g.sy + y) * g.sx + x);
#if NMHD_FAST_ARITH
  flux_cell_order(g, g.order2, w, flux, at(a, b, c), o, y, dt, ax0, ax1);
#else
  // the order a constant in each of two copies of the code
  if (g.order2) flux_cell_order(g, true, w, flux, at(a, b, c), o, y, dt, ax0, ax1);
  else flux_cell_order(g, false, w, flux, at(a, b, c), o, y, dt, ax0, ax1);
#endif
}

}  // namespace sfx
}  // namespace cell

// The tensor maps of one solver's buffers (make_epilogue_maps): the fused
// epilogue's and the staged flux kernels'.
struct EpilogueMaps {
  cell::epi::EpiMaps m;
  cell::sfx::FluxMaps f;
};

}  // namespace nmhd
