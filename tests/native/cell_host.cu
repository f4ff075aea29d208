// Host build of the single-box step's face arithmetic (nmhd_b200/csrc/
// mhd_math.cuh: minbee reconstruction and the HLLD flux), for the CPU tests
// only.  The library's kernels compile the same functions for sm_100a with
// -fmad=false and IEEE division and square root; here gcc rounds every float
// and double operation separately (-ffp-contract=off, SSE arithmetic), so the
// results are the device's and the tests can compare them bitwise with the
// oracle on a CPU.  Not part of the library; nothing in nmhd_b200 loads it.
#include "../../nmhd_b200/csrc/cell_flux_staged.cuh"
#include "../../nmhd_b200/csrc/fields.h"

extern "C" {

// lr: dl, dr, ul, ur, vl, vr, wl, wr, pl, pr, byl, byr, bzl, bzr (HlldIn order)
void cellh_hlld_f32(float gamma, float bx, const float *lr, float *out) {
  nmhd::HlldIn in;
  float *dst = &in.dl;
  for (int i = 0; i < 14; ++i) dst[i] = lr[i];
  nmhd::hlld_flux(gamma, bx, in, out);
}

void cellh_hlld_many_f32(float gamma, const float *bx, const float *lr, float *out, long n) {
  for (long i = 0; i < n; ++i) cellh_hlld_f32(gamma, bx[i], lr + 14 * i, out + 7 * i);
}

// hlld_flux_ranged alone: ok[i] says whether it took the state; and the plain
// arithmetic it stands in for.
void cellh_hlld_ranged_f32(float gamma, const float *bx, const float *lr, float *ranged, float *plain, int *ok, long n) {
  const nmhd::Denominator gm1 = nmhd::denominator(gamma - 1.0f);
  for (long i = 0; i < n; ++i) {
    nmhd::HlldIn in;
    float *dst = &in.dl;
    for (int k = 0; k < 14; ++k) dst[k] = lr[14 * i + k];
    ok[i] = nmhd::hlld_flux_ranged(gamma, gm1, bx[i], in, ranged + 7 * i);
    nmhd::hlld_flux_plain(gamma, bx[i], in, plain + 7 * i);
  }
}

void cellh_reconstruct_f32(const float *x, float *lr, long n) {
  for (long i = 0; i < n; ++i) nmhd::reconstruct4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3], lr[2 * i], lr[2 * i + 1]);
}

// reconstruct4_with alone: ok[i] says whether its slopes were in range.
void cellh_reconstruct_ranged_f32(const float *x, float *lr, int *ok, long n) {
  for (long i = 0; i < n; ++i) {
    nmhd::Ranged q;
    nmhd::reconstruct4_with(q, x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3], lr[2 * i], lr[2 * i + 1]);
    q.positive(1.0f);
    ok[i] = q.hold();
  }
}

}  // extern "C"

// The columns of a box nx cells wide that the staging of a tile at x0 copies into
// a row of one of its boxes (0: the flux kernel's, 1..: the update kernel's), in
// chunks of W floats: out[position - origin], -1 where nothing is copied;
// `inside` false where a chunk leaves the row of the box.  Row position p stands
// for x0 + *origin + p; positions [*begin, *end) are read.
namespace {
template <int kBegin, int kEnd, int W>
int copied(int x0, int origin, int nx, int *out) {
  using C = nmhd::cell::RowChunks<kBegin, kEnd, W>;
  int inside = 1;
  for (int c = 0; c < C::count; ++c) {
    const int pos = C::first + W * c, col = nmhd::cell::row_column<W>(x0 + origin + pos, nx);
    inside = inside && col >= 0 && col + W <= nx;
    for (int i = 0; i < W; ++i) out[pos + i] = col + i;
  }
  return inside;
}
template <int kBegin, int kEnd>
int copied(int W, int x0, int o, int nx, int *out, int *origin, int *begin, int *end) {
  *origin = o, *begin = kBegin, *end = kEnd;
  return W == 4   ? copied<kBegin, kEnd, 4>(x0, o, nx, out)
         : W == 2 ? copied<kBegin, kEnd, 2>(x0, o, nx, out)
                  : copied<kBegin, kEnd, 1>(x0, o, nx, out);
}
template <class B>
int copied_box(int W, int x0, int nx, int *out, int *origin, int *begin, int *end) {
  return copied<B::XO, B::XO + B::NI>(W, x0, B::OI - B::XO, nx, out, origin, begin, end);
}
}  // namespace

extern "C" int cellh_staged_columns(int box, int W, int x0, int nx, int *out, int *origin, int *begin, int *end) {
  using namespace nmhd::cell;
  for (int i = 0; i < 40; ++i) out[i] = -1;
  switch (box) {
    case 0: return copied<sfx::kReadBegin, sfx::kReadEnd>(W, x0, -sfx::XO, nx, out, origin, begin, end);
    case 1: return copied_box<epi::VelBox>(W, x0, nx, out, origin, begin, end);
    case 2: return copied_box<epi::XYF>(W, x0, nx, out, origin, begin, end);
    case 3: return copied_box<epi::YXF>(W, x0, nx, out, origin, begin, end);
    case 4: return copied_box<epi::ZYF>(W, x0, nx, out, origin, begin, end);
    default: return -1;
  }
}

// one_run() over a made-up address space: m allocations [begin[i], end[i]), the
// rest pageable, or unknown to the driver.
extern "C" int cellh_one_run(const uintptr_t *fields, long n, const uintptr_t *begin, const uintptr_t *end, int m,
                             int known) {
  const float *f[8];
  for (int v = 0; v < 8; ++v) f[v] = reinterpret_cast<const float *>(fields[v]);
  nmhd::Allocation held = {};
  return nmhd::one_run(f, (size_t)n, held, [&](const void *p) {
    nmhd::Allocation a = {known != 0, 0, 0};
    for (int i = 0; i < m; ++i)
      if (begin[i] <= (uintptr_t)p && (uintptr_t)p < end[i]) a.begin = begin[i], a.end = end[i];
    return a;
  });
}

// A face's flux from the four cells of its stencil: x holds 4 x (rho, u, v, w, p, By
// sum, Bz sum), the last two sums of two face values; by hlld_flux_ranged() on the
// states of reconstruct4_with() (ok[i]: whether it takes them) and by the plain
// arithmetic on the means.
extern "C" void cellh_face_f32(float gamma, const float *bx, const float *x, float *ranged, float *plain, int *ok,
                               long n) {
  const nmhd::Denominator gm1 = nmhd::denominator(gamma - 1.0f);
  for (long i = 0; i < n; ++i) {
    const float *c = x + 28 * i;
    nmhd::HlldIn a, b;
    nmhd::Ranged q;
    nmhd::Ieee unchecked;
    float *pa = &a.dl, *pb = &b.dl;
    for (int v = 0; v < 7; ++v) {
      const float y[4] = {c[v], c[7 + v], c[14 + v], c[21 + v]};
      if (v == 0 || v == 4) nmhd::cell::sfx::face_states(unchecked, y, pa[2 * v], pa[2 * v + 1]);
      else if (v < 5) nmhd::cell::sfx::face_states(q, y, pa[2 * v], pa[2 * v + 1]);
      else nmhd::cell::sfx::face_means(q, y, pa[2 * v], pa[2 * v + 1]);
      const float h = v < 5 ? 1.0f : 0.5f;
      nmhd::reconstruct4(h * y[0], h * y[1], h * y[2], h * y[3], pb[2 * v], pb[2 * v + 1]);
    }
    ok[i] = nmhd::hlld_flux_with(q, gamma, gm1, bx[i], a, [&](int k, float v) { ranged[7 * i + k] = v; });
    nmhd::hlld_flux_plain(gamma, bx[i], b, plain + 7 * i);
  }
}

// face_means() alone, and reconstruct4() of the means.
extern "C" void cellh_means_f32(const float *sums, float *ranged, float *plain, int *ok, long n) {
  for (long i = 0; i < n; ++i) {
    const float *s = sums + 4 * i;
    nmhd::Ranged q;
    nmhd::cell::sfx::face_means(q, s, ranged[2 * i], ranged[2 * i + 1]);
    q.positive(1.0f);
    ok[i] = q.hold();
    nmhd::reconstruct4(0.5f * s[0], 0.5f * s[1], 0.5f * s[2], 0.5f * s[3], plain[2 * i], plain[2 * i + 1]);
  }
}

extern "C" int cellh_likely_in_range(float d, float p, float bx, float by, float bz) {
  return nmhd::likely_in_range(d, p, bx, by, bz);
}
