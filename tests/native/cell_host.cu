// Host build of the single-box step's face arithmetic (nmhd_b200/csrc/
// mhd_math.cuh: minbee reconstruction and the HLLD flux), for the CPU tests
// only.  The library's kernels compile the same functions for sm_100a with
// -fmad=false and IEEE division and square root; here gcc rounds every float
// and double operation separately (-ffp-contract=off, SSE arithmetic), so the
// results are the device's and the tests can compare them bitwise with the
// oracle on a CPU.  Not part of the library; nothing in nmhd_b200 loads it.
#include "../../nmhd_b200/csrc/mhd_math.cuh"

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
