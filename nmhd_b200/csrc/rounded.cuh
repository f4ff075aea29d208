// Correctly rounded float quotients and square roots without a range check of
// their own, for code that checks its operands once for many of them.
//
// The Riemann solver divides four times by one denominator and takes 16 to 18
// quotients and 7 roots a face.  With one reciprocal a denominator and one range
// test a face in place of the compiler's divisions, 16 steps of the 256x128x64
// box went from 10.31 to 9.47 ms; a face whose operands leave the ranges below
// takes the plain arithmetic.
//
// Quotient a/b.  From y ~ 1/b (the hardware approximation, at most 1 ulp off)
// one Newton step gives h = RN(1/b) (for every b of a binade, as the check
// below finds).  t = RN(a h) is within 1.5 ulp of a/b, r = a - b t is exact in
// one fused multiply-add, and RN(t + r h) is off by at most 3 * 2^-25 ulp before
// its rounding (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990; Muller et al., Handbook of
// Floating-Point Arithmetic, 4.7).  It can then differ from RN(a/b) only for
// quotients that near a midpoint, |2^k a - (2m+1) b| <= 4 over the integer
// significands: tests/native/rounded_check.cu lists all of them up to 8, and
// every root over two binades, and runs them on the GPU.
//
// Square root of x: from y ~ 1/sqrt(x), g = x y is corrected by y/2 times the
// exact residual x - g^2 (Markstein, same paper).
//
// Ranges: |b| in [2^-40, 2^31], a = 0 or |a| >= 2^-73, |a/b| < 2^127, x in
// [2^-90, 2^90]; no intermediate then overflows, and no residual loses bits to
// underflow.  A zero quotient may come back as +0 where it is -0.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace nmhd {

// 1/x and 1/sqrt(x), approximately (the host build of the tests rounds them).
__host__ __device__ __forceinline__ float approx_inverse(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}
__host__ __device__ __forceinline__ float approx_inverse_root(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (float)(1.0 / sqrt((double)x));
#endif
}

// RN(1/b).
__host__ __device__ __forceinline__ float inverse(float b) {
  const float y = approx_inverse(b);
  return fmaf(y, fmaf(-b, y, 1.0f), y);
}

// A denominator b with RN(1/b).
struct Denominator {
  float b, h;
};
__host__ __device__ __forceinline__ Denominator denominator(float b) { return Denominator{b, inverse(b)}; }

__host__ __device__ __forceinline__ bool denominator_in_range(float b) { return b >= 0x1p-40f && b <= 0x1p30f; }

// RN(a/b).
__host__ __device__ __forceinline__ float quotient(float a, const Denominator &d) {
  const float t = a * d.h;
  return fmaf(fmaf(-d.b, t, a), d.h, t);
}

// RN(sqrt(x)).
__host__ __device__ __forceinline__ float root(float x) {
  const float y = approx_inverse_root(x);
  const float g = x * y;
  return fmaf(fmaf(-g, g, x), 0.5f * y, g);
}

__host__ __device__ __forceinline__ unsigned float_bits(float v) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(v);
#else
  unsigned u;
  memcpy(&u, &v, 4);
  return u;
#endif
}

// Whether the operands seen so far lie in the ranges above, kept as extremes
// of their bit patterns.  positive(): in [2^-40, 2^24], as the largest distance
// above the lower bound (unsigned: smaller, negative and NaN values wrap or lie
// far above).  tiny(): 0 or at least 2^-73, as the least pattern less one (0
// becomes the largest).  Two accumulators and one instruction a value: more of
// either cost the Riemann solver spills.
struct Ranges {
  static constexpr unsigned kLow = (127u - 40u) << 23, kHigh = (127u + 24u) << 23, kTiny = (127u - 73u) << 23;
  unsigned far = 0u, least = 0xffffffffu;
  __host__ __device__ __forceinline__ void positive(float v) {
    const unsigned u = float_bits(v) - kLow;
    far = u > far ? u : far;
  }
  __host__ __device__ __forceinline__ void tiny(float v) {  // v >= 0
    const unsigned u = float_bits(v) - 1u;
    least = u < least ? u : least;
  }
  __host__ __device__ __forceinline__ bool hold() const { return far <= kHigh - kLow && least >= kTiny - 1u; }
};

// Whether a cell's faces are likely to hold (known before they are solved): its
// density and pressure are in the range of positive(), as its faces' must be, and
// its field is 0 or not so weak that products of two components leave tiny()'s.
__host__ __device__ __forceinline__ bool likely_in_range(float d, float p, float bx, float by, float bz) {
  Ranges r;
  r.positive(d);
  r.positive(p);
  r.tiny(fmaxf(fmaxf(fabsf(bx), fabsf(by)), fabsf(bz)) * 0x1p-36f);  // 0 or at least 2^-37
  return r.hold();
}

// Arithmetic of code written once over its quotients and roots: div() checks
// its numerator (div_bounded() also from above, by 2^60), ratio() and root()
// leave their operands to positive(), and hold() says at the end whether every
// operand was in range.
//
// Ranged: the operations above, to be repeated with Ieee where hold() is false.
struct Ranged {
  Ranges r;
  __host__ __device__ __forceinline__ void positive(float v) { r.positive(v); }
  __host__ __device__ __forceinline__ void slope(float v) { r.tiny(v); }
  __host__ __device__ __forceinline__ static Denominator under(float b) { return denominator(b); }
  __host__ __device__ __forceinline__ static float ratio(float a, const Denominator &d) { return quotient(a, d); }
  __host__ __device__ __forceinline__ float div(float a, const Denominator &d) {
    r.tiny(fabsf(a));
    return quotient(a, d);
  }
  __host__ __device__ __forceinline__ float div_bounded(float a, const Denominator &d, float least = 0x1p-40f) {
    // |a| 2^-36 + 2^-40 <= 2^24
    r.positive(fmaf(fabsf(a), 0x1p-36f, least));
    return div(a, d);
  }
  // 2^-40 if all are finite, else NaN, which is in no range.
  __host__ __device__ __forceinline__ static float finite(float a, float b, float c, float d) {
    return fmaf(a, 0.0f, fmaf(b, 0.0f, fmaf(c, 0.0f, fmaf(d, 0.0f, 0x1p-40f))));
  }
  __host__ __device__ __forceinline__ static float root(float x) { return nmhd::root(x); }
  __host__ __device__ __forceinline__ bool hold() const { return r.hold(); }
};

// The compiler's division and square root, for any operands.
struct Ieee {
  __host__ __device__ __forceinline__ static void positive(float) {}
  __host__ __device__ __forceinline__ static void slope(float) {}
  __host__ __device__ __forceinline__ static Denominator under(float b) { return Denominator{b, 0.0f}; }
  __host__ __device__ __forceinline__ static float ratio(float a, const Denominator &d) { return a / d.b; }
  __host__ __device__ __forceinline__ static float div(float a, const Denominator &d) { return a / d.b; }
  __host__ __device__ __forceinline__ static float div_bounded(float a, const Denominator &d, float = 0.0f) { return a / d.b; }
  __host__ __device__ __forceinline__ static float finite(float, float, float, float) { return 1.0f; }
  __host__ __device__ __forceinline__ static float root(float x) { return sqrtf(x); }
  __host__ __device__ __forceinline__ static bool hold() { return true; }
};

}  // namespace nmhd
