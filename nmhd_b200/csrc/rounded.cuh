// Correctly rounded float quotients and square roots without a range check of
// their own, for code that checks its operands once for many of them.
//
// The compiler's IEEE division tests its operands, branches and joins again at
// every quotient (4 of its ~12 instructions), and inverts the denominator anew
// each time.  The Riemann solver divides four times by one denominator and
// takes 16 to 18 quotients and 7 roots a face, so it uses these instead and
// sends a face whose operands leave the ranges below to the plain arithmetic.
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
// Ranges: |b| in [2^-40, 2^31], a = 0 or |a| in [2^-90, 2^80], x in [2^-90,
// 2^90]; no intermediate then overflows, and no residual loses bits to
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
// of their bit patterns (NaN, infinities and, for positive(), negative values
// compare above every finite bound).
struct Ranges {
  unsigned least = 0x7fffffffu, most = 0u;  // values that must lie in [2^-40, 2^30]
  unsigned zleast = 0xffffffffu, zmost = 0u;  // values that must be 0 or in [2^-90, 2^80]
  __host__ __device__ __forceinline__ void positive(float v) {
    const unsigned u = float_bits(v);
    least = u < least ? u : least;
    most = u > most ? u : most;
  }
  __host__ __device__ __forceinline__ void nonzero(float v) {
    const unsigned u = float_bits(v) & 0x7fffffffu;
    least = u < least ? u : least;
    most = u > most ? u : most;
  }
  __host__ __device__ __forceinline__ void numerator(float v) {
    const unsigned u = float_bits(v) << 1;
    zmost = u > zmost ? u : zmost;
    zleast = u - 1u < zleast ? u - 1u : zleast;  // 0 becomes the largest
  }
  __host__ __device__ __forceinline__ bool hold() const {
    constexpr unsigned one = 127u;
    return least >= (one - 40u) << 23 && most <= (one + 30u) << 23 && zleast >= ((one - 90u) << 24) - 1u &&
           zmost <= (one + 80u) << 24;
  }
};

}  // namespace nmhd
