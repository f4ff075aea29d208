// Runs the quotients and roots of nmhd_b200/csrc/rounded.cuh on the GPU against
// the compiler's IEEE operations, over every case in which they could differ:
//   every root over [1, 4), scaled by even powers of two;
//   every reciprocal over [1, 2);
//   for every significand b the significands a whose quotient lies within
//   |2^k a - m b| <= 8 of a multiple of half an ulp, at both ends of the range
//   of numerators and denominators.
// Prints the number of cases and of mismatches.
#include <cstdio>

#include "../../nmhd_b200/csrc/rounded.cuh"

namespace {

using namespace nmhd;

struct Counts {
  unsigned long long cases, mismatches;
};

__device__ void tell(Counts *c, float got, float want) {
  atomicAdd(&c->cases, 1ull);
  if (__float_as_uint(got) != __float_as_uint(want)) atomicAdd(&c->mismatches, 1ull);
}

__global__ void roots(Counts *c) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 1u << 24) return;
  const float x = __uint_as_float(0x3f800000u + i);
  const float scales[3] = {1.0f, 0x1p-90f, 0x1p88f};
  for (float s : scales) tell(c, root(s * x), __fsqrt_rn(s * x));
}

__global__ void inverses(Counts *c) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 1u << 23) return;
  const float x = __uint_as_float(0x3f800000u + i);
  const float scales[3] = {1.0f, 0x1p-40f, -0x1p30f};
  for (float s : scales) tell(c, inverse(s * x), __frcp_rn(s * x));
}

__global__ void quotients(Counts *c) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 1u << 23) return;
  // 2^k A - m B = j with B = 2^t B': A = (j / 2^t) (2^(k-t))^-1 modulo B'
  const unsigned long long B = (1u << 23) + i;
  const int t = __ffsll(B) - 1;
  if (t > 3) return;  // |j| >= 16
  const unsigned long long odd = B >> t;
  for (int k = 24; k <= 25; ++k) {  // quotients in [1, 2) and in (1/2, 1)
    unsigned long long inv = 1 % odd;
    for (int n = 0; n < k - t; ++n) inv = inv * ((odd + 1) / 2) % odd;
    const unsigned long long lo = k == 24 ? B : 1u << 23, hi = k == 24 ? 1u << 24 : B;
    for (int j = -8; j <= 8; ++j) {
      if (j & ((1 << t) - 1)) continue;
      const unsigned long long r = (unsigned long long)((j / (1 << t) + (long long)odd) % (long long)odd);
      unsigned long long A = r * inv % odd;
      if (A < lo) A += (lo - A + odd - 1) / odd * odd;
      for (int n = 0; n < 32 && A < hi; ++n, A += odd) {
        const float a = __uint_as_float(0x3f800000u + (unsigned)(A - (1u << 23))), b = __uint_as_float(0x3f800000u + i);
        const float as[4] = {1.0f, 0x1p-90f, 0x1p79f, -1.0f}, bs[4] = {1.0f, 0x1p30f, -0x1p-40f, 0x1p-3f};
        for (int s = 0; s < 4; ++s)
          tell(c, quotient(as[s] * a, denominator(bs[s] * b)), __fdiv_rn(as[s] * a, bs[s] * b));
      }
    }
  }
}

}  // namespace

int main() {
  Counts *c = nullptr, h[3] = {};
  cudaError_t e = cudaMalloc(&c, sizeof h);
  if (e == cudaSuccess) e = cudaMemset(c, 0, sizeof h);
  if (e == cudaSuccess) {
    roots<<<(1 << 24) / 256, 256>>>(c);
    inverses<<<(1 << 23) / 256, 256>>>(c + 1);
    quotients<<<(1 << 23) / 256, 256>>>(c + 2);
    e = cudaMemcpy(h, c, sizeof h, cudaMemcpyDeviceToHost);
  }
  cudaFree(c);
  if (e != cudaSuccess) {
    std::printf("%s\n", cudaGetErrorString(e));
    return 1;
  }
  for (const Counts &k : h) std::printf("%llu %llu\n", k.cases, k.mismatches);
  return 0;
}
