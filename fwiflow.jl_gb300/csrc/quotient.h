// The quotient of the CPML formulas (sweeps and marching kernels; also compiled
// for the host, where it is compared with the division).
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define FWIGB_QUOTIENT __device__ __forceinline__
#define FWIGB_QUOTIENT_CALL static __device__ __noinline__
#else
#define FWIGB_QUOTIENT inline
#define FWIGB_QUOTIENT_CALL inline
#endif

namespace fwigb {

// (a product that is not contracted into a following sum)
FWIGB_QUOTIENT float product(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}

// a / K rounded to nearest, for K in [1, 2]: the bits of the division for every
// a. The estimate a r with r = 1 / K rounded is corrected by its residual
// (Markstein, IBM J. Res. Dev. 34, 1990), which takes an exact residual. That of
// a small a need not be a float (it is a multiple of 2^-172), so that it is formed
// 2^24 times as large, from K and r scaled accordingly; the corrected quotient is
// rounded once, subnormal or not. In the subnormal range too the correction errs by
// less than the exact quotient lies from the middle of two floats: by K 2^-26
// units of the last place against 2^-24 / K (and the middle itself is hit only by
// K = 2, whose r is exact).
constexpr float kQuotientScale = 0x1p24f;

// The quotient of a large a (or one that is not finite), for which the scaled
// one might overflow; its residual is a float as it is.
FWIGB_QUOTIENT float over_large(float a, float K_scaled, float r_scaled) {
  const float K = product(K_scaled, 1.0f / kQuotientScale), r = product(r_scaled, kQuotientScale), q = product(a, r);
  return fabsf(a) < INFINITY ? fmaf(fmaf(K, q, -a), -r, q) : a;
}
FWIGB_QUOTIENT_CALL float call_over_large(float a, float K_scaled, float r_scaled) {
  return over_large(a, K_scaled, r_scaled);
}

// CALL: a large a takes a function call instead of instructions in place, which
// leaves the sweeps' few registers to the rest. ms a gradient, call / in place
// (three operations in all, neither exact below 2^-100 nor finite from infinity on):
// 16 shots of 352 x 832, 100 steps 18.9 / 19.2 (18.8); two 1120 x 3152 shots, 40
// steps 10.87 / 11.0 (10.84); marching, two 192 x 264 grids, 300 steps 4.15 / 4.06
// (3.96). (With the division 37.9 became 42.0 ms on 16 such shots, 200 steps: its
// path for numerators near the smallest floats is taken all the time in an
// absorbing layer, where the fields die out.) F2 has them in place (fwd_velocity_edge).
template <bool CALL = true>
FWIGB_QUOTIENT float over(float a, float K_scaled, float r_scaled) {
  const float b = product(a, kQuotientScale), q = product(b, r_scaled);
  float y = fmaf(fmaf(K_scaled, q, -b), -r_scaled, q);
  if (!(fabsf(a) < 0x1p103f)) y = CALL ? call_over_large(a, K_scaled, r_scaled) : over_large(a, K_scaled, r_scaled);
  return y;
}

}  // namespace fwigb
