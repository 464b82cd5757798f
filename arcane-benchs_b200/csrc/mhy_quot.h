// mhy_quot.h -- correctly rounded FP64 reciprocals and quotients without a
// branch, for operands in a checked range (host and device, the same bits).
//
// From P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990:
//   - if y1 is within one ulp of 1/y, then e = 1 - y y1 is exact with one fma
//     and RN(y1 + y1 e) = RN(1/y), unless the significand of y is all ones:
//     1/y is then just above the middle between a power of two and the next
//     number, so RN(1/y) is that next number, and setting the last bit of
//     either neighbour gives it;
//   - with r = RN(1/y), q0 = RN(x r) and e = x - y q0 (exact with one fma),
//     RN(q0 + e r) = RN(x/y),
// as long as nothing underflows or overflows.  y1 comes from a seed y0 of
// relative error d < 2^-18 by one step of third order, y0 (1 + d + d^2): its
// error is d^3 < 2^-54 (half an ulp at most) plus the rounding of that step.
//
// The range: 2^-960 <= |x|, |q0| < 2^960 for a nonzero x and 2^-959 <= |y| <
// 2^960, all tested on the exponents: the residual of the quotient is then a
// multiple of 2^-1065 and nothing overflows.  Where an operand leaves the range
// (zero y, subnormals, infinities, NaN), bad gets a nonzero value and the
// caller computes x / y again.  8e9 random and adversarial pairs that raised
// nothing agreed with x / y and 1 / y.
//
// Why: the compiler's division takes a branch to a slow path at every quotient,
// so the independent quotients of a sweep (FP64 results take tens of cycles)
// follow one another; without branches they overlap.  Measured on B200, FP64:
// node sweep along x 105 -> 84 us on Sedov 128^3 and 107 -> 62 us on a shock
// tube of 211x97x61 with vanLeer (four quotients a slope); a whole cycle
// 1254 -> 1159 us and 1105 -> 817 us.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define MHY_Q_HD __host__ __device__ __forceinline__
#else
#define MHY_Q_HD inline
#endif

namespace mhy {

MHY_Q_HD uint32_t q_hi(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t u; memcpy(&u, &x, 8); return (uint32_t)(u >> 32);
#endif
}
MHY_Q_HD uint32_t q_lo(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t u; memcpy(&u, &x, 8); return (uint32_t)u;
#endif
}
MHY_Q_HD double q_make(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t u = (uint64_t)hi << 32 | lo; double x; memcpy(&x, &u, 8); return x;
#endif
}
MHY_Q_HD double q_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return fma(a, b, c);
#endif
}

// Biased exponents [lo, hi) as an unsigned interval of the high word with the sign shifted out.
#define MHY_Q_OUT(h, lo, hi) ((uint32_t)((h) + (h) - ((uint32_t)(lo) << 21)) >= ((uint32_t)((hi) - (lo)) << 21))

// RN(1/y) from a seed y0 with |1 - y y0| < 2^-18.
MHY_Q_HD double rcp_from_seed(double y, double y0, unsigned& bad) {
  const double d = q_fma(-y, y0, 1.0);
  const double y1 = q_fma(y0, q_fma(d, d, d), y0);
  const double r = q_fma(y1, q_fma(-y, y1, 1.0), y1);
  const uint32_t h = q_hi(y);
  if (MHY_Q_OUT(h, 64, 1983)) bad = 1u;
  const uint32_t ones = (q_lo(y) & (h | 0xfff00000u)) == 0xffffffffu ? 1u : 0u;
  return q_make(q_hi(r), q_lo(r) | ones);
}

// The plain 1 / y with the check of y that quo_from_rcp leaves to whoever forms r.
MHY_Q_HD double rcp_checked(double y, unsigned& bad) {
  const uint32_t h = q_hi(y);
  if (MHY_Q_OUT(h, 64, 1983)) bad = 1u;
  return 1.0 / y;
}

// RN(x/y) with r = RN(1/y) of a y inside the range: whoever formed r has raised
// bad for any other y (rcp_from_seed and rcp_checked do).  Only x and q0 are
// tested here, and that does not see every y outside the range: a zero x over a
// y whose 1/y is 0 or infinite gives NaN.  A zero x gives the zero of the right
// sign (q0's).
MHY_Q_HD double quo_from_rcp(double x, double y, double r, unsigned& bad) {
  const double q0 = x * r;
  const double q = q_fma(q_fma(-q0, y, x), r, q0);
  const uint32_t h0 = q_hi(q0), hx = q_hi(x);
  if (x != 0.0 && (MHY_Q_OUT(hx, 63, 1983) || MHY_Q_OUT(h0, 63, 1983))) bad = 1u;
  return q_make((q_hi(q) & 0x7fffffffu) | (h0 & 0x80000000u), q_lo(q));
}

#if defined(__CUDACC__)
// The seed: the reciprocal approximation instruction (about 20 good bits).
__device__ __forceinline__ double rcp_seed(double y) {
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(y));
  return y0;
}
__device__ __forceinline__ double rcp_fast(double y, unsigned& bad) { return rcp_from_seed(y, rcp_seed(y), bad); }
__device__ __forceinline__ double quo_fast(double x, double y, unsigned& bad) {
  return quo_from_rcp(x, y, rcp_fast(y, bad), bad);
}
#endif

}  // namespace mhy
