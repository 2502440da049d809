// exactdiv.h -- correctly rounded FP64 quotients without a branch each, for
// operands whose exponents rule out overflow and underflow.
//
// Why: divisions by one b repeat its reciprocal, and in the flux kernels consecutive
// divisions of a thread were seen to wait for one another. Here the reciprocal is
// formed once (rcp), each quotient takes four operations (quot), and the operands'
// exponents are tested with the range predicates, whose results a caller collects over
// a group of quotients; if one fails, the caller recomputes the group with `/`. The
// results are the same bits as `/`. (Staged x2 fluxes of the 512 x 256 torus: 10.7
// against 18.9 million warp instructions, 28.5 against 41 us, PPM4's shared face values
// included.)
//
// Method (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990; Muller et al., Handbook of
// Floating-Point Arithmetic, section "Division using fused multiply-add"):
//   * y0 = 1/b to 2^-19 or better; one cubic Newton step gives a y within an
//     ulp of 1/b; y + y (1 - b y), with 1 - b y exact, is then RN(1/b) unless
//     the mantissa of b is all ones (in_range_den refuses those);
//   * q = RN(a y + RN(a y_lo)) with y_lo = y (1 - b y) is a faithful rounding of
//     a / b: a (y + y_lo) is a / b to 2^-100, and the two roundings are half
//     an ulp each;
//   * with y = RN(1/b) and q faithful, r = a - b q is exact and RN(q + r y) is
//     RN(a / b) (Markstein's theorem).
// A zero numerator gives a zero (the sign of -0 / b is not kept; quot_s keeps
// it). tests/test_exactdiv.py and, on the device and with its first approximation,
// tests/test_gpu_exactdiv.py compare with `/` on random operands and on quotients
// built to lie next to a rounding boundary.
#ifndef PANGU_EXACTDIV_H
#define PANGU_EXACTDIV_H

#include <cmath>
#include <cstring>

#if defined(__CUDACC__)
#define XD_FN __host__ __device__ __forceinline__
#else
#define XD_FN inline
#endif

namespace xd {

XD_FN double fma_(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
XD_FN double mul_(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
XD_FN unsigned hi_bits(double x) {
#if defined(__CUDA_ARCH__)
  return (unsigned)__double2hiint(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return (unsigned)(b >> 32);
#endif
}
XD_FN unsigned lo_bits(double x) {
#if defined(__CUDA_ARCH__)
  return (unsigned)__double2loint(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return (unsigned)b;
#endif
}
XD_FN double with_hi(double x, unsigned hi) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo_bits(x));
#else
  const unsigned long long b = ((unsigned long long)hi << 32) | lo_bits(x);
  double r;
  std::memcpy(&r, &b, 8);
  return r;
#endif
}

// Ranges in which no value under- or overflows: denominators in
// [2^-400, 2^60), numerators 0 or in [2^-960, 2^400). The quotient is then normal
// (2^-1020 < |q| < 2^800) and the residual a - b q a multiple of 2^-1066. The
// numerators' range reaches that low because fields that spread from zero into
// a gas at rest fall off by many decades per cell.
XD_FN constexpr unsigned expo(int e) { return (1023u + (unsigned)e) << 20; }

// Denominator: exponent in range, mantissa not all ones.
XD_FN bool in_range_den(double b) {
  return (((hi_bits(b) & 0x7fffffffu) - expo(-400)) < (expo(60) - expo(-400))) &
         (lo_bits(b) != 0xffffffffu);
}
// Numerator that is not zero in ordinary use.
XD_FN bool in_range(double a) {
  return ((hi_bits(a) & 0x7fffffffu) - expo(-960)) < (expo(400) - expo(-960));
}
// Numerator that often is zero.
XD_FN bool in_range0(double a) {
  const unsigned h = hi_bits(a) & 0x7fffffffu;
  return ((h - expo(-960)) < (expo(400) - expo(-960))) | ((h | lo_bits(a)) == 0u);
}

// |a| below 2^e.
XD_FN bool below(double a, int e) { return (hi_bits(a) & 0x7fffffffu) < expo(e); }

struct Rcp {
  double nb, y, yl;  // -b, RN(1/b), and y (1 - b y)
};

// RN(1/b) for an in-range denominator, from a first approximation y0 of 1/b
// (|1 - b y0| < 2^-19).
XD_FN double recip_from(double b, double y0) {
  double e = fma_(-b, y0, 1.0);
  e = fma_(e, e, e);
  double y = fma_(y0, e, y0);
  e = fma_(-b, y, 1.0);
  return fma_(y, e, y);
}
XD_FN Rcp rcp_from(double b, double y0) {
  const double y = recip_from(b, y0);
  return {-b, y, mul_(y, fma_(-b, y, 1.0))};
}

#if defined(__CUDACC__)
__device__ __forceinline__ double rcp_seed(double b) {
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  return y0;
}
__device__ __forceinline__ Rcp rcp(double b) { return rcp_from(b, rcp_seed(b)); }
__device__ __forceinline__ double recip(double b) { return recip_from(b, rcp_seed(b)); }
#endif

// RN(a / b) for in-range operands.
XD_FN double quot(double a, const Rcp &r) {
  const double q = fma_(a, r.yl, mul_(a, r.y));
  return fma_(fma_(r.nb, q, a), r.y, q);
}
// The same, with the sign of a zero quotient (b > 0).
XD_FN double quot_s(double a, const Rcp &r) {
  const double q = quot(a, r);
  return with_hi(q, hi_bits(q) | (hi_bits(a) & 0x80000000u));
}

// RN(a / 12). y = RN(1/12) is 1/3 ulp below 1/12, so RN(a y) is faithful as it
// is: |a/12 - RN(a y)| <= (a 2^-53 / 3 + 2^-54) < 2^-53 for a scaled to [1, 1.5)
// (quotient in [2/3, 1), ulp 2^-53), and likewise below one ulp for a in
// [1.5, 2).
XD_FN double div12(double a) {
  constexpr double y = 1.0 / 12.0;
  const double q = mul_(a, y);
  const double r = fma_(fma_(-12.0, q, a), y, q);
  return with_hi(r, hi_bits(r) | (hi_bits(a) & 0x80000000u));
}

}  // namespace xd
#endif  // PANGU_EXACTDIV_H
