// sg_pairmath.h - powers and quotients of the EAM pair functions (sg_forces.cuh): single IEEE
// operations in a fixed order, none of them contracted, so that a host compiler's results, which the
// tests compare with exact ones, are the device's bit for bit.
#pragma once
#ifdef __CUDACC__
#define SG_PAIRMATH __device__ __forceinline__
#else
#include <cmath>
#define SG_PAIRMATH inline
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
#endif

namespace sg {

// x^20, and x^20 with x^19, by repeated squaring on error-free float pairs: the square of
// (h, l) is (h h, fma(h, h, -h h) + 2 h l), three instructions, so both powers come out rounded
// from about 46 bits (error at most 0.501 ulp; powf documents 4) for a fraction of two powf calls.
// Below 2^-110, where the low parts leave FP32's range, it grows to 2 ulp and in the subnormal numbers
// to a few of their units: the pair functions add such a power to 1.
// The PLAIN metal passes are bound by instruction issue (63-65% of the issue slots); with these and the
// shared reciprocals below k_force_metal takes 50.8 us instead of 68.7 and k_rho 29.4 instead of 32.0 on
// bulk Au (55,296 atoms, ncu).
// The pair functions call them with |x| below 2; past 64 the powers come near the largest float,
// where the pairs' error terms would turn an infinity into a NaN: powf decides there (and for NaN).
struct FPair {
  float h, l;
};
SG_PAIRMATH FPair pairSquare(FPair a) {
  FPair r;
  r.h = __fmul_rn(a.h, a.h);
  r.l = __fmaf_rn(__fadd_rn(a.h, a.h), a.l, __fmaf_rn(a.h, a.h, -r.h));
  return r;
}
// a b rounded to float
SG_PAIRMATH float pairProduct(FPair a, FPair b) {
  const float p = __fmul_rn(a.h, b.h);
  const float e = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.h, -p)));
  return __fadd_rn(p, e);
}
SG_PAIRMATH float pow20(float x) {
  if (!(fabsf(x) < 64.f)) return powf(x, 20.f);
  const FPair x4 = pairSquare(pairSquare(FPair{x, 0.f}));
  return pairProduct(pairSquare(pairSquare(x4)), x4);
}
SG_PAIRMATH void pow19and20(float x, float &x19, float &x20) {
  if (!(fabsf(x) < 64.f)) {
    x19 = powf(x, 19.f);
    x20 = powf(x, 20.f);
    return;
  }
  const FPair x2 = pairSquare(FPair{x, 0.f}), x4 = pairSquare(x2), x16 = pairSquare(pairSquare(x4));
  FPair x3;
  x3.h = __fmul_rn(x2.h, x);
  x3.l = __fmaf_rn(x2.l, x, __fmaf_rn(x2.h, x, -x3.h));
  x19 = pairProduct(x16, x3);
  x20 = pairProduct(x16, x4);
}
// a / b with r = 1 / b rounded to nearest: the quotient a r corrected once by its exact remainder
// is a / b rounded to nearest (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990), the same bits as the IEEE division but for the sign of a zero, for b
// from 1 to 2^126 and |a| from 2^-100 b on (by b = 1, any finite a).  The pair functions divide by each of
// two denominators three or four times; one reciprocal serves them all.
SG_PAIRMATH float divBy(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return __fmaf_rn(__fmaf_rn(-b, q, a), r, q);
}

}  // namespace sg
#undef SG_PAIRMATH
