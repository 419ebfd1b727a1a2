// The FP64 near field's kernel evaluation.
#pragma once

namespace dfb {

#ifdef __CUDACC__
// Approximate FP64 reciprocal square root (the PTX instruction
// rsqrt.approx.ftz.f64, about FP32 accuracy); callers refine it by Newton
// steps y <- y (3/2 - R y^2 / 2), each of which doubles the correct bits.
__device__ __forceinline__ double rsqrt_approx64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
#endif

// Squared distances below 1e-16 are coincident points' (P2P.hpp:66).  The bits
// are compared as unsigned numbers: a squared distance is not negative, and a
// NaN of either sign (a coordinate that is NaN) counts as a large one, so that
// it reaches the potentials.
constexpr unsigned kNearR2Hi = 0x3C9CD2B2u;  // the high word of 1e-16
__device__ __forceinline__ bool coincident(double R) {
  return (unsigned long long)__double_as_longlong(R) < 0x3C9CD2B297D889BCull;
}

// sin(pi/2 u) / u and cos(pi/2 u) for |u| <= 1/2, z = u^2: polynomials of degree
// 6 and 7 in z, fitted with the Remez exchange in 50 digits and rounded to
// doubles.  The rounding is what is left: with these coefficients the sine is
// off by 5.0e-17 relative, the cosine by 1.6e-17 (an ulp is 1.1e-16 to 2.2e-16).
template <class F>
__device__ __forceinline__ F quarter_sin(F z) {
  F p = fma(z, F(5.633721016484235e-08), F(-3.598641754487236e-06));
  p = fma(z, p, F(0.00016044115029166428));
  p = fma(z, p, F(-0.00468175413228242));
  p = fma(z, p, F(0.07969262624603957));
  p = fma(z, p, F(-0.6459640975062443));
  return fma(z, p, F(1.5707963267948966));
}
template <class F>
__device__ __forceinline__ F quarter_cos(F z) {
  F p = fma(z, F(-6.321892625650177e-09), F(4.7106156592722383e-07));
  p = fma(z, p, F(-2.5202036991591028e-05));
  p = fma(z, p, F(0.0009192602742250428));
  p = fma(z, p, F(-0.020863480763315442));
  p = fma(z, p, F(0.2536695079010469));
  p = fma(z, p, F(-1.2337005501361697));
  return fma(z, p, F(1.0));
}

// exp(i k r) / r of one pair in FP64 (0 for R < 1e-16, P2P.hpp:66), without
// the factor 1 / (4 pi), with kq = 2 k / pi.  An FP64 instruction takes two
// issue cycles, every other one, so both counts matter (41 FP64 instructions
// here; the reduction by pi/2 in two parts with rint and Taylor series took
// 48 and two conversions): 1/r from the approximate
// reciprocal square root by one cubic step y + y e (1/2 + 3/8 e),
// e = 1 - R y^2 (|e| < 2^-19: the next term is below 2^-58); the phase in
// quarter turns, r kq = n + u with |u| <= 1/2, u by one exactly rounded FMA
// and n's low bits from the mantissa of r kq + 1.5 * 2^52.  kq is rounded once,
// so all pairs share its relative error (up to 1.1e-16): at k r near 35 the
// phase's mean error can reach a few 1e-15, as much as its scatter (3.6e-15
// rms, from rounding r); reducing by pi/2 in two parts shares less (3e-16)
// with the same scatter and larger maxima.
// GUARD = false: the caller knows R0 >= 1e-16.
template <bool GUARD>
__device__ __forceinline__ double2 green64_r(double R0, double kq) {
  double R = R0;
  if (GUARD) R = __hiloint2double((int)max((unsigned)__double2hiint(R0), kNearR2Hi), __double2loint(R0));
  const double y0 = rsqrt_approx64(R);
  const double e = fma(-(R * y0), y0, 1.0);
  double y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
  const double r = R * y;
  const double t = fma(r, kq, 6755399441055744.0);  // + 1.5 * 2^52
  const double u = fma(r, kq, -(t - 6755399441055744.0));
  const int q = __double2loint(t);
  const double z = u * u;
  const double ps = quarter_sin(z), pc = quarter_cos(z);
  if (GUARD && coincident(R0)) y = 0.;
  // quadrant q: sin and cos of the whole phase are (sr, cr), (cr, -sr),
  // (-sr, -cr), (-cr, sr); both signs of q & 2 go into 1/r
  const double K = __hiloint2double(__double2hiint(y) ^ (int)((unsigned)q << 30 & 0x80000000u), __double2loint(y));
  const double sr = u * K * ps, cr = K * pc;
  return make_double2((q & 1) ? -sr : cr, (q & 1) ? cr : sr);
}
__device__ __forceinline__ double2 green64(double dx, double dy, double dz, double kq) {
  return green64_r<true>(fma(dx, dx, fma(dy, dy, dz * dz)), kq);
}

}  // namespace dfb
