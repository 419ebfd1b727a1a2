// The FP64 near field's kernel evaluation on the host: special values, and
// its error against quad precision.
#include <algorithm>
#include <cassert>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include <quadmath.h>

#define __device__
#define __forceinline__ inline
struct double2 {
  double x, y;
};
static double2 make_double2(double x, double y) { return {x, y}; }
static uint64_t bits(double x) {
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
}
static double from_bits(uint64_t b) {
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}
static int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static int __double2loint(double x) { return (int)bits(x); }
static long long __double_as_longlong(double x) { return (long long)bits(x); }
static double __hiloint2double(int hi, int lo) { return from_bits((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo); }
using std::fma;
static __float128 fma(__float128 a, __float128 b, __float128 c) { return fmaq(a, b, c); }
using std::max;
// an estimate off by up to 2^-20, to either side
static double rsqrt_approx64(double x) { return 1. / std::sqrt(x) * (1. + ((bits(x) & 1) ? 9e-7 : -9e-7)); }

#include "../../defmm_b200/csrc/green64.cuh"

int main() {
  using dfb::green64_r;
  // coincident pairs give nothing, pairs at 1e-8 count
  for (double R : {0., 1e-300, 1e-20, std::nextafter(1e-16, 0.)}) {
    const double2 g = green64_r<true>(R, 3.);
    assert(g.x == 0. && g.y == 0.);
  }
  assert(std::fabs(green64_r<true>(1e-16, 3.).x * 1e-8 - 1.) < 1e-14);
  // a NaN distance (of either sign) gives NaN, guarded or not
  for (uint64_t sign : {uint64_t(0), uint64_t(1) << 63})
    for (uint64_t low : {uint64_t(0), uint64_t(5), uint64_t(0xffffffff)}) {
      const double R = from_bits(0x7ff8000000000000ull | sign | low);
      const double2 a = green64_r<true>(R, 3.), b = green64_r<false>(R, 3.);
      assert(std::isnan(a.x) && std::isnan(a.y) && std::isnan(b.x) && std::isnan(b.y));
    }
  // where the guard does not act it changes nothing
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> U(0., 1.);
  for (int i = 0; i < 100000; i++) {
    const double R = std::pow(10., -15.9 + 20. * U(rng)), kq = 100. * U(rng);
    const double2 a = green64_r<true>(R, kq), b = green64_r<false>(R, kq);
    assert(a.x == b.x && a.y == b.y);
  }
  // the rounded coefficients, evaluated in quad precision, against sin and cos:
  // half an ulp of the leading ones (1.1e-16 of 1.57, the sine's) bounds what
  // rounding can do, the stated 5.0e-17 and 1.6e-17 what it did
  __float128 es = 0, ec = 0;
  for (int i = 1; i <= 20000; i++) {
    const __float128 u = (__float128)i / 40000, z = u * u;
    const __float128 s = sinq(M_PI_2q * u), c = cosq(M_PI_2q * u);
    es = std::max(es, fabsq(u * dfb::quarter_sin(z) / s - 1));
    ec = std::max(ec, fabsq(dfb::quarter_cos(z) - c));
  }
  if (es > 5.05e-17Q || ec > 1.65e-17Q) {
    std::printf("sine %.3g, cosine %.3g\n", (double)es, (double)ec);
    return 1;
  }
  std::puts("ok");
  return 0;
}
