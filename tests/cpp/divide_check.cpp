// Errors of SharedDivisor against exact quotients, in units in the last place.
#include <stdint.h>
#include <stdio.h>

#include <cmath>
#include <limits>

#include "sns_divide.cuh"

typedef __float128 quad;  // 113 bits: quotients to 2^-60 ulp

static uint64_t state = 88172645463325252ull;
static uint64_t rnd() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}
static double mantissa() { return 1.0 + (double)(rnd() >> 12) * std::ldexp(1.0, -52); }

static double worst = 0, worst_tiny = 0;
static long differ = 0, total = 0;

static void check(double den, double v) {
  const double q = sns::SharedDivisor(den).under(v), d = v / den;
  const quad off = (quad)q - (quad)v / (quad)den;
  const quad err = off < 0 ? -off : off;
  const double a = std::fabs(d);
  int e = -1073;
  if (a > 0) std::frexp(a, &e);
  // (in quad: the smallest double is no number of use in a double quotient)
  const quad ulp = (quad)std::fmax(std::ldexp(1.0, e - 53), std::numeric_limits<double>::denorm_min());
  const double units = (double)(err / ulp);
  total++;
  if (a < std::ldexp(1.0, -960)) {
    worst_tiny = std::fmax(worst_tiny, units);
  } else {
    differ += q != d;
    worst = std::fmax(worst, units);
  }
}

int main() {
  // every |k|^2 of boxes up to 1024 per side, four numerators each
  for (int k2 = 1; k2 <= 3 * 512 * 512; k2++)
    for (int i = 0; i < 4; i++) check(k2, std::ldexp(mantissa(), (int)(rnd() % 120) - 60));
  // 1 + nu K/2 |k|^2, and any divisor from 1 on
  for (int i = 0; i < 4000000; i++) {
    check(1.0 + std::ldexp(mantissa(), (int)(rnd() % 40) - 30), std::ldexp(mantissa(), 20));
    check(std::ldexp(mantissa(), (int)(rnd() % 200)), -std::ldexp(mantissa(), (int)(rnd() % 400) - 200));
  }
  for (int i = 0; i < 1000000; i++)
    check(1.0 + std::ldexp(mantissa(), (int)(rnd() % 40) - 20),
          std::ldexp(mantissa(), -(int)(rnd() % 110) - 960));
  // what is not a number of that range
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  int special = 0;
  const double dens[] = {1.0, 3.0, 1.5e9, inf};
  const double vs[] = {0.0, -0.0, inf, -inf, nan, 1e308, -1.7976931348623157e308};
  for (double d : dens)
    for (double v : vs) {
      const double q = sns::SharedDivisor(d).under(v), w = v / d;
      if (!((q != q && w != w) || q == w)) special++;
    }
  printf("%.17g %.17g %ld %ld %d\n", worst, worst_tiny, differ, total, special);
  return 0;
}
