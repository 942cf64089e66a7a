// mul_int wherever mul_int_ok admits both factors, against the product, at
// the ends of the admitted range: every binade within four of either end and
// the middle ones, the first, a middle and the last significand of each, both
// signs.  Prints the products compared and the number different.
#include <cmath>
#include <cstdio>
#include <vector>

#include "ddmath.cuh"

using namespace a2c;

int main() {
  std::vector<double> v;
  for (int e : {-1022, -1021, -515, -514, -513, -512, -511, -510, -509, -508, -1, 0, 1, 508, 509, 510, 511, 512, 513, 514, 515, 1023})
    for (double m : {1.0, 1.5, 1.9999999999999998})
      for (double sign : {1.0, -1.0}) v.push_back(sign * std::ldexp(m, e));
  v.push_back(0.0);
  v.push_back(std::ldexp(1.0, -1074));
  v.push_back(HUGE_VAL);
  v.push_back(std::nan(""));
  long n = 0, bad = 0;
  for (double a : v)
    for (double b : v) {
      if (!dd::mul_int_ok(a) || !dd::mul_int_ok(b)) continue;
      ++n;
      bad += !(dd::mul_int(a, b) == a * b);
    }
  std::printf("%ld %ld\n", n, bad);
  return 0;
}
