// Compares, bit for bit on the host, the fast FP64 forms of the device code
// with the plain ones they stand for: ddmath.cuh's quick exp, log and pow
// (where their rounding test settles the result) and fexp_mid, and
// mul_int, and
// eam64_pair.cuh's pair functions and quotients.  argv: form, count, seed.
// Prints "<compared> <settled> <different>".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>

#include "eam64_pair.cuh"

using namespace a2c;

int main(int argc, char **argv) {
  if (argc < 4) return 2;
  const std::string form = argv[1];
  const long count = std::atol(argv[2]);
  std::mt19937_64 g(std::strtoull(argv[3], nullptr, 10));
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long n = 0, settled = 0, bad = 0;
  auto tally = [&](bool ok, double q, double want) {
    ++n;
    if (!ok) return;
    ++settled;
    if (!(q == want)) ++bad;  // zeros compare equal whatever their sign: the kernels only add them to sums
  };
  for (long i = 0; i < count; ++i) {
    double q = 0.0;
    if (form == "exp") {
      const double x = i % 3 == 0 ? (U(g) - 0.5) * 1398 : i % 3 == 1 ? (U(g) - 0.5) * 40 : (U(g) - 0.5) * std::ldexp(1.0, -(int)(g() % 60));
      const bool ok = dd::quick_cr_exp(x, q);
      tally(ok, q, dd::series_exp(x));
      double up = 0.0, down = 0.0;
      const int both = dd::quick_cr_exp_both(x, up, down);
      tally(both & 1, up, dd::series_exp(x));
      tally(both & 2, down, dd::series_exp(-x));
    } else if (form == "log") {
      const double t = U(g);
      const double x = i % 4 == 0 ? std::exp((t - 0.5) * 1300) : i % 4 == 1 ? t / (1.0 - t) : i % 4 == 2 ? 1.0 + (t - 0.5) * std::ldexp(1.0, -(int)(g() % 50)) : 60 * t;
      if (!(x > 1e-300 && x < 1e300)) continue;
      const bool ok = dd::quick_cr_log(x, q);
      tally(ok, q, dd::series_log(x));
    } else if (form == "pow") {
      const double ys[3] = {1.18860, 2.18860, 3.18860};  // F_H's exponents
      const double u = i % 2 ? 0.0540638 + 60 * U(g) : 0.0540638 + 5 * std::exp((U(g) - 1) * 20);
      const double y = i % 7 == 6 ? (U(g) - 0.5) * 20 : ys[i % 3];
      const bool ok = dd::quick_cr_pow(u, y, q);
      tally(ok, q, dd::series_pow(u, y));
    } else if (form == "fexp") {
      const double x = i % 2 ? (U(g) - 0.5) * 1415.9 : (U(g) - 0.5) * std::ldexp(80.0, -(int)(g() % 70));
      tally(true, dd::fexp_mid(x), dd::fexp(x));
      // near multiples of ln2/64, where the reduced argument is small
      const double y = (double)((long)(g() % 80000) - 40000) * 0.010830424696249145 + (U(g) - 0.5) * std::ldexp(1.0, -(int)(g() % 30));
      tally(true, dd::fexp_fixed(x), dd::fexp(x));
      if (std::fabs(y) < 708) tally(true, dd::fexp_fixed(y), dd::fexp(y));
    } else if (form == "mul") {  // both significands random, short, or all ones at the end
      auto value = [&](long k) {
        unsigned long long b = (g() >> 12) | (0x3ffull - 500 + g() % 1000) << 52 | g() << 63;
        if (k % 4 == 1) b = b >> 26 << 26;
        if (k % 4 == 2) b |= 0xfffffffffff00ull;
        double x;
        std::memcpy(&x, &b, sizeof(x));
        return x;
      };
      const double a = value(i), b = value(i / 4);
      tally(dd::mul_int_ok(a) && dd::mul_int_ok(b), dd::mul_int(a, b), a * b);
    } else if (form == "quotient") {
      const double b = std::ldexp(1.0 + U(g), (int)(g() % 8) - 4);
      double a = (U(g) - 0.5) * std::ldexp(1.0, (int)(g() % 900) - 450);
      if (i % 7 == 0) a = b * (double)(g() % 4096);
      if (i % 97 == 0) a *= 1e-290;
      tally(true, eam64::divide(a, eam64::divisor(b)), a / b);
      tally(true, eam64::div5(b), b / 5.0);
    } else if (form == "pair") {
      const double radii[5] = {5.0, 5.05, 5.35, 3.0, 1.0};
      const double e = i % 11 == 0 ? 1e-5 * (1 + U(g)) : 1e-5;
      const double s = i % 5 == 0   ? 0.9 + 5 * U(g)
                       : i % 5 == 1 ? radii[g() % 5] + (U(g) - 0.5) * 1e-4
                       : i % 5 == 2 ? radii[g() % 5] + ((int)(g() % 9) - 4) * e
                       : i % 5 == 3 ? 0.01 * std::exp(std::log(30000.0) * U(g))
                                    : 1.5 + 3.6 * U(g);
      const eam64::Divisor h = eam64::divisor(2.0 * e);
      for (int t = 0; t < 4; ++t) {
        const bool iPd = t & 1, jPd = t & 2;
        const eam64::PairPoint p = eam64::pair_point(iPd, jPd, s, e, h);
        const double fP = eam64::f_Pd_d(s, e), fH = eam64::f_H_d(s, e);
        tally(true, p.da, jPd ? fP : fH);
        tally(true, p.db, iPd ? fP : fH);
        tally(true, p.phi, iPd && jPd ? eam64::phi_Pd(s) : iPd || jPd ? eam64::phi_PdH(s) : eam64::phi_H(s));
        tally(true, p.dphi,
              iPd && jPd ? eam64::phi_Pd_d(s, e) : iPd || jPd ? eam64::phi_PdH_d(s, e) : eam64::phi_H_d(s, e));
      }
      tally(true, eam64::density_point(true, s), eam64::f_Pd(s));
      tally(true, eam64::density_point(false, s), eam64::f_H(s));
    } else {
      return 2;
    }
  }
  std::printf("%ld %ld %ld\n", n, settled, bad);
  return 0;
}
