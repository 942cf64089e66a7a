// The pair functions of eam64.cuh as the FP64 pair kernels evaluate them:
// the same bits (tests/test_fp64_forms.py compares them on the host)
// in fewer FP64 operations.  GB300's FP64 pipe takes two lanes per SM and
// clock, so a warp's FP64 instruction occupies its scheduler's share of the
// pipe for 64 clocks and the count of such instructions is the time of
// these kernels.  What is spared:
//   * phi_Pd(x) holds f_Pd(x1) with x1 = (x / 5) * 5, and f_Pd depends on
//     its argument through r = x / 5 alone.  x1 is x or its neighbor; x1 / 5
//     rounds to the same r whenever x's significand is 1.25 or more (then
//     ulp(r) = ulp(x) / 4 and x1 / 5 lies within 0.4 ulp(r) of r), and often
//     otherwise, so the f_Pd values of f_Pd' serve phi_Pd' too: three
//     evaluations in place of five outside [2, 2.5) and [4, 5) A;
//   * x / 5 by two operations and the other quotients by four, correctly
//     rounded (div5, Divisor);
//   * comparisons with the switch radii on the bits, by integer operations;
//   * multiplications whose factors are known not to be zero on the integer
//     pipes (ddmath.cuh mul_int).
//   * the exponentials mostly on the integer pipes (ddmath.cuh fexp_fixed).
// FP64 instructions per point, all pair types of a bulk site and the
// additions included, and pass 2 at 262,144 sites: about 330 / 127 ms with
// the first three, 221 / 106 ms with the fourth (the pipe at 83% of its two
// lanes, what a chain of FMAs reaches), 170 / 92 ms with all, where the
// pipe, the integer pipes and the latency of both hold each other up: fewer
// FP64 instructions still (the points' products by mul_int: 161) take
// longer (99 ms).
// The fast forms hold for kPairMin <= x < kPairMax (in_pair_range); callers
// take eam64.cuh's functions elsewhere.
#pragma once

#include "eam64.cuh"

#if defined(__CUDACC__)
#define A2C_EAM __host__ __device__ __forceinline__
#else
#define A2C_EAM inline
#endif

namespace a2c {
namespace eam64 {

constexpr double kPairMin = 0.0625, kPairMax = 128.0;

// a > b for positive finite doubles
A2C_EAM bool above(double a, double b) {
  const int ha = dd::hi_word(a), hb = dd::hi_word(b);
  return ha > hb || (ha == hb && (unsigned)dd::lo_word(a) > (unsigned)dd::lo_word(b));
}
// kPairMin <= x < kPairMax, both powers of two
A2C_EAM bool in_pair_range(double x) {
  return (unsigned)(dd::hi_word(x) - 0x3fb00000) < (unsigned)(0x40600000 - 0x3fb00000);
}

// x / 5, correctly rounded for normal results: 1/5 as hi + lo, one fused
// operation on the exact product's head.  A quotient by 5 is at least 1/20
// ulp from every midpoint of two doubles (x - 5 m is a multiple of 1/16 ulp
// of x, and not zero, for a midpoint m), the sum below is within 2^-50 ulp
// of it before its one rounding.
A2C_EAM double div5(double x) { return fma(x, 0.2, dd::mul_int(x, -1.1102230246251565e-17)); }

// Quotients by one divisor b, correctly rounded: z = 1/b rounded to
// nearest, with its error zl a quotient q within one ulp, then Markstein's
// correction q + (a - q b) z (Markstein 1990, theorem on final rounding).
// The remainder must not underflow: exact_for(a) is the range of
// numerators (zero included) for divisors between 2^-100 and 2^100.
struct Divisor {
  double b, z, zl;
};
A2C_EAM Divisor divisor(double b) {
  Divisor d;
  d.b = b;
#if defined(__CUDA_ARCH__)
  d.z = __drcp_rn(b);
#else
  d.z = 1.0 / b;
#endif
  d.zl = fma(-b, d.z, 1.0) * d.z;
  return d;
}
A2C_EAM double quotient(double a, const Divisor &d) {
  const double q = fma(a, d.z, a * d.zl);
  return fma(fma(-d.b, q, a), d.z, q);
}
A2C_EAM bool exact_for(double a) {
  const unsigned h = (unsigned)dd::hi_word(a) & 0x7fffffffu;
  return h - 0x10000000u < 0x60000000u || (h | (unsigned)dd::lo_word(a)) == 0;  // 2^-767 <= |a| < 2^769, or 0
}
// a / d.b for any a
A2C_EAM double divide(double a, const Divisor &d) { return exact_for(a) ? quotient(a, d) : a / d.b; }

// e^x: FIXED, the form with three FP64 operations and a long chain of
// integer ones, for kernels whose warps wait for the FP64 pipe; else the one
// with 13, which is done sooner where a scheduler has one warp to run (512
// sites, pass 2: 0.51 against 0.55 ms).
template <bool FIXED>
A2C_EAM double exp_of(double x) {
  return FIXED ? dd::fexp(x) : dd::fexp_soon(x);
}

// f_Pd as a function of r = x / 5 (potential.cpp:64-98).  Multiplications
// by mul_int where no factor can be zero: below the switch radius r <= 1,
// the quadratics have no real root, and r meets 0.53 and 0.136 only.
template <bool FIXED>
A2C_EAM double f_Pd_at(double r) {
  using dd::mul_int;
  const double x1 = mul_int(r, 5.0);
  if (above(x1, 5.0)) return 0.001510569378297 * exp_of<FIXED>(-0.077976566126292 / 0.001510569378297 * (x1 - 5.0));
  double ra = mul_int(r, mul_int(r - 2.7267629107325706, r) + 1.8716766113599643);
  ra = mul_int(ra, mul_int(r - 2.50290548851635, r) + 1.668549182690922);
  ra = mul_int(ra, mul_int(r - 2.0924467509943674, r) + 1.3150372774478005);
  ra = mul_int(ra, mul_int(r - 1.564328475106985, r) + 0.8987511149780485);
  ra = mul_int(ra, mul_int(r - 1.009780903403673, r) + 0.5124363774128722);
  ra = mul_int(ra, r * (r - 0.5304054524800665) + 0.2169886022464641);
  ra = mul_int(ra, r * (r - 0.1356566408715063) + 0.035852347523891395);
  return -0.02972698211669922 +
         r * (0.6676807403564453 +
              r * (-255.8965835571289 + r * (14673.409149169922 + mul_int(ra, -2.597301181336601e7))));
}
// x1 / 5 for x1 = r * 5, r = x / 5: r itself where x's significand is 1.25
// or more (see above)
A2C_EAM double second_fifth(double x, double r) {
  return (dd::hi_word(x) & 0xfffff) >= 0x40000 ? r : div5(dd::mul_int(r, 5.0));
}
// phi_Pd with r = x / 5 and f = f_Pd(x1) (potential.cpp:126-155).  Below
// the switch radius r <= 1.01; the factor r - 0.424 can be zero, and then
// so is the product from there on.
template <bool FIXED>
A2C_EAM double phi_Pd_at(double r, double f) {
  using dd::mul_int;
  const double x1 = mul_int(r, 5.0);
  if (above(x1, 5.05)) return -0.016958780164980 * exp_of<FIXED>(0.089019679316328 / -0.016958780164980 * (x1 - 5.05));
  double y = mul_int(r - 1.0699996145674568, -79415.24035137112);
  y = mul_int(r - 1.06015072612581, y);
  y = y * (r - 0.42433991011376526);
  if ((dd::hi_word(y) & 0x7fffffff) == 0) return 0.0 + (2 * 0.251546) * f;
  y = mul_int(r + 0.06169160085238687, y);
  y = mul_int(mul_int(r - 2.0586473420376348, r) + 1.0683922574015199, y);
  y = mul_int(mul_int(r - 1.6696359816422877, r) + 0.7337878627470482, y);
  y = mul_int(mul_int(r - 1.1690370066230809, r) + 0.3909805777737639, y);
  y = mul_int(r * (r - 0.2635598721249787) + 0.033551116514910245, y);
  return y + (2 * 0.251546) * f;
}
template <bool FIXED>
A2C_EAM double f_Pd_pos(double x) { return f_Pd_at<FIXED>(div5(x)); }
template <bool FIXED>
A2C_EAM double f_H_pos(double x) {
  if (above(x, 5.35)) return 0.009986990526578 * exp_of<FIXED>(-0.013075667086408 / 0.009986990526578 * (x - 5.35));
  return dd::mul_int(exp_of<FIXED>(dd::mul_int(x, -1.30927)), 11.0025);
}
// phi_PdH (potential.cpp:162-177) and phi_H (185-200): one form, constants
// by pair type
template <bool FIXED>
A2C_EAM double morse_pos(bool pdh, double x) {
  if (above(x, 5.35))
    return pdh ? -3.353001113951400e-04 * exp_of<FIXED>(7.147062196813336e-04 / -3.353001113951400e-04 * (x - 5.35))
               : -0.003702722457147 * exp_of<FIXED>(0.005465945471933 / -0.003702722457147 * (x - 5.35));
  const double D = pdh ? 0.2494540 : 0.0661496, alpha = pdh ? 4.82613 : 3.67263, beta = pdh ? 2.13158 : 1.47797;
  const double t = x - (pdh ? 1.50964 : 2.51980);
  return D * (dd::mul_int(exp_of<FIXED>(-alpha * t), beta) - dd::mul_int(exp_of<FIXED>(-beta * t), alpha));
}

// What one quadrature point of a pair at distance s takes from the pair
// functions: da, db the density derivatives that F'(rho_i) and F'(rho_j)
// multiply (f' of the neighbor's and of the site's own species), the pair
// function and its derivative; derivatives by central differences of step e
// (h: the divisor 2 e).
struct PairPoint {
  double da, db, phi, dphi;
};
#if defined(__CUDACC__)
#define A2C_COLD static __host__ __device__ __noinline__
#else
#define A2C_COLD inline
#endif
// outside the fast forms' range: the plain functions, out of line
A2C_COLD PairPoint pair_point_plain(bool iPd, bool jPd, double s, double e) {
  PairPoint p;
  const double fP = (iPd || jPd) ? f_Pd_d(s, e) : 0.0, fH = (iPd && jPd) ? 0.0 : f_H_d(s, e);
  p.da = jPd ? fP : fH;
  p.db = iPd ? fP : fH;
  p.phi = (iPd && jPd) ? phi_Pd(s) : (iPd || jPd) ? phi_PdH(s) : phi_H(s);
  p.dphi = (iPd && jPd) ? phi_Pd_d(s, e) : (iPd || jPd) ? phi_PdH_d(s, e) : phi_H_d(s, e);
  return p;
}
A2C_COLD double density_plain(bool jPd, double s) { return jPd ? f_Pd(s) : f_H(s); }
#undef A2C_COLD

template <bool FIXED = true>
A2C_EAM PairPoint pair_point(bool iPd, bool jPd, double s, double e, const Divisor &h) {
  const double xp = s + e, xm = s - e;
  PairPoint p;
  if (!in_pair_range(xp) || !in_pair_range(xm)) return pair_point_plain(iPd, jPd, s, e);
  // s, then s + e and s - e in one rolled loop: with the functions written
  // out for each the instruction caches did not hold the kernel (pass 2 at
  // 262,144 sites 112 ms, rolled 106)
  const bool pp = iPd && jPd, pdh = iPd != jPd;
  double fP1 = 0.0, fH1 = 0.0, ph1 = 0.0, dP = 0.0, dH = 0.0;
  p.phi = p.dphi = 0.0;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int v = 0; v < 3; ++v) {
    const double x = v == 0 ? s : v == 1 ? xp : xm;
    double fP = 0.0, fH = 0.0, ph;
    if (pp) {  // f_Pd at r (not needed at s itself), and where it differs at phi_Pd's own fifth
      const double r = div5(x), r2 = second_fifth(x, r);
      double at = v == 0 ? r2 : r, f;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
      for (bool first = true;; first = false) {
        f = f_Pd_at<FIXED>(at);
        if (first) fP = f;
        if (at == r2) break;
        at = r2;
      }
      ph = phi_Pd_at<FIXED>(r, f);
    } else {
      if (v > 0) {
        if (pdh) fP = f_Pd_at<FIXED>(div5(x));
        fH = f_H_pos<FIXED>(x);
      }
      ph = morse_pos<FIXED>(pdh, x);
    }
    if (v == 0) {
      p.phi = ph;
    } else if (v == 1) {
      fP1 = fP;
      fH1 = fH;
      ph1 = ph;
    } else {
      dP = fP1 - fP;
      dH = fH1 - fH;
      p.dphi = divide(ph1 - ph, h);
    }
  }
  const double fP = (iPd || jPd) ? divide(dP, h) : 0.0, fH = pp ? 0.0 : divide(dH, h);
  p.da = jPd ? fP : fH;
  p.db = iPd ? fP : fH;
  return p;
}
// the density a neighbor at distance s adds at one point
template <bool FIXED = true>
A2C_EAM double density_point(bool jPd, double s) {
  if (!in_pair_range(s)) return density_plain(jPd, s);
  return jPd ? f_Pd_pos<FIXED>(s) : f_H_pos<FIXED>(s);
}

}  // namespace eam64
}  // namespace a2c

#undef A2C_EAM
