// Near-correctly-rounded exp, log and pow for the FP64 plain form, built on
// double-double ("dd") arithmetic: Dekker's and Knuth's error-free
// transformations (two-sum, two-product via FMA), as used in Bailey's QD
// library.  Why: the reference differentiates F_H (three pow calls) by a
// central difference with step 1e-5, which multiplies a one-ulp difference
// between two libm implementations by ~1e5.  Rounding the exact value
// correctly makes the device result agree with any accurate C library
// (glibc's pow/exp/log are within ~0.52 ulp) except in rare near-midpoint
// cases, instead of in a sizeable fraction of calls.
//
// Method (published, textbook):
//   exp(a):  k = rint(a/ln2), r = (a - k ln2)/2^10 in dd, e^r - 1 by its
//            Taylor series to r^11 in dd, then (1+s)^(2^10) by ten
//            squarings of the expm1 form s <- 2s + s^2, times 2^k.
//   log(u):  y0 = log(u) in double, one Newton step y = y0 + t - t^2/2
//            with t = u*exp(-y0) - 1 evaluated in dd.
//   pow(u,y) = exp(y * log(u)) with the product and exp in dd.
// The Taylor coefficients 1/n! and ln 2 are mathematical constants split
// into hi + lo doubles.  All functions are __host__ __device__ so the host
// build can be tested against the C library directly.
//
// fexp is the fast exp of the per-pair-point EAM terms: Tang's table-driven
// method with 64 subintervals, x = (64k + j) ln2/64 + r, |r| <= ln2/128,
// e^x = 2^k 2^(j/64) (1 + p(r)), p the degree-6 Taylor polynomial of
// e^r - 1 (truncation < 4e-20), 2^(j/64) held as hi + lo, reduction and
// reconstruction with FMA.  Its error is ~0.5 ulp and, being plain IEEE
// arithmetic, it gives the same bits on the host and on the device, which
// lets the CPU oracle reproduce the GPU plain form exactly.
//
// On the device cr_exp, cr_log and cr_pow first try quick forms (quick_exp,
// quick_log): table-driven argument reduction (Tang 1989, 1990) carried in
// hi + lo doubles, 25-40 FP64 operations with errors below 2^-70, against
// 600-700 for the double-double series above.  Ziv's rounding test (Ziv
// 1991) then decides: when hi + (lo - bound) and hi + (lo + bound) round to
// the same double, every value within the bound rounds to it, the
// double-double result among them, so the quick result has its bits; else (about once in 2^15 calls) the series runs.  GB300
// has two FP64 lanes per SM and clock, so these operation counts are the
// time of the occupancy update and of the per-site functions.  The host
// build keeps the series alone: the oracle stays an independent check.
#pragma once

#include <cmath>
#include <cstring>

namespace a2c {
namespace dd {

#if defined(__CUDACC__)
#define A2C_HD __host__ __device__ __forceinline__
#else
#define A2C_HD inline
#endif

struct D2 {
  double hi, lo;
};

A2C_HD D2 two_sum(double a, double b) {
  const double s = a + b;
  const double bb = s - a;
  const double e = (a - (s - bb)) + (b - bb);
  return {s, e};
}
A2C_HD D2 quick_two_sum(double a, double b) {
  const double s = a + b;
  return {s, b - (s - a)};
}
// a * b rounded, where its rounding error is also carried: never contracted
// with a sum that it enters (k_mixed.cu is compiled with contraction; a
// product fused into the sum would count its error twice).
A2C_HD double rounded_product(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;  // host builds: -ffp-contract=off
#endif
}
A2C_HD D2 two_prod(double a, double b) {
  const double p = rounded_product(a, b);
  return {p, fma(a, b, -p)};
}
A2C_HD D2 add(D2 a, D2 b) {
  D2 s = two_sum(a.hi, b.hi);
  const D2 t = two_sum(a.lo, b.lo);
  s.lo += t.hi;
  s = quick_two_sum(s.hi, s.lo);
  s.lo += t.lo;
  return quick_two_sum(s.hi, s.lo);
}
A2C_HD D2 mul(D2 a, D2 b) {
  D2 p = two_prod(a.hi, b.hi);
  p.lo += a.hi * b.lo + a.lo * b.hi;
  return quick_two_sum(p.hi, p.lo);
}
A2C_HD D2 mul_d(D2 a, double b) {
  D2 p = two_prod(a.hi, b);
  p.lo += a.lo * b;
  return quick_two_sum(p.hi, p.lo);
}

// e^a for a double-double argument; |a| < 700.
A2C_HD D2 exp_dd(D2 a) {
  const D2 LN2 = {0.6931471805599453, 2.3190468138462996e-17};
  const double k = rint(a.hi / LN2.hi);
  D2 r = add(a, mul_d(LN2, -k));
  r.hi *= 0.0009765625;  // 2^-10, exact
  r.lo *= 0.0009765625;
  // Taylor coefficients 1/n!, n = 2..11
  const D2 C[10] = {{0.5, 0.0},
                    {0.16666666666666666, 9.25185853854297e-18},
                    {0.041666666666666664, 2.3129646346357427e-18},
                    {0.008333333333333333, 1.1564823173178714e-19},
                    {0.001388888888888889, -5.300543954373577e-20},
                    {0.0001984126984126984, 1.7209558293420705e-22},
                    {2.48015873015873e-05, 2.1511947866775882e-23},
                    {2.7557319223985893e-06, -1.858393274046472e-22},
                    {2.755731922398589e-07, 2.3767714622250297e-23},
                    {2.505210838544172e-08, -1.448814070935912e-24}};
  // s = r + r^2/2! + ... + r^11/11!  (Horner on the coefficients)
  D2 p = C[9];
  for (int n = 8; n >= 0; --n) p = add(mul(p, r), C[n]);
  D2 s = add(mul(p, mul(r, r)), r);
  for (int i = 0; i < 10; ++i) s = add(mul_d(s, 2.0), mul(s, s));  // (1+s)^2 - 1
  D2 e = add({1.0, 0.0}, s);
  const int ki = (int)k;
  return {ldexp(e.hi, ki), ldexp(e.lo, ki)};
}

// log(u) as double-double, u > 0 finite.
A2C_HD D2 log_dd(double u) {
  const double y0 = log(u);
  const D2 e = exp_dd({-y0, 0.0});
  const D2 t = add(mul_d(e, u), {-1.0, 0.0});  // u e^{-y0} - 1, |t| ~ 1e-16
  const double t2 = 0.5 * t.hi * t.hi;
  return add({y0, 0.0}, add(t, {-t2, 0.0}));
}

A2C_HD double round_dd(D2 a) { return a.hi + a.lo; }

// 2^(j/64), j = 0..63, split into hi + lo
#define A2C_EXP2_TABLE \
    {1.0, 0.0}, \
    {1.0108892860517005, -1.5234778603368577e-17}, \
    {1.0218971486541166, 5.109225028973444e-17}, \
    {1.0330248790212284, 7.600838874027088e-18}, \
    {1.0442737824274138, 8.551889705537965e-17}, \
    {1.0556451783605572, 1.759325738772092e-18}, \
    {1.0671404006768237, -7.899853966841582e-17}, \
    {1.0787607977571199, -6.656660436056593e-17}, \
    {1.0905077326652577, -3.046782079812471e-17}, \
    {1.102382583307841, 5.2660368715706944e-17}, \
    {1.1143867425958924, 1.0410278456845571e-16}, \
    {1.1265216186082418, 5.165856758795457e-17}, \
    {1.1387886347566916, 8.912812676025408e-17}, \
    {1.1511892299529827, 3.250710218863827e-17}, \
    {1.1637248587775775, 3.8292048369240935e-17}, \
    {1.1763969916502812, 5.554203254218079e-17}, \
    {1.189207115002721, 3.982015231465646e-17}, \
    {1.202156731452703, 6.644981499252301e-17}, \
    {1.215247359980469, -7.712630692681488e-17}, \
    {1.22848053610687, -1.89878163130253e-17}, \
    {1.241857812073484, 4.658027591836937e-17}, \
    {1.255380757024691, -6.7113898212968784e-18}, \
    {1.2690509571917332, 2.667932131342186e-18}, \
    {1.2828700160787783, 1.713594918243561e-17}, \
    {1.2968395546510096, 2.5382502794888315e-17}, \
    {1.3109612115247644, -7.181536135519454e-17}, \
    {1.3252366431597413, -2.8587312100388614e-17}, \
    {1.339667524053303, 8.927282594831732e-17}, \
    {1.3542555469368927, 7.70094837980299e-17}, \
    {1.3690024229745905, 9.593797919118849e-17}, \
    {1.383909881963832, -6.770511658794786e-17}, \
    {1.3989796725383112, -9.614213209051323e-17}, \
    {1.4142135623730951, -9.667293313452913e-17}, \
    {1.42961333839197, -1.2031642489053655e-17}, \
    {1.4451808069770467, -3.0237581349939873e-17}, \
    {1.460917794180647, -5.600377186075216e-17}, \
    {1.4768261459394993, -3.483994556892796e-17}, \
    {1.4929077282912648, 1.4192920154284036e-17}, \
    {1.5091644275934228, -1.016455327754295e-16}, \
    {1.5255981507445384, -1.1024941712342561e-16}, \
    {1.5422108254079407, 7.949834809697621e-17}, \
    {1.559004400237837, 3.7812070533575275e-17}, \
    {1.5759808451078865, -1.0136916471278304e-17}, \
    {1.593142151342267, -1.0094406542311964e-16}, \
    {1.6104903319492543, 2.4707192569797888e-17}, \
    {1.6280274218573478, -6.712955084707084e-17}, \
    {1.645755478153965, -1.0125679913674773e-16}, \
    {1.6636765803267364, 5.8909926967131e-17}, \
    {1.681792830507429, 8.199010020581497e-17}, \
    {1.7001063537185235, -8.0237193703977e-18}, \
    {1.718619298122478, -1.851380418263111e-17}, \
    {1.7373338352737062, 3.164389299292957e-17}, \
    {1.7562521603732995, 2.960140695448873e-17}, \
    {1.7753764925265212, 6.429731796556572e-17}, \
    {1.7947090750031072, 1.8227458427912087e-17}, \
    {1.8142521755003989, -9.969531538920349e-17}, \
    {1.8340080864093424, 3.283107224245627e-17}, \
    {1.8539791250833855, 9.761887490727594e-17}, \
    {1.8741676341103, -6.122763413004143e-17}, \
    {1.8945759815869656, 3.4034035352165297e-17}, \
    {1.9152065613971474, -1.0619946056195963e-16}, \
    {1.9360617934922943, 1.0332385960676326e-16}, \
    {1.9571441241754002, 8.960767791036668e-17}, \
    {1.978456026387951, 4.0388753109278167e-17}
#if defined(__CUDACC__)
__device__ const __align__(16) double kExp2TabDev[64][2] = {A2C_EXP2_TABLE};
#endif
static const double kExp2TabHost[64][2] = {A2C_EXP2_TABLE};
#undef A2C_EXP2_TABLE

A2C_HD int hi_word(double x) {
#if defined(__CUDA_ARCH__)
  return __double2hiint(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return (int)(b >> 32);
#endif
}
A2C_HD int lo_word(double x) {
#if defined(__CUDA_ARCH__)
  return __double2loint(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, 8);
  return (int)(unsigned)b;
#endif
}
A2C_HD double from_words(int hi, int lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double(hi, lo);
#else
  const unsigned long long b = ((unsigned long long)(unsigned)hi << 32) | (unsigned)lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// a * b, correctly rounded, in integer operations: the 106-bit product of
// the significands, normalized, rounded to nearest even by one chain of
// carries that also adds the exponent and the sign.  Both factors and the
// product must be normal (mul_int_ok).  About 28 instructions of the integer
// pipes (four 32 x 32 + 64 multiply-adds among them), which a GB300
// scheduler issues in the time its two-lane FP64 pipe needs for half an
// instruction: a kernel bound by that pipe gains by moving multiplications
// off it.
A2C_HD double mul_int(double a, double b) {
  const unsigned ah = (unsigned)hi_word(a), al = (unsigned)lo_word(a);
  const unsigned bh = (unsigned)hi_word(b), bl = (unsigned)lo_word(b);
  const unsigned ma = (ah & 0xfffffu) | 0x100000u;  // a's significand: 53 bits
  const unsigned mb = (bh & 0xfffffu) | 0x100000u;
  const unsigned nh = (mb << 11) | (bl >> 21), nl = bl << 11;  // b's, shifted to 64 bits
  const unsigned long long p0 = (unsigned long long)al * nl;
  const unsigned long long t = (unsigned long long)ma * nl + (p0 >> 32);
  const unsigned long long u = (unsigned long long)al * nh + (unsigned)t;
  const unsigned long long h = (unsigned long long)ma * nh + (t >> 32) + (u >> 32);  // 2^51 <= h < 2^53
  const unsigned s = (unsigned)(h >> 32) < 0x100000u ? 1u : 0u;
  const unsigned e = (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x3ff00000u - (s << 20);
#if defined(__CUDA_ARCH__)
  const unsigned hh = __funnelshift_l((unsigned)h, (unsigned)(h >> 32), s);
  const unsigned hl = __funnelshift_l((unsigned)u, (unsigned)h, s);
  const unsigned lh = __funnelshift_l((unsigned)p0, (unsigned)u, s);
  const unsigned w = ((unsigned)p0 << s) | (hl & 1u);
  unsigned rh, rl;
  asm("{\n\t.reg .u32 c;\n\t"
      "add.cc.u32 c, %2, 0xffffffff;\n\t"    // carry: bits below lh, or (a tie goes to even) an odd result
      "addc.cc.u32 c, %3, 0x7fffffff;\n\t"   // carry: more than half, or half with the above
      "addc.cc.u32 %0, %4, 0;\n\t"
      "addc.u32 %1, %5, %6;\n\t}"
      : "=r"(rl), "=r"(rh)
      : "r"(w), "r"(lh), "r"(hl), "r"(hh), "r"(e));
  return from_words((int)rh, (int)rl);
#else
  const unsigned long long lo = u << 32 | (unsigned)p0;
  const unsigned long long hn = s ? h << 1 | lo >> 63 : h, ln = lo << s;
  const unsigned long long up = ln > 0x8000000000000000ull || (ln == 0x8000000000000000ull && (hn & 1)) ? 1 : 0;
  const unsigned long long r = hn + up + ((unsigned long long)e << 32);
  return from_words((int)(r >> 32), (int)(unsigned)r);
#endif
}
// |x| in [2^-511, 2^512): the product of two such values is normal
A2C_HD bool mul_int_ok(double x) {
  return (unsigned)((hi_word(x) & 0x7ff00000) - 0x20000000) < 0x3ff00000u;
}

// Adding 1.5 2^52 rounds |v| < 2^31 to an integer (ties to even), held in
// the sum's low word.
constexpr double kRoundShift = 6755399441055744.0;

// The same values for |x| < 708 with integer operations where the FP64
// pipe is not needed: rounding by an addition, the integer from the sum's
// low word, the power of two added to the exponent (the result is normal).
// 13 FP64 operations.
A2C_HD double fexp_mid(double x) {
  const double t = x * 92.33248261689366 + kRoundShift;  // x * 64/ln2
  const double n = t - kRoundShift;
  const int ni = lo_word(t);
  double r = fma(-n, 0.010830424696249145, x);
  r = fma(-n, 3.623510646634843e-19, r);
  double p = fma(r, 0.001388888888888889, 0.008333333333333333);
  p = fma(r, p, 0.041666666666666664);
  p = fma(r, p, 0.16666666666666666);
  p = fma(r, p, 0.5);
  p = fma(r * r, p, r);
#if defined(__CUDA_ARCH__)
  const double2 e = *reinterpret_cast<const double2 *>(kExp2TabDev[ni & 63]);
  const double th = e.x, tl = e.y;
#else
  const double th = kExp2TabHost[ni & 63][0], tl = kExp2TabHost[ni & 63][1];
#endif
  const double v = th + fma(th, p, tl);
  return from_words(hi_word(v) + (int)((unsigned)(ni >> 6) << 20), lo_word(v));
}

// The same values again with three FP64 operations, for 2^-8 <= |x| < 708
// (else fexp_mid): n and the reduced argument in integers, and the four
// inner steps of the polynomial, whose results keep to one binade each, as
// fixed-point sums rounded like the FMAs they stand for.  About 210 integer
// instructions for ten FP64 ones: the kernels of the plain form are bound by
// the FP64 pipe (see mul_int).
//
// r = |x| - n ln2/64: the head of ln2/64 is a multiple of 2^-59 and |x| of
// 2^-60, so r before the tail is an exact 64-bit integer in 2^-60; less n
// times the tail, in 2^-114, rounded to 53 bits.  |r| >= 2^-20 is asked for
// (one in 6,000 arguments is nearer a multiple of ln2/64).
#if defined(__CUDACC__)
#define A2C_CALL static __host__ __device__ __noinline__
#else
#define A2C_CALL inline
#endif
struct FixedStep {  // c + r * f, rounded: c and the result in units of 2^u
  // f = fl 2^(ef-63) with fl left-justified; ml: |r| left-justified, with d
  // the shift that brings the product's head into units of 2^u
  static A2C_HD unsigned long long go(unsigned long long c, unsigned long long fl, unsigned long long ml, int d,
                                      bool neg) {
    const unsigned __int128 p = (unsigned __int128)ml * fl;
    const unsigned long long t = (unsigned long long)(p >> 64);
    unsigned long long q = t >> d, f = (t << (64 - d)) | ((unsigned long long)p != 0 ? 1ull : 0ull);
    if (neg) {  // minus (q.f)
      f = 0ull - f;
      q = c - q - (f != 0 ? 1ull : 0ull);
    } else {
      q = c + q;
    }
    return q + (f > 0x8000000000000000ull || (f == 0x8000000000000000ull && (q & 1)) ? 1ull : 0ull);
  }
};
A2C_CALL double fexp_fixed(double x) {
  const unsigned hx = (unsigned)hi_word(x), ah = hx & 0x7fffffffu, lx = (unsigned)lo_word(x);
  if (ah - 0x3f700000u >= 0x40862000u - 0x3f700000u) return fexp_mid(x);
  const bool sx = hx >> 31;
  // n = rint(|x| * 64/ln2)
  const double p = mul_int(from_words((int)ah, (int)lx), 92.33248261689366);
  const unsigned hp = (unsigned)hi_word(p), lp = (unsigned)lo_word(p);
  const unsigned s = 1043u - (hp >> 20);  // 4 to 22: the unit's place in the high word
  const unsigned mp = (hp & 0xfffffu) | 0x100000u;
  const unsigned fr = mp << (32u - s);
  unsigned n = mp >> s;
  n += fr > 0x80000000u || (fr == 0x80000000u && (lp != 0 || (n & 1u))) ? 1u : 0u;
  // r in 2^-60, then in 2^-114
  const unsigned long long m = ((unsigned long long)((ah & 0xfffffu) | 0x100000u) << 32) | lx;
  const long long r0 = (long long)((m << ((ah >> 20) - 1015u)) - (unsigned long long)n * 12486629536330718ull);
  const __int128 v = ((__int128)r0 << 54) - (__int128)((unsigned __int128)n * 7525737178955839ull);
  const bool neg = v < 0;
  const unsigned __int128 w = neg ? -(unsigned __int128)v : (unsigned __int128)v;
  const unsigned long long wh = (unsigned long long)(w >> 64);
  if (wh < (1ull << 30)) return fexp_mid(x);
#if defined(__CUDA_ARCH__)
  const int lz = __clzll((long long)wh);
#else
  const int lz = __builtin_clzll(wh);
#endif
  const unsigned __int128 nv = w << lz;
  const unsigned long long nh = (unsigned long long)(nv >> 64) | ((unsigned long long)nv != 0 ? 1ull : 0ull);
  const unsigned long long mr = (nh + 0x3ff + ((nh >> 11) & 1)) >> 11;  // |r| = mr 2^(-39 - lz)
  if (mr == 0) return fexp_mid(x);                                      // rounded up to a power of two and wrapped
  const unsigned long long ml = mr << 11;
  const bool sr = neg != sx;
  // 1/120 + r/720, 1/24 + r (.), 1/6 + r (.), 1/2 + r (.)
  unsigned long long c = FixedStep::go(4803839602528529ull, 6405119470038039ull << 11, ml, lz, sr);
  c = FixedStep::go(6004799503160661ull, c << 11, ml, lz - 1, sr);
  c = FixedStep::go(6004799503160661ull, c << 11, ml, lz - 1, sr);
  c = FixedStep::go(sr ? 1ull << 53 : 1ull << 52, c << 11, ml, sr ? lz - 2 : lz - 1, sr);
  const unsigned long long hb = c + ((sr ? 1020ull : 1021ull) << 52);
  const double half = from_words((int)(hb >> 32), (int)(unsigned)hb);
  const unsigned long long rb = mr + ((unsigned long long)(1035 - lz) << 52);
  const double r = from_words((int)((unsigned)(rb >> 32) | (sr ? 0x80000000u : 0u)), (int)(unsigned)rb);
  const double q = fma(mul_int(r, r), half, r);
  const int ns = sx ? -(int)n : (int)n, j = ns & 63;
#if defined(__CUDA_ARCH__)
  const double2 e = *reinterpret_cast<const double2 *>(kExp2TabDev[j]);
  const double th = e.x, tl = e.y;
#else
  const double th = kExp2TabHost[j][0], tl = kExp2TabHost[j][1];
#endif
  const double y = th + fma(th, q, tl);
  return from_words(hi_word(y) + (int)((unsigned)(ns >> 6) << 20), lo_word(y));
}

// Results below 2^-1021 are flushed to zero (no argument of the potential
// comes near), above 709.78 overflow to +inf; NaN propagates.
A2C_HD double fexp(double x) {
#if defined(__CUDA_ARCH__)
  if ((hi_word(x) & 0x7fffffff) < 0x40862000) return fexp_fixed(x);  // |x| < 708
#endif
  if (!(x > -708.0)) return (x != x) ? x : 0.0;
  if (x > 709.78) return HUGE_VAL;
  const double n = rint(x * 92.33248261689366);  // x * 64/ln2
  const int ni = (int)n;
  const int j = ni & 63;
  const int k = (ni - j) / 64;
  double r = fma(-n, 0.010830424696249145, x);    // ln2/64, hi
  r = fma(-n, 3.623510646634843e-19, r);           // ln2/64, lo
  double p = fma(r, 0.001388888888888889, 0.008333333333333333);
  p = fma(r, p, 0.041666666666666664);
  p = fma(r, p, 0.16666666666666666);
  p = fma(r, p, 0.5);
  p = fma(r * r, p, r);
#if defined(__CUDA_ARCH__)
  const double th = kExp2TabDev[j][0], tl = kExp2TabDev[j][1];
#else
  const double th = kExp2TabHost[j][0], tl = kExp2TabHost[j][1];
#endif
  return ldexp(th + fma(th, p, tl), k);
}

// fexp's values by fexp_mid wherever that serves
A2C_HD double fexp_soon(double x) {
  return (hi_word(x) & 0x7fffffff) < 0x40862000 ? fexp_mid(x) : fexp(x);
}

// e^(a.hi + a.lo) = 2^k (v.hi + v.lo) with relative error below 2^-70, for
// |a.hi| < 700 and a.lo below an ulp of a.hi.  a = (64 k + j) ln2/64 + r: n times
// the 36-bit head of ln2/64 is exact, the tail product carried in two
// doubles; e^r - 1 = r + r^2/2 + (degree 7 from r^3/6 on, below 2^-25, in
// double); times 2^(j/64) as hi + lo.
A2C_HD D2 quick_exp(D2 a, int &k) {
  const double t = a.hi * 92.33248261689366 + kRoundShift;  // 64/ln2
  const double n = t - kRoundShift;
  const int ni = lo_word(t), j = ni & 63;
  k = (ni - j) / 64;
  const double r1 = fma(-n, 0.010830424696223417, a.hi);  // exact
  const double p = rounded_product(n, 2.572804622327669e-14), pe = fma(n, 2.572804622327669e-14, -p);
  D2 r = two_sum(r1, -p);
  r = two_sum(r.hi, r.lo - pe + a.lo);
  const double v = rounded_product(r.hi, r.hi), ve = fma(r.hi, r.hi, -v);
  double c = fma(r.hi, 1.984126984126984e-04, 1.388888888888889e-03);
  c = fma(r.hi, c, 8.333333333333333e-03);
  c = fma(r.hi, c, 4.1666666666666664e-02);
  c = fma(r.hi, c, 1.6666666666666666e-01);
  c = (r.hi * v) * c;
  const D2 s = quick_two_sum(r.hi, 0.5 * v);
  const double e2 = s.lo + (c + (0.5 * ve + fma(r.hi, r.lo, r.lo)));
#if defined(__CUDA_ARCH__)
  const double th = kExp2TabDev[j][0], tl = kExp2TabDev[j][1];
#else
  const double th = kExp2TabHost[j][0], tl = kExp2TabHost[j][1];
#endif
  const D2 q = two_prod(th, s.hi);
  const D2 h = quick_two_sum(th, q.hi);
  return quick_two_sum(h.hi, h.lo + (q.lo + fma(th, e2, fma(tl, s.hi, tl))));
}

// -log of the 9-bit c below for the 128 intervals of m in [0.707, 1.414):
// c ~ 1/m, hi a multiple of 2^-42, lo the rest.
#define A2C_LOG_TABLE \
    {1.41015625, -0.34370051385326406, -5.438888329899065e-14}, \
    {1.40234375, -0.3381449440087181, 1.686950122813039e-15}, \
    {1.39453125, -0.3325583373000427, -3.390686133672229e-14}, \
    {1.38671875, -0.32694034499581903, -3.428840012666946e-14}, \
    {1.37890625, -0.3212906124538222, 8.788542769971545e-14}, \
    {1.37109375, -0.3156087789864159, 1.1259274624680829e-13}, \
    {1.36328125, -0.30989447772276435, -1.0033796982039214e-13}, \
    {1.359375, -0.30702503529482783, -8.403156304792425e-14}, \
    {1.3515625, -0.3012613305781997, 3.7923164802093147e-14}, \
    {1.34375, -0.2954642128938758, 3.993416384387844e-14}, \
    {1.3359375, -0.28963329258294834, -9.43339818951269e-14}, \
    {1.328125, -0.28376817313073843, 9.3834172236637e-14}, \
    {1.32421875, -0.2808226629008459, -4.188609137863701e-14}, \
    {1.31640625, -0.27490548587275043, -4.8816703646769986e-14}, \
    {1.30859375, -0.26895308734560786, 1.0389630784002988e-13}, \
    {1.30078125, -0.2629650455007777, -1.0364636459896663e-13}, \
    {1.296875, -0.25995752443691345, -1.2621729398885316e-14}, \
    {1.2890625, -0.25391520998095984, -3.600176732637335e-15}, \
    {1.28125, -0.2478361639045943, 1.3029797173308663e-14}, \
    {1.27734375, -0.24478272641772492, 3.399981108361833e-14}, \
    {1.26953125, -0.23864773785021498, 3.997050909530134e-14}, \
    {1.265625, -0.23556607131286, 9.30945949519689e-14}, \
    {1.2578125, -0.22937410106487732, 3.149265065191484e-14}, \
    {1.25, -0.22314355131425145, 4.169796584527195e-14}, \
    {1.24609375, -0.2200136583053336, 5.149667234141408e-14}, \
    {1.23828125, -0.21372432939779173, 7.359580186440514e-14}, \
    {1.234375, -0.21056476910735, 3.6507188831790577e-16}, \
    {1.2265625, -0.2042155414287663, 7.540916511956189e-14}, \
    {1.22265625, -0.20102574606062262, 3.188184937543774e-14}, \
    {1.21484375, -0.1946154676995775, -9.41653814571825e-14}, \
    {1.2109375, -0.19139485299956505, -6.440856150696892e-14}, \
    {1.203125, -0.18492233849406148, 4.9485167661250996e-14}, \
    {1.19921875, -0.18167030310769405, 5.937506333384701e-14}, \
    {1.1953125, -0.17840765747291698, 9.86835038673495e-14}, \
    {1.1875, -0.17185025692674571, 8.649239607212071e-14}, \
    {1.18359375, -0.16855536102980295, -3.714397754170472e-15}, \
    {1.17578125, -0.16193282026938505, 7.179390019295677e-14}, \
    {1.171875, -0.15860503017665906, 2.0472357800461955e-14}, \
    {1.16796875, -0.15526612891108016, -4.3792508292406054e-14}, \
    {1.16015625, -0.1485546943231384, 1.24915489807516e-15}, \
    {1.15625, -0.14518200984457508, 7.718001336828099e-14}, \
    {1.15234375, -0.14179791186029433, 3.698459506697097e-14}, \
    {1.14453125, -0.13499516453748583, -1.8996158041578768e-14}, \
    {1.140625, -0.13157635778861732, -1.0195735223708473e-13}, \
    {1.13671875, -0.12814582269197672, 4.668031403945796e-14}, \
    {1.12890625, -0.12124924363297396, 1.0427241278273008e-13}, \
    {1.125, -0.11778303565643, 4.654729747598445e-14}, \
    {1.12109375, -0.11430477128010352, 4.488953352238699e-14}, \
    {1.1171875, -0.11081436634026431, -2.5799991283069902e-14}, \
    {1.109375, -0.10379679368156758, -7.598636597194141e-14}, \
    {1.10546875, -0.10026945316371894, 4.378637617078398e-14}, \
    {1.1015625, -0.09672962645845473, -9.638067658552277e-14}, \
    {1.09765625, -0.0931772248541165, -6.678708517162898e-14}, \
    {1.08984375, -0.0860343373417436, -5.955922987625643e-14}, \
    {1.0859375, -0.08244366921098845, -8.614512936087814e-14}, \
    {1.08203125, -0.07884006170775137, -2.465018906176612e-14}, \
    {1.078125, -0.07522342123752424, -6.329065958724544e-14}, \
    {1.07421875, -0.07159365318693744, -7.137308225343178e-14}, \
    {1.0703125, -0.06795066190852594, 1.8195060030168815e-14}, \
    {1.0625, -0.06062462181648698, 5.213620639136504e-14}, \
    {1.05859375, -0.056941376400118315, -2.0109399435564958e-14}, \
    {1.0546875, -0.053244514518837605, 2.532168943117445e-14}, \
    {1.05078125, -0.04953393512232651, 4.9880309107981426e-14}, \
    {1.046875, -0.0458095360313564, 6.219834199475792e-14}, \
    {1.04296875, -0.04207121392073532, 4.826314000551128e-14}, \
    {1.0390625, -0.03831886430202758, -1.0902154302203302e-13}, \
    {1.03515625, -0.034552381506728125, 6.839139742328777e-14}, \
    {1.03125, -0.03077165866670839, -4.529814257790929e-14}, \
    {1.02734375, -0.026976587698300136, 9.806050516843177e-14}, \
    {1.0234375, -0.023167059281604452, 7.007359704310036e-14}, \
    {1.01953125, -0.019342962843211353, 8.041853850522586e-14}, \
    {1.015625, -0.015504186535963527, -1.7274567499706107e-15}, \
    {1.01171875, -0.011650617220084314, 1.0903974971735932e-13}, \
    {1.00390625, -0.0038986404156275967, -2.972634690092895e-14}, \
    {1.0, 0.0, 0.0}, \
    {1.0, 0.0, 0.0}, \
    {0.98828125, 0.011787955751970003, 7.223757580209288e-14}, \
    {0.98046875, 0.019724505347767263, 1.1326399700142234e-14}, \
    {0.97265625, 0.027724548014930406, -7.554530328896727e-14}, \
    {0.966796875, 0.03376686247088401, -6.652375062271929e-14}, \
    {0.958984375, 0.041880497245074366, -8.71601984429868e-14}, \
    {0.951171875, 0.05006050195697753, -5.953822004049194e-14}, \
    {0.9453125, 0.05623971832278585, 9.023009281142904e-14}, \
    {0.9375, 0.0645385211375924, -2.1225608044809997e-14}, \
    {0.931640625, 0.07080813415109333, 7.324072905400027e-14}, \
    {0.923828125, 0.07922923654746228, 1.1253882534313481e-13}, \
    {0.91796875, 0.0855919303353403, 6.322009333691484e-14}, \
    {0.91015625, 0.0941389909139616, -9.969653023079706e-14}, \
    {0.904296875, 0.10059757095336863, -9.49206327250953e-14}, \
    {0.8984375, 0.10709813555627079, 9.631011033519217e-14}, \
    {0.892578125, 0.1136412341452342, 6.889214192008475e-14}, \
    {0.884765625, 0.12243249955645297, 2.0797337102277177e-14}, \
    {0.87890625, 0.1290770422751848, -4.2451216089619995e-14}, \
    {0.873046875, 0.1357660304258843, 5.4642560554597724e-14}, \
    {0.8671875, 0.14250006260726877, 1.4256439478199035e-14}, \
    {0.861328125, 0.14927974959255152, 1.1026677017414112e-13}, \
    {0.85546875, 0.15610571466299916, 6.249274931606537e-14}, \
    {0.849609375, 0.16297859395081105, 1.2645632984431417e-14}, \
    {0.845703125, 0.16758689703692653, 9.140819889491412e-14}, \
    {0.83984375, 0.17453941635199044, -9.076231556699796e-14}, \
    {0.833984375, 0.18154061181098768, -1.0445339530284443e-13}, \
    {0.828125, 0.18859116980752333, 2.6693431578015818e-14}, \
    {0.822265625, 0.19569179135714876, -2.239166785505485e-14}, \
    {0.818359375, 0.20045370511729743, 7.262215167738776e-14}, \
    {0.8125, 0.20763936477828793, -4.3425422595242564e-14}, \
    {0.806640625, 0.21487703207844788, 2.714636557077735e-14}, \
    {0.802734375, 0.2197314105433179, -4.472851385991314e-14}, \
    {0.796875, 0.22705745063535687, -1.078736749871691e-14}, \
    {0.79296875, 0.2319714654377094, 6.573097737831975e-14}, \
    {0.787109375, 0.23938806309274696, 7.784172549574863e-14}, \
    {0.783203125, 0.24436319773303694, -9.834201296269778e-14}, \
    {0.77734375, 0.25187261975497677, 9.331234677945918e-14}, \
    {0.7734375, 0.25691041378513546, -1.0822171646799124e-13}, \
    {0.76953125, 0.26197371574153294, 4.102651071698446e-14}, \
    {0.763671875, 0.26961706505403527, 1.0674835088128526e-13}, \
    {0.759765625, 0.27474528142101917, 4.2320076202145394e-14}, \
    {0.755859375, 0.2798999320098119, -8.591298393628546e-14}, \
    {0.75, 0.28768207245184385, -6.292357389008195e-14}, \
    {0.74609375, 0.29290401643288533, 4.727452940514406e-14}, \
    {0.7421875, 0.29815337231912054, -4.4204083338755686e-14}, \
    {0.73828125, 0.3034304294199046, 1.548345993498083e-14}, \
    {0.734375, 0.30873548164959175, 2.1522127491642888e-14}, \
    {0.728515625, 0.3167462053957024, -1.0174753377507561e-14}, \
    {0.724609375, 0.3221225624320141, 5.855316792709415e-14}, \
    {0.720703125, 0.3275279809990934, -1.1281735060685524e-13}, \
    {0.716796875, 0.33296277698491394, 2.3569101751290204e-14}, \
    {0.712890625, 0.33842727145702156, -5.280156204729064e-15}, \
    {0.708984375, 0.3439217907746297, 2.730651892134709e-14}
#if defined(__CUDACC__)
__device__ const double kLogTabDev[128][3] = {A2C_LOG_TABLE};
#endif
static const double kLogTabHost[128][3] = {A2C_LOG_TABLE};
#undef A2C_LOG_TABLE

// log(u) for 1e-300 <= u < 1e300; this value and log_dd's are within `err`
// of each other (2^-71; near 1, where the reduction leaves u unchanged,
// 2^-66 of the value and 2^-90).
// u = 2^e m, z = c m - 1 with |z| < 2^-6.9 exact in two doubles, log u =
// e ln2 - log c + log1p(z); terms from z^3/3 on (below 2^-22) in double.
A2C_HD D2 quick_log(double u, double &err) {
  const int hu = hi_word(u), t = hu - 0x3fe6a09e;
  const int e = t >> 20, i = (t >> 13) & 127;
  const double m = from_words(hu - (e << 20), lo_word(u));
#if defined(__CUDA_ARCH__)
  const double c = kLogTabDev[i][0], lh = kLogTabDev[i][1], ll = kLogTabDev[i][2];
  const double de = __hiloint2double(0x43300000, 0x80000000 ^ e) - 4503601774854144.0;  // e, by its bits
#else
  const double c = kLogTabHost[i][0], lh = kLogTabHost[i][1], ll = kLogTabHost[i][2];
  const double de = (double)e;
#endif
  const D2 p = two_prod(m, c);
  const double z = p.hi - 1.0, zl = p.lo;
  const double v = rounded_product(z, z), ve = fma(z, z, -v);
  double q = fma(z, 9.090909090909091e-02, -0.1);
  q = fma(z, q, 1.1111111111111111e-01);
  q = fma(z, q, -0.125);
  q = fma(z, q, 1.4285714285714285e-01);
  q = fma(z, q, -1.6666666666666666e-01);
  q = fma(z, q, 0.2);
  q = fma(z, q, -0.25);
  q = fma(z, q, 3.333333333333333e-01);
  q = (z * v) * q;
  const D2 s = quick_two_sum(z, -0.5 * v);
  const double s2 = s.lo + (q + fma(-0.5, ve, zl * (1.0 - z + v)));
  const double a = fma(de, 0.6931471805598903, lh);  // exact: both multiples of 2^-42
  const D2 b = two_sum(a, s.hi);
  const double l = b.lo + (s2 + fma(de, 5.497923018708371e-14, ll));
  const D2 r = quick_two_sum(b.hi, l);
  // 2^-66 of it and 2^-90 (the series' absolute error), or 2^-71
  err = a == 0.0 ? fma(fabs(r.hi), 1.3552527156068805e-20, 8.077935669463161e-28) : 4.235164736271502e-22;
  return r;
}

// Ziv's test: true when every value within err of v rounds to `out`.
A2C_HD bool rounds_to(D2 v, double err, double &out) {
  out = v.hi + (v.lo + err);
  return out == v.hi + (v.lo - err);
}
// out times 2^k for a result whose scaled value is a normal double
A2C_HD double scale_normal(double out, int k) { return from_words(hi_word(out) + (k << 20), lo_word(out)); }

// The quick forms: false when the rounding test leaves the result open.
A2C_HD bool quick_cr_exp(double x, double &out) {
  int k;
  const D2 v = quick_exp({x, 0.0}, k);
  const bool ok = rounds_to(v, v.hi * 8.470329472543003e-22, out);  // 2^-70
  out = scale_normal(out, k);
  return ok;
}
// e^x and e^-x, |x| < 700, each with its own test (bits 0 and 1 of the
// result): quick_exp's steps with the reduction shared and the degree-7 tail
// split into its even and odd part, whose rounding stays some 2^-78 of 1.
A2C_HD int quick_cr_exp_both(double x, double &up, double &down) {
  const double t = x * 92.33248261689366 + kRoundShift;
  const double n = t - kRoundShift;
  const int ni = lo_word(t);
  const double r1 = fma(-n, 0.010830424696223417, x);
  const double p = rounded_product(n, 2.572804622327669e-14), pe = fma(n, 2.572804622327669e-14, -p);
  D2 r = two_sum(r1, -p);
  r = quick_two_sum(r.hi, r.lo - pe);
  const double v = rounded_product(r.hi, r.hi), ve = fma(r.hi, r.hi, -v), vh = 0.5 * v;
  const double odd = fma(v, fma(v, 1.984126984126984e-04, 8.333333333333333e-03), 1.6666666666666666e-01);
  const double even = fma(v, 1.388888888888889e-03, 4.1666666666666664e-02);
  const double w = fma(r.hi, r.lo, 0.5 * ve);
  int ok = 0;
  for (int side = 0; side < 2; ++side) {
    const double rh = side ? -r.hi : r.hi, rl = side ? -r.lo : r.lo;
    const int m = side ? -ni : ni, j = m & 63;
    const double c = (rh * v) * fma(rh, even, odd);
    const D2 s = quick_two_sum(rh, vh);
    const double e2 = s.lo + (c + (w + rl));
#if defined(__CUDA_ARCH__)
    const double th = kExp2TabDev[j][0], tl = kExp2TabDev[j][1];
#else
    const double th = kExp2TabHost[j][0], tl = kExp2TabHost[j][1];
#endif
    const D2 q = two_prod(th, s.hi);
    const D2 h = quick_two_sum(th, q.hi);
    const D2 f = quick_two_sum(h.hi, h.lo + (q.lo + fma(th, e2, fma(tl, s.hi, tl))));
    double &out = side ? down : up;
    if (rounds_to(f, f.hi * 8.470329472543003e-22, out)) ok |= 1 << side;  // 2^-70
    out = scale_normal(out, (m - j) / 64);
  }
  return ok;
}
A2C_HD bool quick_cr_log(double u, double &out) {
  double err;
  const D2 v = quick_log(u, err);
  return rounds_to(v, err, out);
}
// y log(u) is off by |y| times the log's error and 2^-104 of itself, which
// is the relative error it adds to the power.
A2C_HD bool quick_cr_pow(double u, double y, double &out) {
  double err;
  const D2 l = mul_d(quick_log(u, err), y);
  if (!(l.hi > -700.0 && l.hi < 700.0)) return false;
  int k;
  const D2 v = quick_exp(l, k);
  const bool ok = rounds_to(v, v.hi * (8.470329472543003e-22 + 1.0625 * fabs(y) * err), out);
  out = scale_normal(out, k);
  return ok;
}

// The series alone, out of line on the device: the quick forms' rare rest.
#if defined(__CUDACC__)
#define A2C_REST static __host__ __device__ __noinline__
#else
#define A2C_REST inline
#endif
A2C_REST double series_exp(double x) { return round_dd(exp_dd({x, 0.0})); }
A2C_REST double series_log(double u) { return round_dd(log_dd(u)); }
A2C_REST double series_pow(double u, double y) {
  const D2 l = mul_d(log_dd(u), y);
  if (!(l.hi > -700.0 && l.hi < 700.0)) return pow(u, y);
  return round_dd(exp_dd(l));
}

// Correctly rounded except in rare near-midpoint cases.
A2C_HD double cr_exp(double x) {
  if (!(x > -700.0 && x < 700.0)) return exp(x);
#if defined(__CUDA_ARCH__)
  double q;
  if (quick_cr_exp(x, q)) return q;
#endif
  return series_exp(x);
}
// cr_exp(x) and cr_exp(-x)
A2C_HD void cr_exp_both(double x, double &up, double &down) {
#if defined(__CUDA_ARCH__)
  if (x > -700.0 && x < 700.0) {
    const int ok = quick_cr_exp_both(x, up, down);
    if (!(ok & 1)) up = series_exp(x);
    if (!(ok & 2)) down = series_exp(-x);
    return;
  }
#endif
  up = cr_exp(x);
  down = cr_exp(-x);
}
A2C_HD double cr_log(double u) {
  if (!(u > 0.0) || !(u < 1.0e300) || u < 1.0e-300) return log(u);
#if defined(__CUDA_ARCH__)
  double q;
  if (quick_cr_log(u, q)) return q;
#endif
  return series_log(u);
}
A2C_HD double cr_pow(double u, double y) {
  if (!(u > 0.0) || !(u < 1.0e300) || u < 1.0e-300 || !(fabs(y) < 1.0e6)) return pow(u, y);
#if defined(__CUDA_ARCH__)
  double q;
  if (quick_cr_pow(u, y, q)) return q;
#endif
  return series_pow(u, y);
}
#undef A2C_REST

#undef A2C_HD

}  // namespace dd
}  // namespace a2c
