// FP64 plain-form kernels: pass 1 (site electron density), pass 2 (energy
// and gradient gather) and the occupancy gradient.  Compiled with
// -fmad=false.  Every per-site sum is formed term by term in the
// reference's order (electrondensity.cpp:20-49, minimizer.cpp:162-351,
// 658-789); the only difference from the CPU arithmetic is the device
// exp/pow/log.
//
// Pass 1 and pass 2 evaluate a warp's quadrature points side by side and
// then add their terms in order: S sites share a warp, a round takes the
// next neighbors of each (32 pairs in pass 1, 8 in pass 2), the lanes
// evaluate the round's points -- 12 per pair, whatever site they belong to
// -- into shared memory, and the lanes that own a site's sums (one in pass
// 1; x, y, z and sigma + V in pass 2) add them.  Why: the FP64 pipe (two
// lanes per SM and clock) bounds these kernels, a warp's instruction holds
// it for 32 lanes whether they work or not, and one thread per site left
// a 512-site system 16 warps, each with 960 points in a row.  S trades the
// two ends (rho_sites_per_warp, grad_sites_per_warp).  With the pair
// functions' fewer operations (eam64_pair.cuh) an evaluation takes, one
// thread per site -> now: 15.3 -> 0.70 ms at 512 sites, 23.0 -> 5.5 ms at
// 10,296, 210.6 -> 108.5 ms at 262,144.  Five blocks of pass 2 per SM in place of
// four: an evaluation of 10,296 sites 5.67 -> 5.38 ms, of 262,144 110.5 -> 108.5.
//
// Geometry: for quadrature point k = 2m (+sqrt(3)) or 2m+1 (-sqrt(3)) only
// coordinate m of R^6 is non-zero, so r_k differs from the pair's base
// vector q_i - q_j in one component.  The reference forms
// r = ((q_i + u_i*xi0) - q_j) - u_j*xi1 with u = sqrt(2)*sigma; adding or
// subtracting an exact zero leaves a value unchanged, so the component-wise
// forms used below are bit-identical to it.
#include <algorithm>
#include <mutex>
#include <vector>

#include "eam64_pair.cuh"

#include "internal.cuh"

namespace a2c {
namespace {

constexpr int kBlock = 128;

struct PairGeo {
  double D[3];      // q_i - q_j (image applied)
  double Pi[3][2];  // (q_i[m] + u_i) - q_j[m], (q_i[m] - u_i) - q_j[m]
  double Pj[3][2];  // D[c] - u_j, D[c] + u_j
  double D2[3];     // D[c]^2
};

__device__ __forceinline__ void image_pos(const SiteArgs &a, const double *box, uint32_t e, double q[3]) {
  const int64_t j = e & kIdMask;
  q[0] = a.X[4 * j];
  q[1] = a.X[4 * j + 1];
  q[2] = a.X[4 * j + 2];
  const uint32_t c = e >> kIdBits;
  if (c != kNoShift) {
    const int m0 = (int)(c % 3u) - 1, m1 = (int)((c / 3u) % 3u) - 1, m2 = (int)(c / 9u) - 1;
    if (m0) q[0] = q[0] + m0 * box[0];
    if (m1) q[1] = q[1] + m1 * box[1];
    if (m2) q[2] = q[2] + m2 * box[2];
  }
}

__device__ __forceinline__ void make_geo(const double qi[3], double ui, const double qj[3], double uj, PairGeo &g) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    g.D[c] = qi[c] - qj[c];
    g.Pi[c][0] = (qi[c] + ui) - qj[c];
    g.Pi[c][1] = (qi[c] + (-ui)) - qj[c];
    g.Pj[c][0] = g.D[c] - uj;
    g.Pj[c][1] = g.D[c] - (-uj);
    g.D2[c] = g.D[c] * g.D[c];
  }
}

// r_k and |r_k| for quadrature point k (quadrature.cpp:111-132 ordering).
__device__ __forceinline__ double point(const PairGeo &g, int k, double r[3], int &comp, double &xi0) {
  const int m = k >> 1, sgn = k & 1;
  r[0] = g.D[0];
  r[1] = g.D[1];
  r[2] = g.D[2];
  double s2;
  if (m < 3) {
    comp = m;
    r[m] = g.Pi[m][sgn];
    xi0 = sgn ? -1.7320508075688772 : 1.7320508075688772;
  } else {
    comp = m - 3;
    r[m - 3] = g.Pj[m - 3][sgn];
    xi0 = 0.0;
  }
  const double a0 = (comp == 0) ? r[0] * r[0] : g.D2[0];
  const double a1 = (comp == 1) ? r[1] * r[1] : g.D2[1];
  const double a2 = (comp == 2) ? r[2] * r[2] : g.D2[2];
  s2 = a0 + a1 + a2;
  return sqrt(s2);
}

constexpr unsigned kAll = 0xffffffffu;
constexpr double kSqrt2 = 1.4142135623730951, kSqrt3 = 1.7320508075688772;

// A neighbor's coordinates (image applied) and displacement sqrt(6) sigma
// in the reference's operation order.
__device__ __forceinline__ double displacement(double sigma) { return (kSqrt2 * sigma) * kSqrt3; }

// a * b by the integer pipes where both are in their range
__device__ __forceinline__ double mul(double a, double b) {
  return dd::mul_int_ok(a) && dd::mul_int_ok(b) ? dd::mul_int(a, b) : a * b;
}

// |r_k| of quadrature point k (quadrature.cpp:111-132 ordering): component m
// of the pair vector replaced by rm.
__device__ __forceinline__ double radius(int m, double rm, double d20, double d21, double d22) {
  const double q = mul(rm, rm);
  return sqrt((m == 0 ? q : d20) + (m == 1 ? q : d21) + (m == 2 ? q : d22));
}

// The site a warp's slot works on and its instance (LIST: batched launch).
struct Site64 {
  int64_t s;
  bool live, iPd;
  const double *box;
  double T;
};
template <bool LIST>
__device__ __forceinline__ Site64 site64(const SiteArgs &a, int64_t k, int64_t n) {
  Site64 r;
  r.live = k < n;
  if (LIST) {
    r.s = r.live ? a.bv.site(k) : 0;
    const InstGeo &g = a.bv.geo_of(r.s);
    r.iPd = r.s - g.start < g.nPd;
    r.box = g.S;
    r.T = g.T;
  } else {
    r.s = r.live ? k : 0;
    r.iPd = r.s < a.nPd;
    r.box = a.box;
    r.T = a.T;
  }
  return r;
}

// A listed pair's inputs, loaded one round ahead of their use.
struct Neighbor64 {
  uint32_t en;
  double q[3], sigma, x, Fp;
};
template <bool FP>
__device__ __forceinline__ Neighbor64 load_neighbor(const SiteArgs &a, int64_t t, bool valid) {
  Neighbor64 v{};
  if (!valid) return v;
  v.en = __ldg(&a.nbr[t]);
  const int64_t j = v.en & kIdMask;
  const double *X = a.X + 4 * j;  // 8-byte loads: the caller's X is aligned to no more
  v.q[0] = __ldg(X);
  v.q[1] = __ldg(X + 1);
  v.q[2] = __ldg(X + 2);
  v.sigma = __ldg(X + 3);
  v.x = __ldg(&a.occ[j]);
  if (FP) v.Fp = __ldg(&a.Fp[j]);
  return v;
}
__device__ __forceinline__ void apply_image(Neighbor64 &v, const double *box) {
  const uint32_t c = v.en >> kIdBits;
  if (c == kNoShift) return;
  const int m0 = (int)(c % 3u) - 1, m1 = (int)((c / 3u) % 3u) - 1, m2 = (int)(c / 9u) - 1;
  if (m0) v.q[0] = v.q[0] + m0 * box[0];
  if (m1) v.q[1] = v.q[1] + m1 * box[1];
  if (m2) v.q[2] = v.q[2] + m2 * box[2];
}

constexpr int kWarps = 4;  // warps per block of both passes

// ---------------------------------------------------------------- pass 1
constexpr int kRhoPairs = 32, kRhoRow = 13;  // 12 terms per pair, padded against bank conflicts
struct RhoShared {
  double qp[32][6];  // per site q + u, q - u of each coordinate
  double qj[3][kRhoPairs], D[3][kRhoPairs], D2[3][kRhoPairs], uj[kRhoPairs], xj[kRhoPairs];
  double term[kRhoPairs * kRhoRow];
};

template <int S, bool LIST>
__global__ void __launch_bounds__(32 * kWarps) k_density64(SiteArgs a) {
  constexpr int NB = kRhoPairs / S;  // pairs of one site per round
  extern __shared__ double2 smem64[];
  RhoShared &sh = reinterpret_cast<RhoShared *>(smem64)[threadIdx.x / 32];
  const int lane = threadIdx.x % 32, slot = lane / NB, sub = lane % NB;
  const int64_t n = LIST ? (int64_t)*a.bv.count : (int64_t)a.nPd + a.nH;
  const double W = a.W;
  const int64_t stride = (int64_t)gridDim.x * kWarps * S;
  for (int64_t first = ((int64_t)blockIdx.x * kWarps + threadIdx.x / 32) * S; first < n; first += stride) {
    const Site64 st = site64<LIST>(a, first + slot, n);
    double qi[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) qi[c] = a.X[4 * st.s + c];
    const double ui = displacement(a.X[4 * st.s + 3]);
    __syncwarp();
    if (sub == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sh.qp[slot][2 * c] = qi[c] + ui;
        sh.qp[slot][2 * c + 1] = qi[c] + (-ui);
      }
    }
    const int64_t b = a.off[st.s], npd = a.npd[st.s], e = a.off[st.s + 1];
    double rho = 0.0;  // in lane s for site slot s (s < S)
    for (int part = 0; part < 2; ++part) {  // the Pd neighbors, then the H neighbors
      const bool jPd = part == 0;
      const int64_t t0 = jPd ? b : b + npd;
      const int cnt = st.live ? (int)(jPd ? npd : e - b - npd) : 0;
      const int rounds = __reduce_max_sync(kAll, (cnt + NB - 1) / NB);
      Neighbor64 v = load_neighbor<false>(a, t0 + sub, sub < cnt);
      for (int r = 0; r < rounds; ++r) {
        const bool valid = r * NB + sub < cnt;
        if (valid) {
          apply_image(v, st.box);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double D = qi[c] - v.q[c];
            sh.qj[c][lane] = v.q[c];
            sh.D[c][lane] = D;
            sh.D2[c][lane] = D * D;
          }
          sh.uj[lane] = displacement(v.sigma);
          sh.xj[lane] = v.x;
        }
        const unsigned vm = __ballot_sync(kAll, valid);
        const int nx = (r + 1) * NB + sub;
        v = load_neighbor<false>(a, t0 + nx, nx < cnt);
        __syncwarp();
#pragma unroll 1
        for (int p = lane; p < kRhoPairs * 12; p += 32) {
          const int q = p / 12, k = p - 12 * q;
          if (!(vm >> q & 1u)) continue;
          const int m = (k < 6 ? k : k - 6) >> 1, sgn = k & 1;
          const double u = sh.uj[q];
          const double rm = k < 6 ? sh.qp[q / NB][2 * m + sgn] - sh.qj[m][q] : sh.D[m][q] - (sgn ? -u : u);
          const double f = eam64::density_point<(S > 2)>(jPd, radius(m, rm, sh.D2[0][q], sh.D2[1][q], sh.D2[2][q]));
          sh.term[q * kRhoRow + k] = (jPd ? f : sh.xj[q] * f) * W;
        }
        __syncwarp();
        if (lane < S) {
#pragma unroll 1
          for (int i = 0; i < NB; ++i) {
            const int q = lane * NB + i;
            if (!(vm >> q & 1u)) break;
            const double *t = sh.term + q * kRhoRow;
#pragma unroll
            for (int k = 0; k < 12; ++k) rho = rho + t[k];
          }
        }
        __syncwarp();
      }
    }
    const Site64 own = site64<LIST>(a, first + lane, n);
    if (lane < S && own.live) {
      a.rho[own.s] = rho;
      a.Fp[own.s] = own.iPd ? eam64::F_Pd_d(rho, a.eps) : eam64::F_H_d(rho, a.eps);
      if (!isfinite(rho)) atomicOr(a.status, kStatusNonfinite);
    }
  }
}

// ---------------------------------------------------------------- pass 2
// Per pair-point the three gradient terms of minimizer.cpp:180-190 (and
// their Pd-H / H-Pd / H-H forms) are, with x_j = 1 for a Pd neighbor:
//   c1 = (((x_j*W)*F'_A(rho_i))*f'_B(s))/s
//   c2 = (((x_j*W)*F'_B(rho_j))*f'_A(s))/s
//   c3 = ((x_j*W)*phi'_AB(s))/s
// and the energy term ((0.5*x_i)*x_j)*W*phi_AB(s); the factors equal to 1
// for Pd sites multiply exactly, so one form serves all four pair types.
// A point's products with its vector's components are staged as 12 rows
// (c1, c2, c3 times x, y, z and, for the points that move site i, the moved
// component times its xi0 = +-sqrt(3)); the sigma rows of the six points
// without a sigma part hold the pair's 12 energy terms, in order, so that
// the lane with sigma also sums V.
constexpr int kGradPairs = 8, kGradPts = 12 * kGradPairs;
constexpr int kGradRow = kGradPts + 3;  // the padding keeps the adding lanes off each other's banks
struct GradShared {
  double qp[kGradPairs][6];
  double qj[3][kGradPairs], D[3][kGradPairs], D2[3][kGradPairs], uj[kGradPairs];
  double A1[kGradPairs], A2[kGradPairs], A3[kGradPairs], AV[kGradPairs];
  double pt[12 * kGradRow];
};

template <int S, bool LIST>
__global__ void __launch_bounds__(32 * kWarps, 5) k_gradient64(SiteArgs a) {
  constexpr int NB = kGradPairs / S;
  extern __shared__ double2 smem64[];
  GradShared &sh = reinterpret_cast<GradShared *>(smem64)[threadIdx.x / 32];
  const int lane = threadIdx.x % 32;
  const int slot = (lane % kGradPairs) / NB, sub = lane % NB;  // pair role: lanes 0-7
  const int own = (lane / 4) % S, comp = lane & 3;              // adding role: lanes 0 to 4 S - 1
  const bool adds = lane < 4 * S;
  const int64_t n = LIST ? (int64_t)*a.bv.count : (int64_t)a.nPd + a.nH;
  const double W = a.W, eps = a.eps;
  const eam64::Divisor h = eam64::divisor(2.0 * eps);
  const int64_t stride = (int64_t)gridDim.x * kWarps * S;
  for (int64_t first = ((int64_t)blockIdx.x * kWarps + threadIdx.x / 32) * S; first < n; first += stride) {
    const Site64 st = site64<LIST>(a, first + slot, n);
    double qi[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) qi[c] = a.X[4 * st.s + c];
    const double ui = displacement(a.X[4 * st.s + 3]);
    const double half_xi = 0.5 * a.occ[st.s], Fpi = a.Fp[st.s];
    __syncwarp();
    if (lane < kGradPairs && sub == 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sh.qp[slot][2 * c] = qi[c] + ui;
        sh.qp[slot][2 * c + 1] = qi[c] + (-ui);
      }
    }
    const unsigned pdmask = __ballot_sync(kAll, st.iPd);  // bit q: pair q's site is Pd
    const int64_t b = a.off[st.s], npd = a.npd[st.s], e = a.off[st.s + 1];
    const Site64 me = site64<LIST>(a, first + own, n);
    double acc = 0.0, V = 0.0;  // the component's sum; V in the sigma lane
    if (adds && comp == 3 && me.live) {
      const double r = a.rho[me.s];
      V = V + (me.iPd ? eam64::F_Pd(r) : a.occ[me.s] * eam64::F_H(r));
    }
    for (int part = 0; part < 2; ++part) {
      const bool jPd = part == 0;
      const int64_t t0 = jPd ? b : b + npd;
      const int cnt = (lane < kGradPairs && st.live) ? (int)(jPd ? npd : e - b - npd) : 0;
      const int rounds = __reduce_max_sync(kAll, (cnt + NB - 1) / NB);
      Neighbor64 v = load_neighbor<true>(a, t0 + sub, sub < cnt);
      for (int r = 0; r < rounds; ++r) {
        const bool valid = r * NB + sub < cnt;
        if (valid) {
          apply_image(v, st.box);
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double D = qi[c] - v.q[c];
            sh.qj[c][lane] = v.q[c];
            sh.D[c][lane] = D;
            sh.D2[c][lane] = D * D;
          }
          sh.uj[lane] = displacement(v.sigma);
          const double xW = v.x * W;
          sh.A1[lane] = xW * Fpi;
          sh.A2[lane] = xW * v.Fp;
          sh.A3[lane] = xW;
          sh.AV[lane] = (half_xi * v.x) * W;
        }
        const unsigned vm = __ballot_sync(kAll, valid);
        const int nx = (r + 1) * NB + sub;
        v = load_neighbor<true>(a, t0 + nx, nx < cnt);
        __syncwarp();
#pragma unroll 1
        for (int p = lane; p < kGradPts; p += 32) {
          const int q = p / 12, k = p - 12 * q;
          if (!(vm >> q & 1u)) continue;
          const int m = (k < 6 ? k : k - 6) >> 1, sgn = k & 1;
          const double u = sh.uj[q];
          const double rm = k < 6 ? sh.qp[q / NB][2 * m + sgn] - sh.qj[m][q] : sh.D[m][q] - (sgn ? -u : u);
          const double s = radius(m, rm, sh.D2[0][q], sh.D2[1][q], sh.D2[2][q]);
          const eam64::PairPoint f = eam64::pair_point<(S > 1)>(pdmask >> q & 1u, jPd, s, eps, h);
          const double av = sh.AV[q], A[3] = {sh.A1[q], sh.A2[q], sh.A3[q]};
          double c[3] = {mul(A[0], f.da), mul(A[1], f.db), mul(A[2], f.dphi)};
          if (eam64::in_pair_range(s)) {
            const eam64::Divisor ds = eam64::divisor(s);
#pragma unroll
            for (int i = 0; i < 3; ++i) c[i] = eam64::divide(c[i], ds);
          } else {
#pragma unroll
            for (int i = 0; i < 3; ++i) c[i] = c[i] / s;
          }
          const double r[3] = {m == 0 ? rm : sh.D[0][q], m == 1 ? rm : sh.D[1][q], m == 2 ? rm : sh.D[2][q]};
          const double xi0 = sgn ? -kSqrt3 : kSqrt3;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            double *o = sh.pt + 4 * i * kGradRow + p;
            const double x = c[i] * r[0], y = c[i] * r[1], z = c[i] * r[2];
            o[0] = x;
            o[kGradRow] = y;
            o[2 * kGradRow] = z;
            if (k < 6) o[3 * kGradRow] = (m == 0 ? x : m == 1 ? y : z) * xi0;
          }
          sh.pt[(4 * (k % 3) + 3) * kGradRow + 12 * q + 6 + k / 3] = mul(av, f.phi);
        }
        __syncwarp();
        if (adds) {
#pragma unroll 1
          for (int i = 0; i < NB; ++i) {
            const int q = own * NB + i;
            if (!(vm >> q & 1u)) break;
            const double *t = sh.pt + comp * kGradRow + 12 * q;
#pragma unroll
            for (int k = 0; k < 6; ++k)
#pragma unroll
              for (int c = 0; c < 3; ++c) acc = acc + t[4 * c * kGradRow + k];
            double w = comp == 3 ? V : acc;  // the sigma lane turns to V
#pragma unroll
            for (int k = 6; k < 12; ++k)
#pragma unroll
              for (int c = 0; c < 3; ++c)
                if (k < 10 || comp < 3) w = w + t[4 * c * kGradRow + k];
            if (comp == 3) V = w;
            else acc = w;
          }
        }
        __syncwarp();
      }
    }
    // minimizer.cpp:220-223 and 282-285
    const double f1 = __shfl_down_sync(kAll, acc, 1, 4), f2 = __shfl_down_sync(kAll, acc, 2, 4);
    if (adds && me.live) {
      const double xi = a.occ[me.s];
      if (comp < 3) {
        const double cq = (1.0 / me.T) * xi;
        a.G[4 * me.s + comp] = acc * cq;
        if (comp == 0 && !isfinite(acc + f1 + f2)) atomicOr(a.status, kStatusNonfinite);
      } else {
        const double sigmai = a.X[4 * me.s + 3];
        const double cs = ((1.0 / me.T) * kSqrt2) * xi, ce = ((3.0 * kB) / sigmai) * xi;
        a.G[4 * me.s + 3] = acc * cs - ce;
        a.Vs[me.s] = V;
        a.Ss[me.s] = dd::cr_log(sigmai) * xi;
        if (!isfinite(V) || !isfinite(acc)) atomicOr(a.status, kStatusNonfinite);
      }
    }
  }
}

// Occupancy gradient, minimizer.cpp:658-789, one thread per H site.  d_send
// receives log(x/(1-x)) + sum_Vx/(kB*T) (or stays 0, as send_H does).
__global__ void __launch_bounds__(kBlock) k_chem64(SiteArgs a, const double coePd0, const double coePd2,
                                                 const double coePd3, const double coeH0, const double coeH1,
                                                 const double coeH2, const double coeH3, const int *full,
                                                 double *send) {
  const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= a.nH) return;
  send[h] = 0.0;
  if (full[h] == 1) return;
  const int64_t s = (int64_t)a.nPd + h;
  const double qi[3] = {a.X[4 * s], a.X[4 * s + 1], a.X[4 * s + 2]};
  const double ui = (1.4142135623730951 * a.X[4 * s + 3]) * 1.7320508075688772;
  const double W = a.W, T = a.T;
  const double *box = a.box;
  const int64_t b = a.off[s], m = b + a.npd[s], e = a.off[s + 1];
  const double nHPd = (double)(m - b);
  double sum = 0.0;
  sum = sum + eam64::F_H(a.rho[s]);
  double tmp = (coeH1 * nHPd) * nHPd;
  for (int64_t t = m; t < e; ++t) {
    const double xj = a.occ[a.nbr[t] & kIdMask];
    tmp = tmp + ((2.0 * coeH2) * nHPd) * xj;
    for (int64_t u = m; u < e; ++u) tmp = tmp + (coeH3 * xj) * a.occ[a.nbr[u] & kIdMask];
  }
  sum = sum + ((0.5 * T) * coeH0) * tmp;
  for (int64_t t = b; t < m; ++t) {  // H-Pd pairs
    const uint32_t en = a.nbr[t];
    const int64_t j = en & kIdMask;
    double qj[3];
    image_pos(a, box, en, qj);
    const double uj = (1.4142135623730951 * a.X[4 * j + 3]) * 1.7320508075688772;
    const double WF = W * a.Fp[j];
    PairGeo g;
    make_geo(qi, ui, qj, uj, g);
#pragma unroll 1
    for (int k = 0; k < 12; ++k) {
      double r[3], xi0;
      int comp;
      const double sk = point(g, k, r, comp, xi0);
      const bool fast = eam64::in_pair_range(sk);
      sum = sum + WF * (fast ? eam64::f_H_pos<true>(sk) : eam64::f_H(sk));
      sum = sum + W * (fast ? eam64::morse_pos<true>(true, sk) : eam64::phi_PdH(sk));
    }
    const int64_t bj = a.off[j], mj = bj + a.npd[j], ej = a.off[j + 1];
    sum = sum + ((T * coePd0) * coePd2) * (double)(mj - bj);
    for (int64_t u = mj; u < ej; ++u) sum = sum + ((T * coePd0) * coePd3) * a.occ[a.nbr[u] & kIdMask];
  }
  for (int64_t t = m; t < e; ++t) {  // H-H pairs
    const uint32_t en = a.nbr[t];
    const int64_t j = en & kIdMask;
    double qj[3];
    image_pos(a, box, en, qj);
    const double uj = (1.4142135623730951 * a.X[4 * j + 3]) * 1.7320508075688772;
    const double xj = a.occ[j];
    const double xWF = (xj * W) * a.Fp[j];
    const double xW = xj * W;
    PairGeo g;
    make_geo(qi, ui, qj, uj, g);
#pragma unroll 1
    for (int k = 0; k < 12; ++k) {
      double r[3], xi0;
      int comp;
      const double sk = point(g, k, r, comp, xi0);
      const bool fast = eam64::in_pair_range(sk);
      sum = sum + xWF * (fast ? eam64::f_H_pos<true>(sk) : eam64::f_H(sk));
      sum = sum + xW * (fast ? eam64::morse_pos<true>(false, sk) : eam64::phi_H(sk));
    }
    const int64_t bj = a.off[j], mj = bj + a.npd[j], ej = a.off[j + 1];
    sum = sum + (((xj * T) * coeH0) * coeH2) * (double)(mj - bj);
    for (int64_t u = mj; u < ej; ++u) sum = sum + (((xj * T) * coeH0) * coeH3) * a.occ[a.nbr[u] & kIdMask];
  }
  const double x0 = a.occ[s];
  if (x0 > 0.0 && x0 < 1.0) send[h] = dd::cr_log(x0 / (1.0 - x0)) + sum / (kB * T);
}

__global__ void k_eam64(int which, const double *in, int64_t n, double eps, double *out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = in[i];
  double r;
  switch (which) {
    case 0: r = eam64::F_Pd(v); break;
    case 1: r = eam64::F_Pd_d(v, eps); break;
    case 2: r = eam64::F_H(v); break;
    case 3: r = eam64::F_H_d(v, eps); break;
    case 4: r = eam64::f_Pd(v); break;
    case 5: r = eam64::f_Pd_d(v, eps); break;
    case 6: r = eam64::f_H(v); break;
    case 7: r = eam64::f_H_d(v, eps); break;
    case 8: r = eam64::phi_Pd(v); break;
    case 9: r = eam64::phi_Pd_d(v, eps); break;
    case 10: r = eam64::phi_PdH(v); break;
    case 11: r = eam64::phi_PdH_d(v, eps); break;
    case 12: r = eam64::phi_H(v); break;
    default: r = eam64::phi_H_d(v, eps); break;
  }
  out[i] = r;
}

SiteArgs site_args(a2c_gpp_ctx *c, const double *dX) {
  SiteArgs a;
  a.nPd = c->p.nPd;
  a.nH = c->p.nH;
  a.T = c->p.T;
  a.W = c->p.QWp;
  a.eps = c->p.eps;
  for (int d = 0; d < 3; ++d) a.box[d] = c->p.box[d];
  a.X = dX;
  a.occ = c->d_occ;
  a.off = c->d_off;
  a.nbr = c->d_nbr;
  a.npd = c->d_npd;
  a.rho = c->d_rho;
  a.Fp = c->d_Fp;
  a.G = c->d_G;
  a.Vs = c->d_Vs;
  a.Ss = c->d_Ss;
  a.status = c->d_status;
  return a;
}

// Sites per warp.  Few sites: a warp per site or two, all lanes on its
// points, though one to eight lanes then do its additions; many: the
// additions of 8 (32 in pass 1) sites fill the lanes.  Measured on a GB300
// (152 SMs), ms for the choices named:
//   pass 1, 2 / 8 / 32 sites: 512 sites 0.18 / 0.54 / 1.9, 5,832 0.65 / 0.71
//     / 1.9, 8,000 0.92 / 0.71 / 1.9, 32,768 3.5 / 2.33 / 2.42, 64,000 6.7 /
//     4.55 / 4.38, 110,592 11.5 / 7.3 / 6.6;
//   pass 2, 1 / 2 / 4 / 8 sites: 512 sites 0.51 / 0.98 / 1.7 / 3.3, 1,728
//     1.13 / 1.28 / 1.7 / 3.3, 2,744 1.9 / 1.7 / 2.2 / 3.7, 5,832 3.7 / 2.7 /
//     3.0 / 4.3, 8,000 5.5 / 4.1 / 3.8 / 4.5, 13,824 8.5 / 6.9 / 6.9 / 6.0,
//     110,592 67 / 49 / 42 / 40.
// Results do not depend on it.
int rho_sites_per_warp(int64_t n, int sms) { return n < 42 * (int64_t)sms ? 2 : n < 330 * (int64_t)sms ? 8 : 32; }
int grad_sites_per_warp(int64_t n, int sms) {
  return n < 16 * (int64_t)sms ? 1 : n < 46 * (int64_t)sms ? 2 : n < 80 * (int64_t)sms ? 4 : 8;
}

// Blocks resident on the device at once for a kernel with its shared
// memory, asked once per kernel and device under a lock.
int resident_blocks(const void *fn, int smem, int dev) {
  struct Entry {
    const void *fn;
    int dev, blocks;
  };
  static std::mutex m;
  static std::vector<Entry> cache;
  std::lock_guard<std::mutex> lock(m);
  for (const Entry &e : cache)
    if (e.fn == fn && e.dev == dev) return e.blocks;
  int nb = 0;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, 32 * kWarps, smem);
  (void)cudaGetLastError();
  if (nb < 1) return 1;  // not cached: asked again next time
  cache.push_back({fn, dev, nb * device_sms(dev)});
  return cache.back().blocks;
}

template <class Shared>
a2c_status launch_warps(void (*fn)(SiteArgs), int sites, const SiteArgs &a, int64_t n, bool list, a2c_gpp_ctx *c) {
  constexpr int smem = (int)sizeof(Shared) * kWarps;
  const int cap = resident_blocks((const void *)fn, smem, c->device);
  int64_t blocks = (n + (int64_t)sites * kWarps - 1) / ((int64_t)sites * kWarps);
  if (list) blocks = std::min<int64_t>(blocks, cap);  // the list's length is only known on the device
  fn<<<(unsigned)blocks, 32 * kWarps, smem, c->stream>>>(a);
  A2C_CUDA(cudaGetLastError());
  return A2C_OK;
}

template <bool LIST>
a2c_status density64(a2c_gpp_ctx *c, const SiteArgs &a, int64_t n) {
  switch (rho_sites_per_warp(n, device_sms(c->device))) {
    case 2: return launch_warps<RhoShared>(k_density64<2, LIST>, 2, a, n, LIST, c);
    case 8: return launch_warps<RhoShared>(k_density64<8, LIST>, 8, a, n, LIST, c);
    default: return launch_warps<RhoShared>(k_density64<32, LIST>, 32, a, n, LIST, c);
  }
}
template <bool LIST>
a2c_status gradient64(a2c_gpp_ctx *c, const SiteArgs &a, int64_t n) {
  switch (grad_sites_per_warp(n, device_sms(c->device))) {
    case 1: return launch_warps<GradShared>(k_gradient64<1, LIST>, 1, a, n, LIST, c);
    case 2: return launch_warps<GradShared>(k_gradient64<2, LIST>, 2, a, n, LIST, c);
    case 4: return launch_warps<GradShared>(k_gradient64<4, LIST>, 4, a, n, LIST, c);
    default: return launch_warps<GradShared>(k_gradient64<8, LIST>, 8, a, n, LIST, c);
  }
}

}  // namespace

a2c_status launch_density64(a2c_gpp_ctx *c, const double *dX) {
  if (c->N == 0) return A2C_OK;
  return density64<false>(c, site_args(c, dX), c->N);
}

a2c_status launch_gradient64(a2c_gpp_ctx *c, const double *dX, double *dG) {
  if (c->N == 0) return A2C_OK;
  SiteArgs a = site_args(c, dX);
  a.G = dG;
  return gradient64<false>(c, a, c->N);
}

a2c_status launch_eval64_list(a2c_gpp_ctx *c, const double *dX, double *dG, const BatchView &bv) {
  if (c->N == 0) return A2C_OK;
  SiteArgs a = site_args(c, dX);
  a.G = dG;
  a.bv = bv;
  A2C_TRY(density64<true>(c, a, c->N));
  return gradient64<true>(c, a, c->N);
}

a2c_status launch_eam64(a2c_gpp_ctx *c, int which, const double *d_in, int64_t n, double *d_out) {
  if (n <= 0) return A2C_OK;
  k_eam64<<<grid_for(n, 256), 256, 0, c->stream>>>(which, d_in, n, c->p.eps, d_out);
  A2C_CUDA(cudaGetLastError());
  return A2C_OK;
}

a2c_status launch_chem64(a2c_gpp_ctx *c, const double *dX, double /*gamma_bd*/, double *d_send, const int *d_full) {
  if (c->p.nH == 0) return A2C_OK;
  SiteArgs a = site_args(c, dX);
  const double *cp = c->p.coe_Pd, *ch = c->p.coe_H;
  k_chem64<<<grid_for(c->p.nH, kBlock), kBlock, 0, c->stream>>>(a, cp[0], cp[2], cp[3], ch[0], ch[1], ch[2], ch[3],
                                                                 d_full, d_send);
  A2C_CUDA(cudaGetLastError());
  return A2C_OK;
}

}  // namespace a2c
