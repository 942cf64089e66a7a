// Cell-list neighbor build.  Replaces findNeighbors (neighbors.cpp:8-115,
// KD-tree + inclusive d^2 <= rc^2 test, self excluded) followed by
// Minimizer::findLocalNeighbors (minimizer.cpp:833-1144: refilter at rc, Pd
// shell counts PdPdnum, first H shell HH1).  Compiled with -fmad=false so
// the distance test reproduces the reference's arithmetic exactly: the
// neighbor SETS are bit-exact; each list is sorted by global id (the
// reference's order is a KD-tree traversal artefact).
//
// Periodic dimensions use the minimum image, which the reference lacks: the
// image multiplier m = -rint((q_j - q_i)/L) is fixed at build time and
// stored in the entry's top bits, as the reference holds its lists fixed
// through a solve.
//
// Skin (Verlet) lists: with a skin s > 0 the cell-list build makes extended
// candidate lists at rc + s (findNeighbors' _ext lists) and the lists at rc
// are re-filtered from them on the device with the same acceptance test
// (findLocalNeighbors, minimizer.cpp:833-1144).  While no site has moved
// more than s/2 since the extended build, every pair now within rc was
// within rc + s then, and filtering each sorted extended list in order gives
// exactly the lists a full build would.
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>

#include "internal.cuh"

namespace a2c {
namespace {

constexpr int kMaxPerSite = 1000;  // neighbors.cpp:42 (maxNei)

struct GridArgs {
  int n[3];
  int scan_all[3];  // fewer than 2 reach + 1 cells: visit every cell once
  int reach;        // cells to either side that the cutoff can span
  int periodic[3];
  double box[3];
  double rc, rc2, A75, A125;
  int nPd;
  int64_t N;
  const double *X;
  // FP32 prefilter (see prefilter below): positions as float, the largest
  // |coordinate| (as float bits; both from k_scan_positions), the box as float
  const float4 *Xf = nullptr;
  const unsigned *qmax_bits = nullptr;
  float boxf[3] = {0.f, 0.f, 0.f}, invboxf[3] = {0.f, 0.f, 0.f}, Lmaxf = 0.f, rcf = 0.f;
  float rc2f = 0.f, A75f = 0.f, A125f = 0.f;  // the FP64 thresholds rounded to float
  float lof[3] = {0.f, 0.f, 0.f}, invcsf[3] = {0.f, 0.f, 0.f}, csf[3] = {0.f, 0.f, 0.f};  // cell grid
};

// The reference's acceptance test (KDTree.h:250-254 Chebyshev prefilter,
// neighbors.cpp:77-82 self and squared distance) in FP64, with the image
// shift m (fixed by the FP32 prefilter, or decoded from an entry).
__device__ __forceinline__ bool exact_test(const GridArgs &g, int64_t i, int64_t j, const int m[3], uint32_t &entry,
                                           double &d2) {
  if (i == j) return false;
  double dd[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double qi = g.X[4 * i + d];
    double qj = g.X[4 * j + d];
    if (m[d] != 0) qj = qj + m[d] * g.box[d];
    dd[d] = qj - qi;
    if (fabs(dd[d]) > g.rc) return false;
  }
  d2 = dd[0] * dd[0] + dd[1] * dd[1] + dd[2] * dd[2];
  if (d2 > g.rc2) return false;
  if (m[0] < -1 || m[0] > 1 || m[1] < -1 || m[1] > 1 || m[2] < -1 || m[2] > 1) return false;
  entry = (uint32_t)j | ((uint32_t)((m[0] + 1) + 3 * (m[1] + 1) + 9 * (m[2] + 1)) << kIdBits);
  return true;
}

// FP32 prefilter: rejects candidates farther than rc + guard in any
// coordinate or in distance, and picks the image m of the rest.  guard
// bounds the FP32 error of a coordinate difference (coordinates rounded to
// float, one subtraction, the image shift) four times over, so a pair the
// FP64 test accepts is never rejected here; a pair within rc + guard has a
// unique nearest image because the box exceeds 2 (rc + guard) (checked on
// the host before the prefilter is used), so m is the image the FP64
// division rint((qj - qi) / L) would pick.
__device__ __forceinline__ float prefilter_guard(const GridArgs &g) {
  const float qmax = __uint_as_float(*g.qmax_bits);
  return 1e-4f + 1.9073486328125e-6f * (qmax + g.Lmaxf + g.rcf);  // 2^-19 (qmax + L + rc)
}
// The FP32 pass over one candidate: coordinate differences with the image
// m, and their squared length (box and its inverse are 0 in a free
// direction: m = 0).  false: farther than rc + guard (rejected).
__device__ __forceinline__ bool prefilter(const GridArgs &g, float4 fi, float4 fj, float lim, int m[3], float dd[3],
                                          float &d2f) {
  dd[0] = fj.x - fi.x;
  dd[1] = fj.y - fi.y;
  dd[2] = fj.z - fi.z;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float t = dd[d] * g.invboxf[d] + 12582912.0f;  // rounds to an integer (1.5 2^23), kept in its low bits
    dd[d] = dd[d] - (t - 12582912.0f) * g.boxf[d];
    m[d] = 0x4B400000 - __float_as_int(t);
  }
  d2f = dd[0] * dd[0] + dd[1] * dd[1] + dd[2] * dd[2];
  return fmaxf(fmaxf(fabsf(dd[0]), fabsf(dd[1])), fabsf(dd[2])) <= lim && d2f <= lim * lim;
}

// Whether the FP32 values decide every comparison the FP64 test and the
// shell counts make of this pair: each |coordinate difference| at least
// guard inside rc, d^2 at least `band` away from rc^2 and, where the shell
// class is used (shells of a Pd site's Pd neighbors: both thresholds; the
// first H shell of an H site: the lower one; a Pd-H pair: none), from 0.75
// a^2 and 1.25 a^2.  A coordinate difference is off by at most guard/4 (see
// prefilter_guard), so d^2 is off by at most 2 sqrt(3) |d| guard/4 + 3
// (guard/4)^2 plus three FP32 roundings of d^2, which band = 2 guard (rc +
// 1) + 1e-5 bounds for every d up to rc + guard.  The second and third Pd-H
// shells of the fcc lattice lie at 0.75 a^2 and 1.25 a^2: held against
// thresholds that nothing reads, about one of a site's pairs went to the
// FP64 test, whose 25 operations on the narrow FP64 pipe took as long as
// all its candidates' FP32 tests.
__device__ __forceinline__ bool fp32_decides(const GridArgs &g, const float dd[3], float d2f, float guard, bool iPd,
                                             bool jPd) {
  const float band = 2.0f * guard * (g.rcf + 1.0f) + 1e-5f, inner = g.rcf - guard;
  return fabsf(dd[0]) < inner && fabsf(dd[1]) < inner && fabsf(dd[2]) < inner && d2f < g.rc2f - band &&
         (iPd != jPd || (fabsf(d2f - g.A75f) > band && (!iPd || fabsf(d2f - g.A125f) > band)));
}

__device__ __forceinline__ uint32_t encode(int64_t j, const int m[3]) {
  return (uint32_t)j | ((uint32_t)((m[0] + 1) + 3 * (m[1] + 1) + 9 * (m[2] + 1)) << kIdBits);
}

// The shell class of a pair for the Pd shell counts and the first H shell
// (minimizer.cpp:935-947, 999-1004): 0 below 0.75 a^2, 1 strictly between
// 0.75 a^2 and 1.25 a^2, 2 otherwise.
template <class T>
__device__ __forceinline__ int shell_class(T d2, T A75, T A125) {
  return d2 < A75 ? 0 : (d2 > A75 && d2 < A125 ? 1 : 2);
}

// Candidate j of site i.  The FP32 pass rejects everything farther than
// rc + guard and accepts every pair whose decisions it settles
// (fp32_decides: nearly all), its shell class from the FP32 values too (d^2
// lies at least the guard band away from both thresholds, so the FP32
// comparisons give the FP64 answers; GB300's FP64 pipe made the widened
// comparisons the refilter's bound); the rest take the FP64 test.  lim <= 0
// (the prefilter cannot be used: a periodic box of at most 2 (rc + guard))
// takes the image from the FP64 division and the FP64 test.
__device__ __forceinline__ bool pair_test(const GridArgs &g, int i, float4 fi, float lim, int j, float4 fj,
                                          uint32_t &entry, int &cls) {
  int m[3];
  float dd[3], d2f;
  const bool near = prefilter(g, fi, fj, lim, m, dd, d2f);
  if (i == j || (lim > 0.0f && !near)) return false;
  if (lim > 0.0f && fp32_decides(g, dd, d2f, lim - g.rcf, i < g.nPd, j < g.nPd) &&
      max(max(abs(m[0]), abs(m[1])), abs(m[2])) <= 1) {
    entry = encode(j, m);
    cls = shell_class(d2f, g.A75f, g.A125f);
    return true;
  }
  if (!(lim > 0.0f)) {
#pragma unroll
    for (int d = 0; d < 3; ++d)
      m[d] = g.periodic[d] ? -(int)rint((g.X[4 * (int64_t)j + d] - g.X[4 * (int64_t)i + d]) / g.box[d]) : 0;
  }
  double d2;
  if (!exact_test(g, i, j, m, entry, d2)) return false;
  cls = shell_class(d2, g.A75, g.A125);
  return true;
}

// The prefilter's cutoff for this build, or 0 when it cannot be used.
__device__ __forceinline__ float prefilter_lim(const GridArgs &g) {
  const float lim = g.rcf + prefilter_guard(g);
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (g.periodic[d] && !(0.5f * g.boxf[d] > lim * 1.0001f)) return 0.0f;
  return lim;
}

// Doubles as unsigned integers in the same order, and back.
__device__ __forceinline__ unsigned long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return (unsigned long long)b ^ ((unsigned long long)(b >> 63) | 0x8000000000000000ull);
}
double from_order_key(unsigned long long k) {
  const unsigned long long b = k >> 63 ? k ^ 0x8000000000000000ull : ~k;
  double x;
  std::memcpy(&x, &b, sizeof(x));
  return x;
}
// The largest unsigned v of a full warp, for 64-bit values
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
  return (unsigned long long)hi << 32 | lo;
}

// One pass over the positions X (device memory, or host memory the device
// reads, copied then to Xout): the entry points' checks -- kPosMoved when a
// site is more than sqrt(lim2) from Xref (may be null), kPosNonfinite,
// kPosOutside for a periodic coordinate outside [-L/2, 3L/2] --, the
// positions as float for the prefilter with the largest |coordinate|, and
// the extents of the free directions (which the cell grid needs).
__global__ void k_scan_positions(const double *X, double *Xout, const double *Xref, int64_t n, double lim2, double L0,
                                 double L1, double L2, int per, float4 *Xf, PosScan *out) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t t = s < n ? s : n - 1;  // every lane takes part in the reductions
  const double x = X[4 * t], y = X[4 * t + 1], z = X[4 * t + 2], w = X[4 * t + 3];
  int f = 0;
  if (s < n) {
    if (Xout) {
      Xout[4 * s] = x;
      Xout[4 * s + 1] = y;
      Xout[4 * s + 2] = z;
      Xout[4 * s + 3] = w;
    }
    Xf[s] = make_float4((float)x, (float)y, (float)z, 0.0f);
    if (!isfinite(x) || !isfinite(y) || !isfinite(z) || !isfinite(w)) f |= kPosNonfinite;
    if (((per & 1) && (x < -0.5 * L0 || x > 1.5 * L0)) || ((per & 2) && (y < -0.5 * L1 || y > 1.5 * L1)) ||
        ((per & 4) && (z < -0.5 * L2 || z > 1.5 * L2)))
      f |= kPosOutside;
    if (Xref) {
      const double dx = x - Xref[4 * s], dy = y - Xref[4 * s + 1], dz = z - Xref[4 * s + 2];
      if (dx * dx + dy * dy + dz * dz > lim2) f |= kPosMoved;
    }
  }
  f = __reduce_or_sync(0xffffffffu, f);
  const float q = fmaxf(fabsf((float)x), fmaxf(fabsf((float)y), fabsf((float)z)));
  const unsigned qm = __reduce_max_sync(0xffffffffu, __float_as_uint(q));  // a NaN's bits are the largest
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    if (f) atomicOr(&out->flags, f);
    // one ulp up: the float rounding of |q| may round down
    if (qm + 1u > out->qmax_bits) atomicMax(&out->qmax_bits, qm + 1u);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (per >> d & 1) continue;
    const unsigned long long k = order_key(d == 0 ? x : d == 1 ? y : z);
    const unsigned long long hi = warp_max(k), lo = ~warp_max(~k);
    if (lane == 0) {
      if (hi > out->hi[d]) atomicMax(&out->hi[d], hi);
      if (lo < out->lo[d]) atomicMin(&out->lo[d], lo);
    }
  }
}

// ------------------------------------------------------------- cell list
// A site's place in the cell grid, in FP32: its coordinate wrapped into the
// periodic box (or from the lowest site of a free direction), and the cell
// it falls in.  The wrapped coordinate is off by less than 2^-21 (qmax + L)
// and stays with its cell where rounding takes it just outside the box; the
// cells are wider than the cutoff by 16 times that (make_grid), so every
// pair within the cutoff lies in neighboring cells.
__device__ __forceinline__ float grid_pos(const GridArgs &g, float x, int d) {
  return g.periodic[d] ? x - g.boxf[d] * floorf(x * g.invboxf[d]) : x - g.lof[d];
}
__device__ __forceinline__ int grid_cell(const GridArgs &g, float t, int d) {
  return min(max((int)floorf(t * g.invcsf[d]), 0), g.n[d] - 1);
}

// The sites of a cell lie together in cpos (grid position, id in w), so the
// cells along x of one (y, z) row are one run of memory.  Cell and rank
// within the cell by one atomic; the order within a cell does not matter
// (the fill sorts each list).
__global__ void k_cell_count(GridArgs g, int2 *cell, int *ccount) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.N) return;
  const float4 f = g.Xf[s];
  const int c0 = grid_cell(g, grid_pos(g, f.x, 0), 0), c1 = grid_cell(g, grid_pos(g, f.y, 1), 1),
            c2 = grid_cell(g, grid_pos(g, f.z, 2), 2);
  const int c = (c2 * g.n[1] + c1) * g.n[0] + c0;
  cell[s] = make_int2(c, atomicAdd(&ccount[c], 1));
}

__global__ void k_cell_fill(GridArgs g, const int2 *cell, const int *cstart, float4 *cpos) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= g.N) return;
  const int2 c = cell[s];
  const float4 f = g.Xf[s];
  cpos[cstart[c.x] + c.y] =
      make_float4(grid_pos(g, f.x, 0), grid_pos(g, f.y, 1), grid_pos(g, f.z, 2), __int_as_float((int)s));
}

constexpr unsigned kAll = 0xffffffffu;
constexpr int kListWarps = 8;  // sites (one per warp) of a block of the list kernels
constexpr int kQueue = 64;     // candidates awaiting the pair test: below 32, plus one step's

// A warp's scratch of scan_cells: the runs of cpos it looks through (first
// slot minus the candidates before it, the site as the run's sites see it),
// the candidates before each run, and the queue.
constexpr int kRuns = 50;  // 25 rows, each in at most two pieces
struct ScanShared {
  float4 run[kRuns];  // x, y, z; w: int bits of first - before
  int before[kRuns + 1];
  int queue[kQueue];
};

// The candidates of site i (at grid position p), a warp at a time.  Lane r
// takes the r-th (y, z) row of cells within reach and finds the run of
// cells of the row that the cutoff sphere can touch (two runs where the row
// crosses a periodic boundary); then the lanes take the runs' sites 32 at a
// time, end to end over the runs, through a distance test that rejects only
// what is farther than rc + 2 guard, and queue the rest in shared memory;
// each 32 of the queue go through the whole pair test.  Cells half the
// cutoff wide (reach 2) leave about 220 candidates of a bulk site's 80
// neighbors, where the 27 cells a cutoff wide held 580.  emit(j, entry,
// cls, hit, mask) is called by all lanes with the mask of those that hold a
// neighbor.  Periodic directions seen whole take the nearest image.
template <class Emit>
__device__ __forceinline__ void scan_cells(const GridArgs &g, const int *cstart, const float4 *cpos, int i, float4 p,
                                           ScanShared &sh, Emit emit) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const float4 fi = g.Xf[i];
  const float lim = prefilter_lim(g), far = g.rcf + 2.0f * prefilter_guard(g), far2 = far * far;
  const float pos[3] = {p.x, p.y, p.z};
  int c[3], lo[3], hi[3];
  bool wrap = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c[d] = grid_cell(g, pos[d], d);
    lo[d] = g.scan_all[d] ? 0 : c[d] - g.reach;
    hi[d] = g.scan_all[d] ? g.n[d] - 1 : c[d] + g.reach;
    if (!g.periodic[d]) {
      lo[d] = max(lo[d], 0);
      hi[d] = min(hi[d], g.n[d] - 1);
    }
    wrap = wrap || (g.scan_all[d] && g.periodic[d]);
  }
  // this lane's row: cells (a, b), where it lies, and its run of x cells
  const int wide = hi[1] - lo[1] + 1;
  const int a = lo[2] + lane / wide, b = lo[1] + lane % wide;
  float y = p.y, z = p.z, x1 = p.x;
  int first0 = 0, len0 = 0, first1 = 0, len1 = 0;
  if (a <= hi[2]) {
    // distance of the site from the row in y and z, less the slack that
    // rounding a position into its cell can take
    constexpr float slack = 2e-3f;
    float rest = far2;
    if (!g.scan_all[1]) {
      const float t = fmaxf(fmaxf((float)b * g.csf[1] - p.y, p.y - (float)(b + 1) * g.csf[1]) - slack, 0.0f);
      rest = fmaf(-t, t, rest);
    }
    if (!g.scan_all[2]) {
      const float t = fmaxf(fmaxf((float)a * g.csf[2] - p.z, p.z - (float)(a + 1) * g.csf[2]) - slack, 0.0f);
      rest = fmaf(-t, t, rest);
    }
    int l = lo[0], h = hi[0];
    if (!g.scan_all[0]) {
      const float w = sqrtf(fmaxf(rest, 0.0f)) + slack;
      l = max(l, (int)floorf((p.x - w) * g.invcsf[0]));
      h = min(h, (int)floorf((p.x + w) * g.invcsf[0]));
    }
    if (rest > 0.0f && l <= h) {
      const int ca = a < 0 ? a + g.n[2] : a >= g.n[2] ? a - g.n[2] : a;
      const int cb = b < 0 ? b + g.n[1] : b >= g.n[1] ? b - g.n[1] : b;
      z = a < 0 ? p.z + g.boxf[2] : a >= g.n[2] ? p.z - g.boxf[2] : p.z;
      y = b < 0 ? p.y + g.boxf[1] : b >= g.n[1] ? p.y - g.boxf[1] : p.y;
      const int *row = cstart + (ca * g.n[1] + cb) * g.n[0];
      const int l0 = max(l, 0), h0 = min(h, g.n[0] - 1);
      if (l0 <= h0) {
        first0 = __ldg(&row[l0]);
        len0 = __ldg(&row[h0 + 1]) - first0;
      }
      if (l < 0) {
        first1 = __ldg(&row[l + g.n[0]]);
        len1 = __ldg(&row[min(h, -1) + g.n[0] + 1]) - first1;
        x1 = p.x + g.boxf[0];
      } else if (h >= g.n[0]) {
        first1 = __ldg(&row[max(l, g.n[0]) - g.n[0]]);
        len1 = __ldg(&row[h - g.n[0] + 1]) - first1;
        x1 = p.x - g.boxf[0];
      }
    }
  }
  __syncwarp();
  int total = 0, runs = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int len = k ? len1 : len0;
    const unsigned some = __ballot_sync(kAll, len > 0);
    if (!some) continue;
    int at = len;  // inclusive sum over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kAll, at, o);
      if (lane >= o) at += v;
    }
    if (len > 0) {
      const int r = runs + __popc(some & below), before = total + at - len;
      sh.run[r] = make_float4(k ? x1 : p.x, y, z, __int_as_float((k ? first1 : first0) - before));
      sh.before[r] = before;
    }
    total += __shfl_sync(kAll, at, 31);
    runs += __popc(some);
  }
  if (lane == 0) sh.before[runs] = total;
  __syncwarp();
  int q = 0;
  auto test = [&](int n) {  // the last n of the queue
    uint32_t e = 0;
    int cls = 0, j = -1;
    bool hit = false;
    if (lane < n) {
      j = sh.queue[q - n + lane];
      hit = pair_test(g, i, fi, lim, j, __ldg(&g.Xf[j]), e, cls);
    }
    q -= n;
    const unsigned mask = __ballot_sync(kAll, hit);
    if (mask) emit(j, e, cls, hit, mask);
  };
  int r = 0;  // this lane's run
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = min(t0 + lane, total - 1);
    while (t >= sh.before[r + 1]) ++r;
    const float4 s = sh.run[r];
    const float4 f = __ldg(&cpos[__float_as_int(s.w) + t]);
    float dx = f.x - s.x, dy = f.y - s.y, dz = f.z - s.z;
    if (wrap) {
      if (g.scan_all[0]) dx = dx - rintf(dx * g.invboxf[0]) * g.boxf[0];
      if (g.scan_all[1]) dy = dy - rintf(dy * g.invboxf[1]) * g.boxf[1];
      if (g.scan_all[2]) dz = dz - rintf(dz * g.invboxf[2]) * g.boxf[2];
    }
    const bool in = t0 + lane < total && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= far2;
    const unsigned mask = __ballot_sync(kAll, in);
    if (!mask) continue;
    if (in) sh.queue[q + __popc(mask & below)] = __float_as_int(f.w);
    q += __popc(mask);
    __syncwarp();
    if (q >= 32) {
      test(32);
      __syncwarp();
    }
  }
  if (q) test(q);
}

// The counts of a site's list, gathered 32 candidates at a time; equal in
// all lanes.
struct ListCounts {
  int n = 0, nP = 0, n1 = 0, sh0 = 0, sh1 = 0;
  // mask: the lanes with a neighbor; pd: those with a Pd neighbor
  __device__ __forceinline__ void add(bool iPd, bool jPd, int cls, bool hit, unsigned mask, unsigned pd) {
    const unsigned c0 = __ballot_sync(kAll, hit && cls == 0);
    n += __popc(mask);
    nP += __popc(pd);
    if (iPd) {  // minimizer.cpp:935-947
      sh0 += __popc(pd & c0);
      sh1 += __popc(__ballot_sync(kAll, hit && jPd && cls == 1));
    } else {  // minimizer.cpp:999-1004
      n1 += __popc(c0 & ~pd);
    }
  }
  // npd, shell and hh1count may be null (extended lists)
  __device__ __forceinline__ void store(const GridArgs &g, int i, bool iPd, int64_t *count, int *npd,
                                        int64_t *hh1count, int *shell, int *most) const {
    count[i] = n;
    if (npd) npd[i] = nP;
    if (iPd) {
      if (shell) {
        shell[3 * i] = sh0;
        shell[3 * i + 1] = sh1;
        shell[3 * i + 2] = nP - sh0 - sh1;
      }
    } else if (hh1count) {
      hh1count[i - g.nPd] = n1;
    }
    if (n > *(volatile int *)most) atomicMax(most, n);
  }
};

// An entry with its id on top, so that entries compare by id.
__device__ __forceinline__ uint32_t by_id(uint32_t e) { return __funnelshift_l(e, e, 32 - kIdBits); }
__device__ __forceinline__ uint32_t from_by_id(uint32_t k) { return __funnelshift_r(k, k, 32 - kIdBits); }

// Writes the warp's n keys of src (shared memory, 16-byte aligned, room for
// a multiple of 4; any order, all different) in increasing order to out:
// each goes to its rank, the count of smaller keys, two per lane a pass.
template <class Out>
__device__ __forceinline__ void write_sorted(uint32_t *src, int n, Out out) {
  const int lane = threadIdx.x & 31;
  if (n + lane < ((n + 3) & ~3)) src[n + lane] = ~0u;
  __syncwarp();
  for (int r = lane; r - lane < n; r += 64) {
    const uint32_t k0 = r < n ? src[r] : 0u, k1 = r + 32 < n ? src[r + 32] : 0u;
    int r0 = 0, r1 = 0;
    for (int t = 0; t < n; t += 4) {
      const uint4 v = *reinterpret_cast<const uint4 *>(src + t);
      r0 += (v.x < k0) + (v.y < k0) + (v.z < k0) + (v.w < k0);
      r1 += (v.x < k1) + (v.y < k1) + (v.z < k1) + (v.w < k1);
    }
    if (r < n) out(r0, k0);
    if (r + 32 < n) out(r1, k1);
  }
}

// Room for a list of n entries, and the dynamic shared memory of a block of
// k_cell_lists at that room (at most 64 KB, at kMaxPerSite).
constexpr int list_room(int n) { return (n + 31) & ~31; }
constexpr size_t list_smem(int room) { return sizeof(uint32_t) * 2 * (size_t)room * kListWarps; }

// The list of every site, sorted by id -- Pd neighbors, then H neighbors --
// at out[i * room] or, with off, at out[off[i]], with its counts; a list
// longer than `room` is only counted (the host then calls again with the
// lists' offsets and the longest one's length).  Warp k takes the k-th site
// of cpos, so that a block's sites share cells and find their candidates in
// the L1.  The neighbors gather in the warp's shared memory (two areas of
// `room` entries, Pd and H), where each finds its rank.
__global__ void __launch_bounds__(32 * kListWarps) k_cell_lists(GridArgs g, const int *cstart, const float4 *cpos,
                                                                uint32_t *out, const int64_t *off, int room,
                                                                int64_t *count, int *npd, int64_t *hh1count,
                                                                int *shell, int *most) {
  extern __shared__ uint4 lists[];
  __shared__ ScanShared scan[kListWarps];
  const int64_t k = (int64_t)blockIdx.x * kListWarps + threadIdx.x / 32;
  if (k >= g.N) return;
  const int lane = threadIdx.x & 31;
  uint32_t *const pd = reinterpret_cast<uint32_t *>(lists) + (size_t)(threadIdx.x / 32) * 2 * room,
                  *const h = pd + room;
  const float4 p = __ldg(&cpos[k]);
  const int i = __float_as_int(p.w);
  const bool iPd = i < g.nPd;
  const unsigned below = (1u << lane) - 1u;
  ListCounts c;
  scan_cells(g, cstart, cpos, i, p, scan[threadIdx.x / 32], [&](int j, uint32_t e, int cls, bool hit, unsigned mask) {
    const bool jPd = j < g.nPd;
    const unsigned mine = __ballot_sync(kAll, hit && jPd);
    if (hit) {
      const int at = jPd ? c.nP + __popc(mine & below) : c.n - c.nP + __popc(mask & ~mine & below);
      if (at < room) (jPd ? pd : h)[at] = by_id(e);
    }
    c.add(iPd, jPd, cls, hit, mask, mine);
  });
  if (lane == 0) c.store(g, i, iPd, count, npd, hh1count, shell, most);
  if (c.n > room) return;
  __syncwarp();
  uint32_t *const list = out + (off ? off[i] : (int64_t)i * room);
  const int nP = c.nP;
  write_sorted(pd, nP, [&](int r, uint32_t v) { list[r] = from_by_id(v); });
  write_sorted(h, c.n - nP, [&](int r, uint32_t v) { list[nP + r] = from_by_id(v); });
}

// What the host needs to go on after the counts, into its pinned memory.
struct ListReport {
  long long total, total1;
  int most;
};
__global__ void k_report(const int64_t *total, const int64_t *total1, const int *most, ListReport *out) {
  out->total = *total;
  out->total1 = total1 ? *total1 : 0;
  out->most = *most;
}

// Skin refilter, one exact pass over the extended lists, a warp per site:
// site i's neighbors at rc go to tmp[ext_off[i] ...] in the extended list's
// order -- its Pd part, then its H part, each sorted by id, the order
// a full build gives -- with its counts.
__global__ void __launch_bounds__(32 * kListWarps) k_refilter(GridArgs g, const int64_t *ext_off,
                                                              const uint32_t *ext_nbr, uint32_t *tmp, int64_t *count,
                                                              int *npd, int64_t *hh1count, int *shell, int *most) {
  const int i = (int)(blockIdx.x * kListWarps + threadIdx.x / 32);
  if (i >= (int)g.N) return;
  const int lane = threadIdx.x & 31;
  const int64_t b = ext_off[i];
  const int len = (int)(ext_off[i + 1] - b);
  const bool iPd = i < g.nPd;
  const float4 fi = g.Xf[i];
  const float lim = prefilter_lim(g);
  ListCounts c;
  for (int t0 = 0; t0 < len; t0 += 32) {
    uint32_t e = 0;
    int cls = 0, j = -1;
    bool hit = false;
    if (t0 + lane < len) {
      j = (int)(__ldg(&ext_nbr[b + t0 + lane]) & kIdMask);
      hit = pair_test(g, i, fi, lim, j, __ldg(&g.Xf[j]), e, cls);
    }
    const unsigned mask = __ballot_sync(kAll, hit);
    if (hit) tmp[b + c.n + __popc(mask & ((1u << lane) - 1u))] = e;
    c.add(iPd, j < g.nPd, cls, hit, mask, __ballot_sync(kAll, hit && j < g.nPd));
  }
  if (lane == 0) c.store(g, i, iPd, count, npd, hh1count, shell, most);
}

// The lists of k_cell_lists (at i * stride) or k_refilter (at src_off[i])
// packed at their offsets, and each H site's first H shell (hh1; null for
// extended lists).  tmp may be nbr, with src_off = off: lists in place.
__global__ void __launch_bounds__(32 * kListWarps) k_pack(GridArgs g, const int64_t *src_off, int stride,
                                                          const uint32_t *tmp, const int64_t *off, uint32_t *nbr,
                                                          const int64_t *hh1_off, int *hh1, int *status) {
  const int i = (int)(blockIdx.x * kListWarps + threadIdx.x / 32);
  if (i >= (int)g.N) return;
  const int lane = threadIdx.x & 31;
  const int64_t b = off[i];
  const int n = (int)(off[i + 1] - b);
  const uint32_t *src = tmp + (src_off ? src_off[i] : (int64_t)i * stride);
  const bool first = hh1 && i >= g.nPd;
  const float4 fi = g.Xf[i];
  const float lim = prefilter_lim(g);
  const int64_t h0 = first ? hh1_off[i - g.nPd] : 0;
  const int n1 = first ? (int)(hh1_off[i - g.nPd + 1] - h0) : 0;
  int w1 = 0;
  for (int t0 = 0; t0 < n; t0 += 32) {
    const bool has = t0 + lane < n;
    const uint32_t ent = has ? src[t0 + lane] : 0u;
    if (has) nbr[b + t0 + lane] = ent;
    if (!first) continue;
    const int j = (int)(ent & kIdMask);
    uint32_t en;
    int cls = 2;
    const bool h = has && j >= g.nPd && pair_test(g, i, fi, lim, j, __ldg(&g.Xf[j]), en, cls) && cls == 0;
    const unsigned m1 = __ballot_sync(kAll, h);
    const int at = w1 + __popc(m1 & ((1u << lane) - 1u));
    if (h && at < n1) hh1[h0 + at] = j - g.nPd;
    w1 += __popc(m1);
  }
  if (w1 != n1 && lane == 0) atomicOr(status, kStatusBadIndex);
}

// The scratch of a list build or re-filter, kept with the context.
// (Stream-ordered allocations per call went back to the system at every
// synchronization of the call and cost it more than its kernels.)  About 90
// bytes a site in `base`, at most 40 in `cells`; `tmp` holds 4 bytes for
// each of a site's `stride` entries, at most 512 bytes a site or twice the
// lists themselves, whichever is more, and is given back when the context
// needs the memory for something else (context_malloc).
struct ListWork {
  void *base = nullptr;     // one allocation for the views below
  uint32_t *tmp = nullptr;  // lists before they are packed
  int64_t tmp_cap = 0;
  int stride = 96, ext_stride = 128;  // entries per site there (a multiple of 4)
  int *cells = nullptr;  // the cell grid: counts, offsets, and the scratch of their scan
  int64_t cells_cap = 0;
  // views of base
  double *stage = nullptr;  // 4N
  float4 *Xf = nullptr, *cpos = nullptr;
  int2 *cell = nullptr;
  int64_t *count = nullptr, *hh1c = nullptr;
  int *npd = nullptr, *most = nullptr;
  PosScan *scan = nullptr;
  void *cub = nullptr;
  size_t cub_bytes = 0;
  ListReport *report = nullptr;  // in the context's pinned memory, as is
  PosScan *scanned = nullptr;    // the last scan
};

a2c_status work_for(a2c_gpp_ctx *c, ListWork **out) {
  if (!c->list_work) {
    c->list_work = new (std::nothrow) ListWork();
    if (!c->list_work) return A2C_ERR_NOMEM;
  }
  ListWork *w = (ListWork *)c->list_work;
  *out = w;
  if (w->base) return A2C_OK;
  w->report = (ListReport *)(c->h_small + kHostReport);
  w->scanned = (PosScan *)(w->report + 1);
  static_assert(sizeof(ListReport) + sizeof(PosScan) <= sizeof(double) * (kHostSmall - kHostReport), "pinned area");
  const int64_t N = std::max<int64_t>(c->N, 1), nH = c->p.nH;
  size_t b0 = 0, b1 = 0;
  A2C_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b0, (const int64_t *)nullptr, (int64_t *)nullptr, N + 1, c->stream));
  A2C_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b1, (const int64_t *)nullptr, (int64_t *)nullptr, nH + 1, c->stream));
  constexpr int kParts = 10;
  const size_t bytes[kParts] = {sizeof(double) * 4 * N, sizeof(float4) * N,       sizeof(float4) * N,
                                sizeof(int2) * N,       sizeof(int64_t) * (N + 1), sizeof(int64_t) * (nH + 1),
                                sizeof(int) * N,        sizeof(int),               sizeof(PosScan),
                                std::max(b0, b1)};
  size_t at[kParts + 1] = {0};
  for (int k = 0; k < kParts; ++k) at[k + 1] = (at[k] + bytes[k] + 255) & ~(size_t)255;
  if (context_malloc(c, &w->base, at[kParts]) != cudaSuccess) return A2C_ERR_NOMEM;
  char *p = (char *)w->base;
  w->stage = (double *)(p + at[0]);
  w->Xf = (float4 *)(p + at[1]);
  w->cpos = (float4 *)(p + at[2]);
  w->cell = (int2 *)(p + at[3]);
  w->count = (int64_t *)(p + at[4]);
  w->hh1c = (int64_t *)(p + at[5]);
  w->npd = (int *)(p + at[6]);
  w->most = (int *)(p + at[7]);
  w->scan = (PosScan *)(p + at[8]);
  w->cub = p + at[9];
  w->cub_bytes = bytes[9];
  return A2C_OK;
}

a2c_status scan_exclusive(ListWork *w, const int64_t *in, int64_t *out, int64_t n, cudaStream_t st) {
  A2C_CUDA(cub::DeviceScan::ExclusiveSum(w->cub, w->cub_bytes, in, out, n, st));
  return A2C_OK;
}

// Cells of a grid whose tables stay with the context; a larger one (a
// sparse system in free directions) gives them back after the build.
constexpr int64_t cells_kept(int64_t n_sites) { return 4 * n_sites + 4096; }

// Cell grid for cutoff `cut` (`reach` cells to either side span it), from the extents
// of the free directions; with scan null (a list re-filter, which uses no
// cells) they are left nominal.
int64_t make_grid(const a2c_gpp_ctx *c, const PosScan *scan, double cut, GridArgs &g) {
  const int64_t N = c->N;
  const a2c_gpp_params &p = c->p;
  g = GridArgs{};
  g.N = N;
  g.nPd = p.nPd;
  g.X = c->d_X;
  g.rc = cut;
  g.rc2 = cut * cut;
  g.A75 = p.a_Pd * p.a_Pd * 0.75;
  g.A125 = p.a_Pd * p.a_Pd * 1.25;
  g.rcf = (float)cut;
  g.rc2f = (float)g.rc2;
  g.A75f = (float)g.A75;
  g.A125f = (float)g.A125;
  for (int d = 0; d < 3; ++d)
    if (p.periodic[d]) {
      g.boxf[d] = (float)p.box[d];
      g.invboxf[d] = (float)(1.0 / p.box[d]);
      g.Lmaxf = std::max(g.Lmaxf, (float)p.box[d]);
    }
  int64_t ncell = 1;
  // wider than the cutoff by the FP32 grid positions' error, 16 times over
  // (see grid_pos), and what rounding a position in cells can add
  float qmax = 0.0f;
  if (scan) std::memcpy(&qmax, &scan->qmax_bits, sizeof(qmax));
  const double wide = cut + 4e-3 + 8e-6 * ((double)qmax + g.Lmaxf);
  double extent[3];
  for (int d = 0; d < 3; ++d) {
    g.periodic[d] = p.periodic[d] ? 1 : 0;
    g.box[d] = p.box[d];
    double ext = cut;
    if (g.periodic[d]) {
      ext = p.box[d];
    } else if (scan && N > 0) {
      const double lo = from_order_key(scan->lo[d]);
      g.lof[d] = (float)lo;
      ext = from_order_key(scan->hi[d]) - lo;
    }
    extent[d] = ext;
  }
  // cells half the cutoff wide, unless they would far outnumber the sites
  for (g.reach = 2; g.reach >= 1; --g.reach) {
    ncell = 1;
    for (int d = 0; d < 3; ++d) {
      const double cells = std::floor(extent[d] / (wide / g.reach));
      const int n = cells >= 1.0 ? (int)std::min(cells, 512.0) : 1;  // (a NaN extent: 1)
      g.n[d] = n;
      g.csf[d] = (float)(extent[d] / n);
      g.invcsf[d] = (extent[d] > 0.0) ? (float)(n / extent[d]) : 1.0f;
      g.scan_all[d] = n < 2 * g.reach + 1 ? 1 : 0;
      ncell *= n;
    }
    if (g.reach == 1 || ncell <= cells_kept(N)) break;
  }
  return ncell;
}

template <class T>
a2c_status grow(a2c_gpp_ctx *c, T **p, int64_t *cap, int64_t need) {
  if (need <= *cap) return A2C_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  if (context_malloc(c, (void **)p, sizeof(T) * std::max<int64_t>(need, 1)) != cudaSuccess) return A2C_ERR_NOMEM;
  *cap = need;
  return A2C_OK;
}

// The positions X (or, with X null, those in c->d_X) scanned into the
// context's scratch; waits for the result.
a2c_status scan_positions(a2c_gpp_ctx *c, ListWork *w, const double *X, double *Xout, const double *Xref,
                          PosScan *res) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  std::memset(res, 0, sizeof(*res));
  if (N <= 0) return A2C_OK;
  int per = 0;
  for (int d = 0; d < 3; ++d) per |= c->p.periodic[d] ? 1 << d : 0;
  const double half = 0.5 * c->skin;
  // flags, qmax and hi start at 0, lo at all ones
  A2C_CUDA(cudaMemsetAsync(w->scan, 0, sizeof(PosScan), st));
  A2C_CUDA(cudaMemsetAsync(w->scan->lo, 0xff, sizeof(w->scan->lo), st));
  k_scan_positions<<<grid_for(N, 256), 256, 0, st>>>(X ? X : c->d_X, Xout, Xref, N, half * half, c->p.box[0],
                                                     c->p.box[1], c->p.box[2], per, w->Xf, w->scan);
  A2C_CUDA(cudaGetLastError());
  A2C_CUDA(cudaMemcpyAsync(w->scanned, w->scan, sizeof(PosScan), cudaMemcpyDeviceToHost, st));
  A2C_CUDA(cudaStreamSynchronize(st));
  *res = *w->scanned;
  return A2C_OK;
}

// After the counts: offsets, the totals on the host, room for the lists
// (for which tmp, and what it holds, may have to go: null then).
a2c_status place_lists(a2c_gpp_ctx *c, ListWork *w, bool ext) {
  const int64_t N = c->N;
  const int nH = c->p.nH;
  cudaStream_t st = c->stream;
  int64_t *off = ext ? c->d_ext_off : c->d_off;
  A2C_TRY(scan_exclusive(w, (const int64_t *)w->count, off, N + 1, st));
  if (!ext) A2C_TRY(scan_exclusive(w, (const int64_t *)w->hh1c, c->d_hh1_off, (int64_t)nH + 1, st));
  k_report<<<1, 1, 0, st>>>(off + N, ext ? nullptr : c->d_hh1_off + nH, w->most, w->report);
  A2C_CUDA(cudaGetLastError());
  A2C_CUDA(cudaStreamSynchronize(st));
  const ListReport r = *w->report;
  if (r.most > kMaxPerSite) return A2C_ERR_NEIGHBOR_OVERFLOW;
  if (ext) {
    A2C_TRY(grow(c, &c->d_ext_nbr, &c->ext_cap, r.total));
    c->ext_total = r.total;
  } else {
    A2C_TRY(grow(c, &c->d_nbr, &c->nbr_cap, r.total));
    A2C_TRY(grow(c, &c->d_hh1, &c->hh1_cap, r.total1));
    c->nbr_total = r.total;
    c->hh1_total = r.total1;
    c->max_neighbors = r.most;
  }
  return A2C_OK;
}

a2c_status clear_counts(a2c_gpp_ctx *c, ListWork *w) {
  cudaStream_t st = c->stream;
  A2C_CUDA(cudaMemsetAsync(c->d_status, 0, sizeof(int), st));
  A2C_CUDA(cudaMemsetAsync(w->count + c->N, 0, sizeof(int64_t), st));
  A2C_CUDA(cudaMemsetAsync(w->hh1c + c->p.nH, 0, sizeof(int64_t), st));
  A2C_CUDA(cudaMemsetAsync(w->most, 0, sizeof(int), st));
  return A2C_OK;
}

// The lists at rc are new: the span guard's positions and reach.
a2c_status lists_done(a2c_gpp_ctx *c, double cut) {
  ++c->nbr_version;
  for (int d = 0; d < 3; ++d) c->list_reach[d] = c->p.periodic[d] ? 0.0 : cut;
  if (c->d_xlist && c->N > 0)
    A2C_CUDA(cudaMemcpyAsync(c->d_xlist, c->d_X, sizeof(double) * 4 * c->N, cudaMemcpyDeviceToDevice, c->stream));
  return A2C_OK;
}

// Every site into its cell: the cells' offsets (cstart) and, in their order,
// the sites (w->cpos).
a2c_status fill_cells(a2c_gpp_ctx *c, ListWork *w, const GridArgs &g, int64_t ncell, const int **cstart) {
  cudaStream_t st = c->stream;
  size_t cub_bytes = 0;
  A2C_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, (const int *)nullptr, (int *)nullptr, ncell + 1, st));
  const int64_t room = (ncell + 1 + 63) & ~(int64_t)63;  // 256-byte parts
  A2C_TRY(grow(c, &w->cells, &w->cells_cap, 2 * room + (int64_t)(cub_bytes + sizeof(int) - 1) / (int64_t)sizeof(int)));
  int *const ccount = w->cells, *const start = ccount + room;
  A2C_CUDA(cudaMemsetAsync(ccount, 0, sizeof(int) * (ncell + 1), st));
  k_cell_count<<<grid_for(c->N, 256), 256, 0, st>>>(g, w->cell, ccount);
  A2C_CUDA(cudaGetLastError());
  A2C_CUDA(cub::DeviceScan::ExclusiveSum(start + room, cub_bytes, (const int *)ccount, start, ncell + 1, st));
  k_cell_fill<<<grid_for(c->N, 256), 256, 0, st>>>(g, w->cell, start, w->cpos);
  A2C_CUDA(cudaGetLastError());
  *cstart = start;
  return A2C_OK;
}

// Lists (rc, or rc + skin for the extended lists, which have no shells or
// first H shells) from a cell list over the scanned positions.  One pass
// makes the sorted lists at a fixed stride (at first 96, 128 for extended
// lists) and a copy packs them.  Lists that do not fit it, or for whose
// stride there is no memory, are counted by that pass and written at their
// offsets by a second; the stride then grows to the longest list unless a
// few long ones would make it more than twice what the lists take.  Bound by
// instruction issue and the latency of the candidate loads (about 2,100
// instructions a site by a warp).  At 262,144 sites the pass takes 568 us and the copy
// 137; one thread per site that walked its 27 cells twice, to count and to
// fill, and sorted in global memory took 930 + 1,500 us; a warp per site over
// those 27 cells in two passes took 576 + 862 us.
a2c_status lists_from_cells(a2c_gpp_ctx *c, const PosScan &scan, double cut, bool ext) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  GridArgs g;
  const int64_t ncell = make_grid(c, &scan, cut, g);
  ListWork *w;
  A2C_TRY(work_for(c, &w));
  g.Xf = w->Xf;
  g.qmax_bits = &w->scan->qmax_bits;
  const unsigned blocks = grid_for(N, kListWarps);
  const int *cstart = nullptr;
  if (N > 0) A2C_TRY(fill_cells(c, w, g, ncell, &cstart));
  auto pass = [&](uint32_t *out, const int64_t *off, int room) -> a2c_status {
    const size_t smem = list_smem(room);
    // always the largest size: the attribute is the kernel's, and another
    // thread may be about to launch it for its own context
    if (smem + sizeof(ScanShared) * kListWarps > 48 * 1024)
      A2C_CUDA(cudaFuncSetAttribute(k_cell_lists, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)list_smem(list_room(kMaxPerSite))));
    k_cell_lists<<<blocks, 32 * kListWarps, smem, st>>>(g, cstart, w->cpos, out, off, room, w->count,
                                                        ext ? w->npd : c->d_npd, ext ? nullptr : w->hh1c,
                                                        ext ? nullptr : c->d_shell, w->most);
    A2C_CUDA(cudaGetLastError());
    return A2C_OK;
  };
  int &stride = ext ? w->ext_stride : w->stride;
  int room = stride;
  if (grow(c, &w->tmp, &w->tmp_cap, N * stride) != A2C_OK) room = 0;
  A2C_TRY(clear_counts(c, w));
  if (N > 0) A2C_TRY(pass(w->tmp, nullptr, room));
  A2C_TRY(place_lists(c, w, ext));
  if (N > 0) {
    const int most = w->report->most;  // place_lists has refused more than kMaxPerSite
    const int64_t *off = ext ? c->d_ext_off : c->d_off;
    uint32_t *nbr = ext ? c->d_ext_nbr : c->d_nbr;
    const bool in_place = most > room || !w->tmp;
    if (in_place) A2C_TRY(pass(nbr, off, list_room(most)));
    if (!in_place || !ext) {
      k_pack<<<blocks, 32 * kListWarps, 0, st>>>(g, in_place ? off : nullptr, stride, in_place ? nbr : w->tmp, off, nbr,
                                                 c->d_hh1_off, ext ? nullptr : c->d_hh1, c->d_status);
      A2C_CUDA(cudaGetLastError());
    }
    if (most > stride && N * list_room(most) <= 2 * (int64_t)w->report->total) stride = list_room(most);
    if (ncell > cells_kept(N)) {
      cudaFree(w->cells);  // waits for the kernels that use it
      w->cells = nullptr;
      w->cells_cap = 0;
    }
  }
  return ext ? A2C_OK : lists_done(c, cut);
}

// The lists at rc from the extended lists (the skin path): the same lists,
// shells and first H shells as a build from cells, with one exact test per
// candidate (k_refilter keeps the survivors), over the scanned positions.
// A warp per site: 84 + 48 us at 92,160 sites, where one thread per site
// (scattered loads, every lane its own list) took 126 + 92.
a2c_status refilter_lists(a2c_gpp_ctx *c) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  GridArgs g;
  make_grid(c, nullptr, c->p.rc, g);  // only the cutoff and box are read on this path
  ListWork *w = (ListWork *)c->list_work;
  A2C_TRY(grow(c, &w->tmp, &w->tmp_cap, c->ext_total));
  g.Xf = w->Xf;
  g.qmax_bits = &w->scan->qmax_bits;
  A2C_TRY(clear_counts(c, w));
  const unsigned blocks = grid_for(N, kListWarps);
  if (N > 0) {
    k_refilter<<<blocks, 32 * kListWarps, 0, st>>>(g, c->d_ext_off, c->d_ext_nbr, w->tmp, w->count, c->d_npd, w->hh1c,
                                                   c->d_shell, w->most);
    A2C_CUDA(cudaGetLastError());
  }
  A2C_TRY(place_lists(c, w, false));
  if (!w->tmp && c->ext_total > 0) return A2C_ERR_NOMEM;
  if (N > 0) {
    k_pack<<<blocks, 32 * kListWarps, 0, st>>>(g, c->d_ext_off, 0, w->tmp, c->d_off, c->d_nbr, c->d_hh1_off, c->d_hh1,
                                               c->d_status);
    A2C_CUDA(cudaGetLastError());
  }
  return lists_done(c, c->p.rc);
}

}  // namespace

cudaError_t context_malloc(a2c_gpp_ctx *c, void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  ListWork *w = (ListWork *)c->list_work;
  if (e == cudaErrorMemoryAllocation && w && w->tmp) {
    cudaFree(w->tmp);  // waits for the kernels that use it
    w->tmp = nullptr;
    w->tmp_cap = 0;
    (void)cudaGetLastError();
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) (void)cudaGetLastError();  // reported here, not by the next launch's check
  return e;
}

void lists_free(a2c_gpp_ctx *c) {
  ListWork *w = (ListWork *)c->list_work;
  if (!w) return;
  for (void *p : {w->base, (void *)w->tmp, (void *)w->cells})
    if (p) cudaFree(p);
  delete w;
  c->list_work = nullptr;
}

a2c_status stage_positions(a2c_gpp_ctx *c, const double *X, const double *mX, PosScan *scan) {
  const int64_t N = c->N;
  cudaStream_t st = c->stream;
  ListWork *w;
  A2C_TRY(work_for(c, &w));
  if (N > 0 && !mX) A2C_CUDA(cudaMemcpyAsync(w->stage, X, sizeof(double) * 4 * N, cudaMemcpyHostToDevice, st));
  A2C_TRY(scan_positions(c, w, mX ? mX : w->stage, mX ? w->stage : nullptr, c->has_ext ? c->d_xref : nullptr, scan));
  if (scan->flags & kPosNonfinite) return A2C_ERR_NONFINITE;
  if (scan->flags & kPosOutside) return A2C_ERR_INVALID;
  if (N > 0) A2C_CUDA(cudaMemcpyAsync(c->d_X, w->stage, sizeof(double) * 4 * N, cudaMemcpyDeviceToDevice, st));
  return A2C_OK;
}

// The positions already in c->d_X, scanned for a build or update.
static a2c_status scan_device(a2c_gpp_ctx *c, PosScan *scan) {
  ListWork *w;
  A2C_TRY(work_for(c, &w));
  return scan_positions(c, w, nullptr, nullptr, c->has_ext ? c->d_xref : nullptr, scan);
}

a2c_status build_neighbors_device(a2c_gpp_ctx *c, const PosScan *scan) {
  PosScan own;
  if (!scan) {
    A2C_TRY(scan_device(c, &own));
    scan = &own;
  }
  c->has_ext = false;  // a full build invalidates the extended lists
  return lists_from_cells(c, *scan, c->p.rc, false);
}

// Skin path: rebuild the extended lists when a site has moved more than
// skin/2 since they were built (or none exist), then re-filter at rc.
// Positions are in c->d_X; scan: what stage_positions found of them (null:
// scanned here).
a2c_status update_neighbors_device(a2c_gpp_ctx *c, const PosScan *scan, int *rebuilt) {
  const int64_t N = c->N;
  PosScan own;
  if (!scan) {
    A2C_TRY(scan_device(c, &own));
    scan = &own;
  }
  const bool need = !c->has_ext || (scan->flags & kPosMoved);
  if (need) {
    c->has_ext = false;  // until the new ones stand: a failed build leaves offsets without their lists
    A2C_TRY(lists_from_cells(c, *scan, c->p.rc + c->skin, true));
    if (N > 0)
      A2C_CUDA(cudaMemcpyAsync(c->d_xref, c->d_X, sizeof(double) * 4 * N, cudaMemcpyDeviceToDevice, c->stream));
    c->has_ext = true;
  }
  if (rebuilt) *rebuilt = need ? 1 : 0;
  return refilter_lists(c);
}

}  // namespace a2c
