// Tile shape of the mixed pair kernels (k_mixed.cu) and the library's choice
// of it.  Plain C++: tests/cpp/tile_check.cpp checks the rule on the host.
#pragma once

#include <cstdint>
#include <functional>

#include "a2c_gpp.h"

namespace a2c {

// Threads per site (1, 2, 4, 8) and threads per block of pass 1 (256, 512,
// 768) and pass 2 (128, 256, 512); 0 = the library's choice.  The rest
// follows from them and the size (effective_tile).
struct Tile {
  int tps = 0, rho_block = 0, grad_block = 0;
  bool own = false;                 // both block sizes are the library's choice
  bool wide = false, twin = false;  // a warp, or two lanes, for a site's tps lanes
  bool copies = false;              // pass 2 with eight copies of its tables
  bool operator==(const Tile &o) const {
    return tps == o.tps && rho_block == o.rho_block && grad_block == o.grad_block && own == o.own && wide == o.wide &&
           twin == o.twin && copies == o.copies;
  }
};
inline bool valid_tile(int tps, int rho_block, int grad_block) {
  return (tps == 0 || tps == 1 || tps == 2 || tps == 4 || tps == 8) &&
         (rho_block == 0 || rho_block == 256 || rho_block == 512 || rho_block == 768) &&
         (grad_block == 0 || grad_block == 128 || grad_block == 256 || grad_block == 512);
}

// Threads per site of the mixed pair kernels when none was chosen: a
// system with fewer than 2048 sites per SM spreads each site over 4 lanes
// so that every SM gets work; a larger one runs one lane per site.
inline int default_threads_per_site(int64_t n_sites, int sms) { return n_sites < (int64_t)sms * 2048 ? 4 : 1; }

// The tile that runs for a chosen one (zeros: the library's choice) on a
// whole system or (list) on a batch's or minimization's site lists.  A tile
// that this function gave, or its three numbers, gives the same tile again:
// block sizes named explicitly count as the library's choice where they are.
inline Tile effective_tile(const Tile &t, int64_t n_sites, int sms, bool list = false) {
  constexpr int kPlain = 256;
  Tile e;
  e.tps = t.tps ? t.tps : default_threads_per_site(n_sites, sms);
  // Block sizes when none was chosen (they change no result).  Pass 1: two
  // blocks fit an SM whatever their size, so 512 threads double its warps
  // (262,144 sites at 4 threads per site: 178 -> 141 us; 33,592: 31 -> 27;
  // 512: 15.4 either way), except with one thread per site (373,248 sites:
  // 233 us at 256, 266 at 512).  Pass 2: 128 threads while there are few
  // blocks to spread (512 sites: 27 against 29 us, 33,592: 54 against 56;
  // 92,160: 115 against 113).
  const int rho = e.tps > 1 ? 512 : kPlain, grad = n_sites < 256 * (int64_t)sms ? 128 : kPlain;
  e.rho_block = t.rho_block ? t.rho_block : rho;
  e.grad_block = t.grad_block ? t.grad_block : grad;
  e.own = e.rho_block == rho && e.grad_block == grad;
  // More lanes per site than its sums' order asks for, at the library's
  // block sizes: a warp for a site while there are few (passes 1 and 2 with
  // 4 / 32 lanes, 512 sites: 16.4 + 26.8 / 8.1 + 18.9 us, 4,096: 16.4 + 26.8
  // / 14.3 + 25.2, 8,000: 16.4 + 29.3 / 19.8 + 37.1), two lanes in place of
  // one (512,000 sites: 315 + 614 / 303 + 580 us, 2,097,152: 1215 + 2559 /
  // 1131 + 2399).
  e.wide = e.own && n_sites <= 27 * (int64_t)sms;
  e.twin = e.own && !e.wide && e.tps == 1;
  // Pass 2's shape of 256 threads (or the library's) has eight copies of
  // f_Pd' under one block of 1024 threads per SM where its warps come near
  // 32 per SM (pass 2 without / with them, 2 threads per site: 33,592 sites
  // 59 / 83 us, 92,160: 125 / 109, 262,144: 293 / 266; 4 threads: 21,952:
  // 45 / 51, 33,592: 58 / 53, 2,097,152: 2,076 / 1,891; two lanes for one:
  // 33,592: 76 / 96, 92,160: 156 / 123).  Lists keep the library's 128-thread
  // blocks where it chooses those: a batch of five lattices with 33,144 sites
  // takes 2,658 us without, 2,740 with them; 30 iterations of one
  // minimization 6.06 / 6.14 ms at 30,720 sites, 6.65 / 6.38 at 38,880.
  e.copies = !e.wide && (e.grad_block == kPlain || (e.grad_block == grad && !list)) &&
             n_sites * (e.twin ? 2 : e.tps) >= 25 * 32 * (int64_t)sms;
  return e;
}

// The tile tuner: threads per site at 256-thread blocks, then the pass-1
// block size, then the pass-2 block size, each stage keeping the fastest;
// time_tile(tile, &ms) measures one candidate.  ms[10] receives these
// candidates' times in that order (may be null).  Then the library's own
// blocks, at its and at the fastest's threads per site, which the stages may
// have passed by: a tuned system is never slower than an untuned one.  The
// result is resolved (effective_tile).
constexpr int kTileCandidates = 10;
inline a2c_status tune_tile(const std::function<a2c_status(const Tile &, float *)> &time_tile, int64_t n_sites, int sms,
                            bool list, Tile *best, float *ms) {
  Tile b{0, 256, 256};
  float best_ms = 0.0f;
  int k = 0;
  auto trial = [&](const Tile &t) -> a2c_status {
    float v = 0.0f;
    const a2c_status s = time_tile(t, &v);
    if (s != A2C_OK) return s;
    if (ms && k < kTileCandidates) ms[k] = v;
    ++k;
    if (b.tps == 0 || v < best_ms) {
      best_ms = v;
      b = t;
    }
    return A2C_OK;
  };
  a2c_status s = A2C_OK;
  for (int q : {1, 2, 4, 8})
    if (!s) s = trial(Tile{q, 256, 256});
  const Tile after_tps = b;
  for (int q : {256, 512, 768})
    if (!s) s = trial(Tile{after_tps.tps, q, after_tps.grad_block});
  const Tile after_rho = b;
  for (int q : {128, 256, 512})
    if (!s) s = trial(Tile{after_rho.tps, after_rho.rho_block, q});
  const Tile own = effective_tile(Tile{}, n_sites, sms, list), same = effective_tile(Tile{b.tps, 0, 0}, n_sites, sms, list);
  if (!s) s = trial(own);
  if (!s && !(same == own)) s = trial(same);
  if (!s) *best = effective_tile(b, n_sites, sms, list);
  return s;
}

}  // namespace a2c
