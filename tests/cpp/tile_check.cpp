// Checks the tile rule (tile.h) on the host over every valid tile and sizes
// around every threshold: the tile that runs, given again as a tile or as
// its three numbers, runs again; the library's choice is one of the tiles
// that can be named; a warp or two lanes per site are taken where the
// library chose the blocks, and only there; and the tuner with made-up
// times: never slower than the library's own tile.  argv: SMs.  Prints the tiles
// checked and how many ran with a warp, two lanes and table copies.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "tile.h"

using namespace a2c;

int main(int argc, char **argv) {
  if (argc < 2) return 2;
  const int sms = std::atoi(argv[1]);
  std::vector<int64_t> sizes;
  for (int64_t at : {1, 27, 100, 108, 200, 216, 256, 400, 432, 800, 864, 2048, 13797})  // sites per SM: the thresholds
    for (int64_t d : {-1, 0, 1}) sizes.push_back(at * sms + d);
  long n = 0, wide = 0, twin = 0, copies = 0;
  auto check = [&](int64_t N, bool list) {
    for (int tps : {0, 1, 2, 4, 8})
      for (int rho : {0, 256, 512, 768})
        for (int grad : {0, 128, 256, 512}) {
          const Tile r = effective_tile(Tile{tps, rho, grad}, N, sms, list);
          ++n;
          wide += r.wide;
          twin += r.twin;
          copies += r.copies;
          if (!valid_tile(r.tps, r.rho_block, r.grad_block) || !r.tps || !r.rho_block || !r.grad_block) return 3;
          if (!(effective_tile(r, N, sms, list) == r)) return 4;
          if (!(effective_tile(Tile{r.tps, r.rho_block, r.grad_block}, N, sms, list) == r)) return 5;
          const Tile lib = effective_tile(Tile{r.tps, 0, 0}, N, sms, list);
          const bool own = r.rho_block == lib.rho_block && r.grad_block == lib.grad_block;
          if (own ? !(r == lib) : (r.wide || r.twin)) return 6;
          if (lib.wide != (N <= 27 * (int64_t)sms) || lib.twin != (!lib.wide && lib.tps == 1)) return 7;
        }
    return 0;
  };
  for (int64_t N : sizes)
    for (bool list : {false, true})
      if (const int bad = check(N, list)) return bad;
  // The tuner over made-up times: whatever tile is fastest among those it
  // times, and a system's own tile if that is faster still.
  for (int64_t N : sizes)
    for (int seed = 0; seed < 50; ++seed) {
      const Tile own = effective_tile(Tile{}, N, sms);
      auto cost = [&](const Tile &t) {
        const Tile r = effective_tile(t, N, sms);
        if (r == own) return seed % 2 ? 0.25f : 0.75f;
        unsigned h = (unsigned)(seed * 7919 + r.tps * 131 + r.rho_block * 17 + r.grad_block);
        h = (h ^ h >> 13) * 2654435761u;
        return 0.3f + (float)(h >> 8) / (float)(1 << 24);
      };
      int calls = 0;
      float least = 1e9f, ms[kTileCandidates];
      Tile best;
      const a2c_status s = tune_tile(
          [&](const Tile &t, float *v) {
            ++calls;
            *v = cost(t);
            if (*v < least) least = *v;
            return A2C_OK;
          },
          N, sms, false, &best, ms);
      if (s != A2C_OK || calls < kTileCandidates + 1 || calls > kTileCandidates + 2) return 8;
      if (cost(best) != least || least > cost(own) || !(effective_tile(best, N, sms) == best)) return 9;
    }
  std::printf("%ld %ld %ld %ld\n", n, wide, twin, copies);
  return 0;
}
