// The item lists of the Hermite-matrix engine on random launches: for every
// slab of a class pair, random masks (quartets in FP64, FP32, both or neither)
// and contraction lengths, the parts of both lists must fit in what the slab's
// masks and lists leave of the region, and cover each entry's primitive
// quartets once.  Prints the launches checked; exits 1 at the first fault.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../../chronusq_public_b200/csrc/cqf_hg_items.hpp"

using namespace cqf;

int main(int argc, char** argv) {
  const int draws = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 g(11);
  auto uni = [&](long long lo, long long hi) {  // over the logarithm
    const double u = std::uniform_real_distribution<>(0, 1)(g);
    return (long long)(lo * std::exp(u * std::log((hi + 1.0) / lo)));
  };
  for (int d = 0; d < draws; d++) {
    const int nBra = (int)uni(1, 300), nKet = (int)uni(1, 3000), nTiles = (nKet + 31) / 32;
    // a region holds at least one bra pair's row of words
    const long long maskWords = std::max<long long>(nTiles, uni(1, 40000));
    const long long room = 2 * maskWords;
    const int top = (int)uni(1, 200), work = (int)uni(1, 1024), mode = (int)uni(1, 5) - 1;
    std::vector<int> npk(nKet);
    for (int& n : npk) n = (int)uni(1, top);
    const HgSlab s = hg_slab(room, nBra, nTiles);
    if (s.words < nTiles) {
      std::printf("no row of words: draw %d\n", d);
      return 1;
    }
    const int slab = (int)std::max<long long>(1, s.words / nTiles);
    for (int ib0 = 0; ib0 < nBra; ib0 += slab) {
      const int n = std::min(slab, nBra - ib0);
      const long long nWords = (long long)n * nTiles;
      if (2 * nWords > room) {
        std::printf("masks and lists past the region: draw %d\n", d);
        return 1;
      }
      if (!s.most) continue;
      long long items = 0;
      for (long long w = 0; w < nWords; w++) {
        const int np = (int)uni(1, top);
        // FP64 only, FP32 only, an even mixture, or one quartet against 31
        uint32_t any = (uint32_t)g(), lo = (uint32_t)g();
        if (nKet % 32 && w % nTiles == nTiles - 1) any &= (1u << nKet % 32) - 1;
        const uint32_t m32 = any & (mode == 0 ? 0u : mode == 1 ? ~0u : mode == 2 ? lo : lo & -lo);
        const uint32_t m[2] = {any & ~m32, m32};
        int k[2] = {0, 0};
        for (int q = 0; q < 32 && w % nTiles * 32 + q < nKet; q++)
          for (int l = 0; l < 2; l++)
            if (m[l] >> q & 1) k[l] += npk[w % nTiles * 32 + q];
        long long mine = 0;
        for (int l = 0; l < 2; l++) {
          if (!m[l]) continue;
          const HgCut c = hg_cut(np, k[l], k[1 - l], work, s.most);
          // every part has at least one primitive on both sides, packed in 8 bits
          if (c.cb < 1 || c.ck < 1 || c.cb > std::min(np, 255) || c.ck > std::min(k[l], 255)) {
            std::printf("empty or unpackable part: draw %d\n", d);
            return 1;
          }
          mine += (long long)c.cb * c.ck;
        }
        items += mine;
        if (mine > s.most || items > room - 2 * nWords) {
          std::printf("draw %d: %lld items of a word (most %d), %lld in room for %lld\n", d, mine,
                      s.most, items, room - 2 * nWords);
          return 1;
        }
      }
    }
  }
  std::printf("%d launches\n", draws);
  return 0;
}
