// Items of the Hermite-matrix engine's contracted classes (cqf_hgemm.cuh): how
// many mask words a slab takes in a launch stream's region, and into how many
// parts an entry of its word lists is cut.
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define CQF_HD __host__ __device__
#else
#define CQF_HD
#endif

namespace cqf {

// A slab of up to `words` words in a region of `room` 8-byte units: per word
// its mask, its entries of the two lists (4 B each) and `most` items of 8 B.
// most = 0: the words are not cut.
struct HgSlab {
  int most;
  long long words;
};
// As many items per word as leave the nBra x nTiles words of a launch in one
// slab, but at least 16 (and never more than a row of words leaves room for)
inline HgSlab hg_slab(long long room, int nBra, int nTiles) {
  const long long row = room / nTiles - 2;
  const int most = (int)std::min(
      std::min(255LL, row), std::max(16LL, room / ((long long)nBra * nTiles) - 2));
  return {most > 1 ? most : 0, most > 1 ? room / (2 + most) : room / 2};
}

// A list entry's parts: the bra's primitives in cb ranges, the kets'
// (concatenated) in ck ones.
struct HgCut {
  int cb, ck;
};
// np: the bra's primitives; nk: those of the entry's kets, other: those of the
// word's kets in the other list; work: primitive quartets of a part.  A word
// with FP64 and FP32 quartets is an entry of both lists, which share its
// `most` >= 2 items as their kets' primitives do: floor(most nk / (nk +
// other)), at least 1, sums to `most` at most.
CQF_HD inline HgCut hg_cut(int np, int nk, int other, int work, int most) {
  const int share =
      other ? (int)((long long)most * nk / ((long long)nk + other)) : most;
  const long long want = ((long long)np * nk + work - 1) / work;
  const int n = want < share ? (int)want : share;
  // the bra's primitives first: a batch holds ket primitives of one of them
  HgCut c;
  c.cb = np < n ? np : n;
  c.cb = c.cb < 1 ? 1 : c.cb;
  c.ck = n / c.cb;
  c.ck = c.ck > nk ? nk : c.ck;
  c.ck = c.ck < 1 ? 1 : c.ck;
  return c;
}

}  // namespace cqf
