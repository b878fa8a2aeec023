// Planning pass of the 1C contractions: which quartets of a class pair survive
// the Schwarz x density screen, and in which precision they run.
#pragma once

#include <algorithm>

#include "cqf_internal.hpp"

namespace cqf {

// Shell-block norm maximum of a quartet in the reference's roles
// (direct.hpp:1693-1736), with the warp-uniform bra pair P: the pair norms
// come from the per-pair array, and the four cross terms are read from the
// column of a bra shell (normsT holds the transpose), so a warp's lanes read
// one column instead of 32 scattered ones.
__device__ __forceinline__ double sh_max_bra(const JKLaunch& a, const PairDev& P,
                                             const PairDev& Q, double nP, double nQ,
                                             bool pRef) {
  const int ns = a.nShell;
  double m;
  if (pRef) {  // rows from P (uniform): B(r, c) = normsT[c + r ns]
    const double* c1 = a.normsT + (size_t)P.s1 * ns;
    const double* c2 = a.normsT + (size_t)P.s2 * ns;
    m = fmax(fmax(__ldg(c1 + Q.s1), __ldg(c2 + Q.s1)), fmax(__ldg(c1 + Q.s2), __ldg(c2 + Q.s2)));
  } else {     // rows from Q, columns from P (uniform): B(r, c) = norms[r + c ns]
    const double* c1 = a.norms + (size_t)P.s1 * ns;
    const double* c2 = a.norms + (size_t)P.s2 * ns;
    m = fmax(fmax(__ldg(c1 + Q.s1), __ldg(c1 + Q.s2)), fmax(__ldg(c2 + Q.s1), __ldg(c2 + Q.s2)));
  }
  return fmax(m, fmax(nP, nQ));
}

// Planning pass of one class pair: for every (bra pair, tile of 32 kets) the
// quartets that survive the Schwarz x density screen, split by precision --
// mask.x: lanes computed in FP64, mask.y: lanes computed in FP32 (mixed
// builds: screening bound below the cut and inside the FP32 range guard).
// Quartet set, screens and counts are those of the reference's loop
// (direct.hpp:1642-1805); in the same class a ket sits at or before its bra
// (each unordered pair of pairs once).  The masks form one row-major
// sequence of words (bra pair, ket tile); a warp takes runs of 32
// consecutive words and appends the indices of its non-empty words to one
// list per precision (lengths in lcount[0 / 1]), so the class kernels visit
// only words that name quartets of their precision.
//
// CUT (launches whose class kernels share a quartet among lanes): a word whose
// quartets have long primitive loops (PLAN_LONG planEach primitive quartets or more)
// carries log2 of the lanes per quartet in its list entry, and is listed as
// eight entries of four kets, so that several warps share it: in the first
// eighth of the words -- pairs come in descending order of their primitive
// counts -- so that the lists hold at most twice the words, or anywhere
// (planAll) where they have room for eight times the words.  Without it one
// lane walked the 4096 primitive quartets of two contractions of eight: 1.4 ms
// of a 2.3 ms build of one water molecule.
constexpr int PLAN_RUN = 32;
constexpr int PLAN_LONG = 4;
constexpr int PLAN_WORD = (1 << 20) - 1;  // list entry: word | sub << 20 | part << 23 | log2 << 24
// Two forms (times: J and K, FP64 unless named).
// * Angular sums up to 2 in launches of up to JK_CUT_WORDS, 14 words for each of
//   the 4736 warps that are resident at eight blocks an SM; 64 primitive
//   quartets a lane.  Without it 6 waters in cc-pVDZ take 3.11 ms for 1.72, up
//   to 2^13 words 2.78; up to 2^18 12 waters would gain (5.98 -> 4.28 ms) and
//   from 16 on nothing changes.  32 a lane: 6 waters in 6-31G(d) 1.11 -> 1.04
//   ms, 4 in cc-pVDZ 1.33 -> 1.46; 128: 1.20 and 1.25.
// * Angular sums up to 4 in launches of up to JK_TINY_WORDS, three words an SM
//   and what the smallest region holds eightfold (JK_MIN_WORDS; JK_TINY_BYTES
//   a word); 8 primitive quartets a lane.  Without it one water in def2-SVP
//   takes 0.60 ms for 0.51 and 2 in 6-31G(d) mixed 1.09 for 0.90; up to one word
//   an SM the latter take 0.98.  4 a lane 2-12% slower, 32 up to 9% slower
//   (def2-SVP) or 6% faster (one water in cc-pVDZ).
// Larger launches have enough quartets to hide the longest loops, and the
// shared form costs registers ((H2O)16 / def2-SVP mixed 6.15 -> 6.45 ms where
// every class pair takes it).  So the host takes it only where the class pair's
// longest contractions reach PLAN_LONG planEach (with it for every small launch
// 6 waters in 3-21G 262 -> 310 us, 10 in def2-SVP 2.15 -> 2.29 ms).
__host__ __device__ constexpr bool jk_split(int lsum) { return lsum <= 4; }
constexpr long long JK_CUT_WORDS = 1 << 16;
constexpr long long JK_TINY_WORDS = 448;
constexpr int JK_CUT_LSUM = 2, JK_TINY_BYTES = 8 + 2 * 8 * 4;  // per word, both lists eightfold
template <bool MIXED, bool CUT>
__global__ void __launch_bounds__(256)
    jk_plan_kernel(const JKLaunch a, uint2* __restrict__ masks, int* __restrict__ list64,
                   int* __restrict__ list32, unsigned int* __restrict__ lcount) {
  const int lane = threadIdx.x & 31;
  const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)((gridDim.x * blockDim.x) >> 5);
  const int nTiles = (a.nKet + WTILE - 1) / WTILE;
  const int nWords = a.nBra * nTiles;
  const int nRuns = (nWords + PLAN_RUN - 1) / PLAN_RUN;
  const double cut = MIXED ? a.fp32_cut : 0.0;
  unsigned long long cVis = 0, cScr = 0, c32 = 0, c64 = 0;
  for (int run = gw; run < nRuns; run += nw) {
    int my64 = -1, my32 = -1, n64 = 0, n32 = 0;
    const int wEnd = min((run + 1) * PLAN_RUN, nWords);
    for (int word = run * PLAN_RUN; word < wEnd; word++) {
      const int ib = word / nTiles, tile = word - ib * nTiles;
      unsigned b64 = 0u, b32 = 0u;
      int sl = 0;  // log2 of the lanes per quartet
      const int ibc = ib + a.braOff;  // the bra's position in its class
      // else: no quartet in this word (above the diagonal, or another shard's bra)
      if (!(a.same && tile * WTILE > ibc) && in_shard(a.braBeg + ib, a.shardIdx, a.shardCnt)) {
        const int jk = tile * WTILE + lane;
        const PairDev P = a.pairs[a.braBeg + ib];
        const bool visited = jk < a.nKet && !(a.same && jk > ibc);
        const double tileMax = __ldg(a.maxNorm) * P.Q * __ldg(a.qWin + a.ketBeg + tile * WTILE);
        bool screened = false, w32 = false;
        auto share = [&](int ketPrim) {
          const int np = P.npp * ketPrim;
          while (np >= PLAN_LONG * a.planEach && sl < 5 && (np >> sl) > a.planEach) sl++;
        };
        if (a.screen && tileMax < a.thresh) {
          screened = true;
        } else if (visited && a.screen) {
          const PairDev Q = a.pairs[a.ketBeg + jk];
          const bool pRef = P.lex >= Q.lex;
          const double bound = sh_max_bra(a, P, Q, __ldg(a.pairNorm + a.braBeg + ib),
                                          __ldg(a.pairNorm + a.ketBeg + jk), pRef) * P.Q * Q.Q;
          screened = bound < a.thresh;
          if (CUT && !screened) share(Q.npp);
          w32 = MIXED && !screened && bound < cut &&
                fp32_range_ok(__ldg(a.pairRange + a.braBeg + ib),
                              __ldg(a.pairRange + a.ketBeg + jk), a.lsum, 0, 0);
        } else if (CUT && visited) {  // 4 waters unscreened 2.65 -> 1.32 ms
          share(a.pairs[a.ketBeg + jk].npp);
        }  // without the screen every quartet runs in FP64
        const unsigned bv = __ballot_sync(0xffffffffu, visited);
        const unsigned bs = __ballot_sync(0xffffffffu, visited && screened);
        b32 = __ballot_sync(0xffffffffu, visited && !screened && w32);
        b64 = bv & ~bs & ~b32;
        cVis += __popc(bv);
        cScr += __popc(bs);
        c32 += __popc(b32);
        c64 += __popc(b64);
      }
      if (lane == 0) masks[word] = make_uint2(b64, b32);
      int entry = word;
      if (CUT) {
        sl = (int)__reduce_max_sync(0xffffffffu, (unsigned)sl);
        entry |= sl << 24;
        if (sl > 1 && (a.planAll || word < nWords / 8)) {  // eight entries, written here
          const unsigned s64 = b64 >> (4 * (lane & 7)) & 15u, s32 = b32 >> (4 * (lane & 7)) & 15u;
          unsigned at = 0;
          if (lane < 8 ? s64 != 0u : (lane < 16 && s32 != 0u))
            at = atomicAdd(lcount + (lane < 8 ? 0 : 1), 1u);
          const int e8 = entry | 1 << 23 | (lane & 7) << 20;
          if (lane < 8) {
            if (s64) list64[at] = e8;
          } else if (lane < 16) {
            if (s32) list32[at] = e8;
          }
          continue;
        }
      }
      if (b64) {
        if (lane == n64) my64 = entry;
        n64++;
      }
      if (b32) {
        if (lane == n32) my32 = entry;
        n32++;
      }
    }
    unsigned int base64 = 0, base32 = 0;
    if (lane == 0) {
      if (n64) base64 = atomicAdd(lcount + 0, (unsigned)n64);
      if (n32) base32 = atomicAdd(lcount + 1, (unsigned)n32);
    }
    base64 = __shfl_sync(0xffffffffu, base64, 0);
    base32 = __shfl_sync(0xffffffffu, base32, 0);
    if (lane < n64) list64[base64 + lane] = my64;
    if (lane < n32) list32[base32 + lane] = my32;
  }
  if (lane == 0) {
    if (cVis) atomicAdd(a.counters + 0, cVis);
    if (cScr) atomicAdd(a.counters + 1, cScr);
    if (c32) atomicAdd(a.counters + 2, c32);
    if (c64) atomicAdd(a.counters + 3, c64);
  }
}

// Launches the pass on the bra pairs [braBeg, braBeg + nBra) of `a` (a slab):
// lcount[0 / 1], zero on entry, receive the lists' lengths.
inline void launch_jk_plan(const JKLaunch& a, bool mixed, bool cut, uint2* masks, int* list64,
                           int* list32, unsigned int* lcount, int nsm, cudaStream_t st) {
  const long long nWords = (long long)a.nBra * ((a.nKet + WTILE - 1) / WTILE);
  const long long nRuns = (nWords + PLAN_RUN - 1) / PLAN_RUN;
  const unsigned gp = (unsigned)std::min<long long>((nRuns + 7) / 8, (long long)nsm * 8);
  if (mixed && cut)
    jk_plan_kernel<true, true><<<gp, 256, 0, st>>>(a, masks, list64, list32, lcount);
  else if (mixed)
    jk_plan_kernel<true, false><<<gp, 256, 0, st>>>(a, masks, list64, list32, lcount);
  else if (cut)
    jk_plan_kernel<false, true><<<gp, 256, 0, st>>>(a, masks, list64, list32, lcount);
  else
    jk_plan_kernel<false, false><<<gp, 256, 0, st>>>(a, masks, list64, list32, lcount);
}

}  // namespace cqf
