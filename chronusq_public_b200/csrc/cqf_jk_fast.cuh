// Closed-shell fast path: real densities flagged Hermitian (symmetric), every
// shell l <= 2.  One thread per unique quartet, generated straight-line
// McMurchie-Davidson code per class and precision (gen/cqf_gen_jk.cuh): a
// planning pass names each quartet's precision, then an FP64 and (mixed
// builds) an FP32 kernel per class compute their quartets; FP64
// accumulation.
//
// Screening, unique-quartet set and degeneracy are those of the generic
// kernel (cqf_jk_kernels.cuh); the digestion uses the canonical quartet order
// instead of the reference's shell roles, which gives the same J and K after
// the final 1/2 (A + A^T) when X is symmetric.
#pragma once

#include "cqf_jk_kernels.cuh"
#include "cqf_jk_plan.cuh"
#include "gen/cqf_gen_jk.cuh"

#include <algorithm>
#include <type_traits>

namespace cqf {

static_assert(JK_THREADS == KETT_TILE, "a ket tile is one block of kets");

template <typename T, int N>
__device__ __forceinline__ void warp_sum(T (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  }
}

// Ket primitive-pair data of one quartet for the generated eri():
// KetAoS reads the PrimPairDev records of the pair (any pair order);
// KetSoA reads the tile-interleaved copy, where the 128 kets of a tile have
// each field of primitive iq contiguous (a warp's load is one coalesced run).
struct KetAoS {
  const PrimPairDev* b;
  const double* q;  // primitive Schwarz bounds of the same pairs (read only when screening)
  __device__ __forceinline__ double Qp(int iq) const { return q[iq]; }
  __device__ __forceinline__ double p(int iq) const { return b[iq].p; }
  __device__ __forceinline__ double Kp(int iq) const { return b[iq].Kp; }
  __device__ __forceinline__ double o2p(int iq) const { return b[iq].o2p; }
  __device__ __forceinline__ double P(int iq, int x) const { return b[iq].P[x]; }
  __device__ __forceinline__ double PA(int iq, int x) const { return b[iq].PA[x]; }
  __device__ __forceinline__ double PB(int iq, int x) const { return b[iq].PB[x]; }
};
template <typename E>  // element type: double, or float for the FP32 copy
struct KetSoAT {
  const E* q;  // tile base + lane
  __device__ __forceinline__ E f(int iq, int k) const {
    return __ldg(q + (iq * KETT_NF + k) * KETT_TILE);
  }
  __device__ __forceinline__ E p(int iq) const { return f(iq, 0); }
  __device__ __forceinline__ E Kp(int iq) const { return f(iq, 1); }
  __device__ __forceinline__ E o2p(int iq) const { return f(iq, 2); }
  __device__ __forceinline__ E P(int iq, int x) const { return f(iq, 3 + x); }
  __device__ __forceinline__ E PA(int iq, int x) const { return f(iq, 6 + x); }
  __device__ __forceinline__ E PB(int iq, int x) const { return f(iq, 9 + x); }
  __device__ __forceinline__ double Qp(int iq) const { return (double)f(iq, 12); }
};
using KetSoA = KetSoAT<double>;

// Rows of the Boys tables for angular sum L (global memory).
template <typename T>
__device__ __forceinline__ const T* boys_rows(const JKLaunch& a, int L);
template <>
__device__ __forceinline__ const double* boys_rows<double>(const JKLaunch& a, int L) {
  return a.boys64 + (size_t)L * BOYS_NPTS * BOYS_ROW64;
}
template <>
__device__ __forceinline__ const float* boys_rows<float>(const JKLaunch& a, int L) {
  return a.boys32 + (size_t)L * BOYS_NPTS * BOYS_ROW32;
}


// Position of the n-th (0-based) set bit of m (n < popc(m)).
__device__ __forceinline__ int nth_set_bit(unsigned m, int n) {
  int pos = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const unsigned lo = m & ((1u << w) - 1u);
    const int c = __popc(lo);
    if (n >= c) {
      n -= c;
      m >>= w;
      pos += w;
    } else {
      m = lo;
    }
  }
  return pos;
}

// Class kernel of one shell-quartet class in one precision (G = GenJK64_x
// or GenJK32_x; FP32 = which mask half and word list it uses).  A work item
// is (run of consecutive entries of the precision's word list -- sized from
// the list's length, at most entriesPerItem -- ket component chunk), handed
// out by a device counter.  A warp walks
// its run's words and packs the quartets they name into batches of 32 lanes
// (nth_set_bit), so every lane of a batch computes a surviving quartet; a
// batch may span two bra pairs.  The batch's integrals of the chunk come
// from generated straight-line McMurchie-Davidson code and are digested per
// density: J_ab warp-reduced when the batch has one bra pair (per lane
// otherwise), J_cd and the four exchange blocks with FP64 atomics.  The FP32
// kernel forms integrals and products in FP32 from the FP32 copy of the
// Cartesian densities; accumulation is FP64 in both.
template <class G, bool FP32, bool SPLIT>
__global__ void __launch_bounds__(JK_THREADS, G::MINB)
    jk_class_kernel(const JKLaunch a, const uint2* __restrict__ masks,
                    const int* __restrict__ list, const unsigned int* __restrict__ lcount,
                    int entriesPerItem, unsigned int* __restrict__ counter) {
  using T = typename G::T;
  constexpr int NA = ncart(G::LA), NB = ncart(G::LB);
  constexpr int NCH = G::NCHUNK;
  constexpr int LSUM = G::LA + G::LB + G::LC + G::LD;
  const T* boys = boys_rows<T>(a, LSUM);
  const T* Xbase = FP32 ? reinterpret_cast<const T*>(a.Xc32) : reinterpret_cast<const T*>(a.Xc);
  const int lane = threadIdx.x & 31;
  const int nTiles = (a.nKet + WTILE - 1) / WTILE;
  const int nEntries = (int)*lcount;  // written by the planning pass
  // entries per item from the list's actual length: about four items per
  // warp of the grid, at most entriesPerItem entries
  const int gridWarps = (int)(gridDim.x * (blockDim.x / 32));
  const int epi = max(1, min(entriesPerItem, (int)((long long)nEntries * NCH /
                                                   (4LL * gridWarps))));
  const int nItems = (nEntries + epi - 1) / epi * NCH;
  const size_t nc = a.ncart;
  const size_t matStride = (size_t)a.ncart * a.ncart;
  // primitive screen threshold: libint's engine precision as the reference
  // sets it, max(eps_double, tau / (max shell-block norm x K^4)), K the
  // largest contraction length (direct.hpp:1563-1589)
  const double peps =
      a.screen ? fmax(2.220446049250313e-16, a.thresh / (__ldg(a.maxNorm) * a.primK4)) : 0.0;
  // SPLIT: lanes per quartet, 2^sl, named by the list entries (jk_plan_kernel)
  int esl = 0;  // of the entry last read
  // entry e of the list: (word index, this precision's mask of it)
  auto entry = [&](int e) {
    const int raw = __ldg(list + e);
    const int w = SPLIT ? raw & PLAN_WORD : raw;
    unsigned m = FP32 ? __ldg(&masks[w].y) : __ldg(&masks[w].x);
    if constexpr (SPLIT) {
      esl = raw >> 24;
      if (raw & (1 << 23)) m &= 15u << (raw >> 20 & 7) * 4;
    }
    return make_int2(w, (int)m);
  };

  for (;;) {
    unsigned int itemU = 0;
    if (lane == 0) itemU = atomicAdd(counter, 1u);
    const int item = (int)__shfl_sync(0xffffffffu, itemU, 0);
    if (item >= nItems) break;
    const int run = item / NCH, ch = item - run * NCH;
    int e = run * epi;
    const int eEnd = min(e + epi, nEntries);
    int2 wm = entry(e);
    unsigned m = (unsigned)wm.y;
    for (;;) {
      // pack the next (up to) 32 named quartets of the run into the lanes, or
      // 32 / 2^sl of entries whose quartets are shared by 2^sl lanes
      int fill = 0, myW = -1, myBit = 0;
      const int sl = SPLIT ? esl : 0, cap = 32 >> sl;
      while (fill < cap && e < eEnd && (!SPLIT || esl == sl)) {
        const int c = __popc(m);
        const int take = min(c, cap - fill);
        const int r = (lane >> sl) - fill;
        if (r >= 0 && r < take) {
          myW = wm.x;
          myBit = nth_set_bit(m, r);
        }
        fill += take;
        if (take == c) {
          if (++e < eEnd) {
            wm = entry(e);
            m = (unsigned)wm.y;
          }
        } else {
          m &= ~((2u << nth_set_bit(m, take - 1)) - 1u);  // drop the bits taken
        }
      }
      if (fill == 0) break;
      const bool work_ = myW >= 0;
      // lane 0 always holds a quartet; idle lanes take its bra pair
      const int w0 = __shfl_sync(0xffffffffu, myW, 0);
      const int wl = work_ ? myW : w0;
      const int ib = wl / nTiles;
      const int jk = (wl - ib * nTiles) * WTILE + myBit;
      const bool oneBra = __all_sync(0xffffffffu, ib == w0 / nTiles);
      const PairDev P = a.pairs[a.braBeg + ib];
      PairDev Q{};  // idle lanes: npp = 0, no primitive loop
      if (work_) Q = a.pairs[a.ketBeg + jk];
      const bool pRef = P.lex >= Q.lex;
      const int s1 = pRef ? P.s1 : Q.s1, s2 = pRef ? P.s2 : Q.s2;
      const int s3 = pRef ? Q.s1 : P.s1, s4 = pRef ? Q.s2 : P.s2;
      const T deg = T(((s1 == s2) ? 1 : 2) * ((s3 == s4) ? 1 : 2) *
                      ((s1 == s3 && s2 == s4) ? 1 : 2));
      const T sJ = work_ ? T(0.5) * deg : T(0), sK = work_ ? T(0.25) * deg : T(0);
      const int jkc = work_ ? jk : 0;
      const long long ko = __ldg(a.tileOff + a.ketTileBeg + jkc / KETT_TILE) + jkc % KETT_TILE;
      T I[G::NI];
      if constexpr (FP32)  // FP32 copies of the pair data: half the load bytes
        G::eri(P, Q, a.pp32, KetSoAT<float>{a.ketT32 + ko}, boys, ch, I, a.ppQ, peps,
               lane & ((1 << sl) - 1), 1 << sl);
      else
        G::eri(P, Q, a.pp, KetSoA{a.ketT + ko}, boys, ch, I, a.ppQ, peps,
               lane & ((1 << sl) - 1), 1 << sl);
      bool mine = work_;  // this lane digests its quartet
      if constexpr (SPLIT) {
        if (sl > 0) {
#pragma unroll
          for (int i = 0; i < G::NI; i++)
            for (int o = (1 << sl) >> 1; o > 0; o >>= 1)
              I[i] += __shfl_xor_sync(0xffffffffu, I[i], o);
          mine = work_ && (lane & ((1 << sl) - 1)) == 0;
        }
      }
#pragma unroll 1
      for (int mt = 0; mt < a.nMat; mt++) {
        const int fl = __ldg(a.flags + mt);
        const bool doJ = !(fl & 2), doK = (fl & 2);
        T jab[NA * NB];
#pragma unroll
        for (int i = 0; i < NA * NB; i++) jab[i] = T(0);
        double* A = a.Ac + mt * matStride;
        G::digest(I, ch, Xbase + mt * matStride, A, nc, P.cA, P.cB, Q.cA, Q.cB, sJ, sK,
                  (fl & 4) ? -sK : sK, doJ && mine, doK && mine, jab);
        if (doJ) {
#pragma unroll
          for (int i = 0; i < NA * NB; i++) jab[i] *= sJ;
          if (oneBra) {  // the lanes share the bra pair: reduce, one atomic each
            warp_sum(jab);
            if (lane == 0) {
#pragma unroll
              for (int i = 0; i < NA * NB; i++)
                if (jab[i] != T(0))
                  atomicAdd(A + (size_t)(P.cA + i / NB) + (size_t)(P.cB + i % NB) * nc,
                            double(jab[i]));
            }
          } else if (mine) {
#pragma unroll
            for (int i = 0; i < NA * NB; i++)
              if (jab[i] != T(0))
                atomicAdd(A + (size_t)(P.cA + i / NB) + (size_t)(P.cB + i % NB) * nc,
                          double(jab[i]));
          }
        }
      }
    }
  }
}

// Upper limit of word-list entries per work item of a class kernel (the
// kernel sizes its items from the list's actual length).
inline int entries_per_item(long long nWords, int nchunk, int nsm) {
  const long long per = nWords * nchunk / ((long long)nsm * 256);
  return (int)std::min<long long>(64, std::max<long long>(1, per));
}

// Launches the planning pass and the generated class kernels of the class
// (la lb | lc ld) (either orientation); false when the class has no
// generated kernel.  masks: the launch stream's region of maskWords uint2
// (mask words of a slab of bra pairs x ceil(nKet / 32) ket tiles, then its
// two word lists); work: the stream's four counters (FP64 / FP32 class
// kernel items, FP64 / FP32 list lengths), zeroed here before each slab.
inline bool launch_jk_fast(JKLaunch a, int la, int lb, int lc, int ld, uint2* masks,
                           long long maskWords, unsigned int* work, int nsm, cudaStream_t st,
                           int blocksPerSm = 8) {
  if (a.nBra == 0 || a.nKet == 0) return true;
  bool done = false;
  auto go = [&](auto tag64, auto tag32, bool swap) {
    using G64 = decltype(tag64);
    using G32 = decltype(tag32);
    JKLaunch b = a;
    if (swap) {
      b.braBeg = a.ketBeg; b.nBra = a.nKet;
      b.ketBeg = a.braBeg; b.nKet = a.nBra;
      b.braTileBeg = a.ketTileBeg; b.ketTileBeg = a.braTileBeg;
    }
    b.lsum = la + lb + lc + ld;
    constexpr bool CUTTABLE = jk_split(G64::LA + G64::LB + G64::LC + G64::LD);
    const bool mixed = b.precision == 1 && b.fp32_cut > 0.0;
    const int nTiles = (b.nKet + WTILE - 1) / WTILE;
    // slabs of bra pairs whose mask words fit the stream's region; each
    // reuses the region and the stream's counters after the last one's
    // kernels (stream order)
    // launches that share quartets among lanes: lists of twice the words (24 B
    // a word), or in the smallest of eight times the words
    const long long all = (long long)b.nBra * nTiles;
    const bool tiny = CUTTABLE && all <= JK_TINY_WORDS && all * JK_TINY_BYTES <= maskWords * 16;
    b.planEach = tiny ? 8 : 64;
    b.planAll = tiny;
    const bool cut = (tiny || (CUTTABLE && b.lsum <= JK_CUT_LSUM && all <= JK_CUT_WORDS &&
                               maskWords >= 2 * nTiles)) &&
                     b.maxPrimQ >= PLAN_LONG * b.planEach;
    const int dup = !cut ? 1 : (tiny ? 8 : 2);
    const int slab = dup == 8 ? b.nBra
                              : (int)std::max<long long>(
                                    1, (cut ? maskWords * 2 / 3 : maskWords) / nTiles);
    for (int ib0 = 0; ib0 < b.nBra; ib0 += slab) {
      JKLaunch c = b;
      c.braBeg = b.braBeg + ib0;
      c.nBra = std::min(slab, b.nBra - ib0);
      c.braOff = b.braOff + ib0;
      cudaMemsetAsync(work, 0, 4 * sizeof(unsigned int), st);
      const long long nWords = (long long)c.nBra * nTiles;
      // word lists: FP64 then FP32, nWords entries each; counts in work[2..3]
      int* list64 = reinterpret_cast<int*>(masks + nWords);
      int* list32 = list64 + dup * nWords;
      launch_jk_plan(c, mixed, cut, masks, list64, list32, work + 2, nsm, st);
      constexpr int WPB = JK_THREADS / 32;
      auto grid = [&](long long items) {
        return (unsigned)std::max<long long>(
            1, std::min<long long>((items + WPB - 1) / WPB, (long long)nsm * blocksPerSm));
      };
      auto launch = [&](auto split) {
        constexpr bool S = decltype(split)::value;
        const long long n = nWords * dup;
        const int e64 = entries_per_item(n, G64::NCHUNK, nsm);
        jk_class_kernel<G64, false, S><<<grid((n + e64 - 1) / e64 * G64::NCHUNK), JK_THREADS, 0,
                                         st>>>(c, masks, list64, work + 2, e64, work);
        if (mixed) {
          const int e32 = entries_per_item(n, G32::NCHUNK, nsm);
          jk_class_kernel<G32, true, S><<<grid((n + e32 - 1) / e32 * G32::NCHUNK), JK_THREADS, 0,
                                          st>>>(c, masks, list32, work + 3, e32, work + 1);
        }
      };
      if constexpr (CUTTABLE) {
        if (cut) launch(std::true_type{});
        else launch(std::false_type{});
      } else {
        launch(std::false_type{});
      }
    }
    done = true;
  };
#define CQF_TRY_CLASS(A_, B_, C_, D_, N64, N32)                                          \
  if (!done && la == A_ && lb == B_ && lc == C_ && ld == D_) go(N64{}, N32{}, false);    \
  if (!done && la == C_ && lb == D_ && lc == A_ && ld == B_) go(N64{}, N32{}, true);
  CQF_GEN_JK_CLASSES(CQF_TRY_CLASS)
#undef CQF_TRY_CLASS
  return done;
}

// ----------------------------------------------------------- Schwarz (fast)
// Diagonal (mu nu|mu nu) of the pairs of one class (LA, LB) with LA, LB <= 2
// from the generated (ab|ab) code, SCHWARZ_LANES threads per (pair, chunk)
// sharing its primitive loop (one thread each took 1.2 ms for contractions of
// eight).  Their shares of each spherical diagonal element are summed by a
// shuffle tree into the chunk's diag[pair][chunk][mu][nu], and the chunks in
// order by the finishing kernel: the bounds order the pair list, which has to
// come out alike in every process of a sharded build, so no sum may depend on
// the order of atomics.
constexpr int SCHWARZ_LANES = 16;
template <class GC>
__global__ void __launch_bounds__(JK_THREADS)
    schwarz_diag_kernel(const PairDev* __restrict__ pairs, const PrimPairDev* __restrict__ pp,
                        const double* __restrict__ boys, const double* __restrict__ sph,
                        const int* __restrict__ sphOff, const ShellDev* __restrict__ shells,
                        int beg, int n, double* diag) {
  constexpr int NA = ncart(GC::LA), NB = ncart(GC::LB), NCH = GC::NCHUNK;
  constexpr int CS = GC::NI / (NA * NB);
  const long long t = (long long)blockIdx.x * JK_THREADS + threadIdx.x;
  const long long item = t / SCHWARZ_LANES;
  const int sub = (int)(t % SCHWARZ_LANES);
  if (item >= (long long)n * NCH) return;
  const int k = (int)(item / NCH), ch = (int)(item % NCH);
  const PairDev P = pairs[beg + k];
  const unsigned group = ((1u << SCHWARZ_LANES) - 1u)
                         << ((threadIdx.x & 31) / SCHWARZ_LANES * SCHWARZ_LANES);
  const ShellDev A = shells[P.shA], B = shells[P.shB];
  const int na = A.pure ? nsph(GC::LA) : NA, nb = B.pure ? nsph(GC::LB) : NB;
  const double* TA = sph + sphOff[GC::LA];
  const double* TB = sph + sphOff[GC::LB];
  auto ta = [&](int c, int mu) { return A.pure ? TA[c * nsph(GC::LA) + mu] : (c == mu ? 1.0 : 0.0); };
  auto tb = [&](int c, int nu) { return B.pure ? TB[c * nsph(GC::LB) + nu] : (c == nu ? 1.0 : 0.0); };
  double I[GC::NI];
  GC::eri(P, P, pp, KetAoS{pp + P.pp_off, nullptr},
                           boys + (size_t)(2 * (GC::LA + GC::LB)) * BOYS_NPTS * BOYS_ROW64, ch, I, nullptr, 0.0,
                           sub, SCHWARZ_LANES);
  for (int mu = 0; mu < na; mu++)
    for (int nu = 0; nu < nb; nu++) {
      double s = 0.0;
      for (int kk = 0; kk < CS; kk++) {
        const int cd = ch * CS + kk;
        if (cd >= NA * NB) break;
        const double tcd = ta(cd / NB, mu) * tb(cd % NB, nu);
        if (tcd == 0.0) continue;
        double sab = 0.0;
        for (int a = 0; a < NA; a++) {
          const double t1 = ta(a, mu);
          if (t1 == 0.0) continue;
          for (int b = 0; b < NB; b++) sab += t1 * tb(b, nu) * I[(a * NB + b) * CS + kk];
        }
        s += tcd * sab;
      }
#pragma unroll
      for (int o = SCHWARZ_LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(group, s, o);
      if (sub == 0) diag[(size_t)item * 36 + mu * 6 + nu] = s;
    }
}

// Q = sqrt(max row sum |diag|) with rows the functions of s1
// (aointegrals_utilities.cxx:78-104); writes the pair and the table.  A warp
// per pair: lanes sum an element's nch chunks, in order.
__global__ void __launch_bounds__(128)
    schwarz_finish_kernel(const PairDev* __restrict__ pairs, const ShellDev* __restrict__ shells,
                          int beg, int n, int nch, int nshell, const double* __restrict__ diag,
                          double* Qtab, PairDev* pairsOut) {
  __shared__ double sd[4][36];
  const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (k >= n) return;
  const PairDev P = pairs[beg + k];
  const ShellDev A = shells[P.shA], B = shells[P.shB];
  const int na = A.pure ? nsph(A.l) : ncart(A.l), nb = B.pure ? nsph(B.l) : ncart(B.l);
  double* d = sd[threadIdx.x >> 5];
  for (int e = lane; e < na * nb; e += 32) {
    const int ij = e / nb * 6 + e % nb;
    double v = 0.0;
    for (int ch = 0; ch < nch; ch++) v += diag[((size_t)k * nch + ch) * 36 + ij];
    d[ij] = v;
  }
  __syncwarp();
  if (lane > 0) return;
  const bool swp = P.shA != P.s1;
  double mx = 0.0;
  if (!swp) {
    for (int i = 0; i < na; i++) {
      double r = 0.0;
      for (int j = 0; j < nb; j++) r += fabs(d[i * 6 + j]);
      mx = fmax(mx, r);
    }
  } else {
    for (int j = 0; j < nb; j++) {
      double r = 0.0;
      for (int i = 0; i < na; i++) r += fabs(d[i * 6 + j]);
      mx = fmax(mx, r);
    }
  }
  const double q = sqrt(mx);
  pairsOut[beg + k].Q = q;
  Qtab[P.s1 + (size_t)P.s2 * nshell] = q;
  Qtab[P.s2 + (size_t)P.s1 * nshell] = q;
}

// Chunks of the class (la lb | la lb), 0 if it has no generated code.
inline int schwarz_chunks(int la, int lb) {
  int n = 0;
#define CQF_SCHWARZ_CHUNKS(A_, B_, C_, D_, N64, N32) \
  if (A_ == la && B_ == lb && C_ == la && D_ == lb) n = N64::NCHUNK;
  CQF_GEN_JK_CLASSES(CQF_SCHWARZ_CHUNKS)
#undef CQF_SCHWARZ_CHUNKS
  return n;
}

// Schwarz bounds of one class with the generated code; false if the class
// has none.  diag: room for the 6 x 6 diagonals of every chunk of `room` / (36
// chunks) pairs, at least one, at a time.
inline bool launch_schwarz_fast(int la, int lb, const PairDev* pairs, const PrimPairDev* pp,
                                const double* boys, const double* sph, const int* sphOff,
                                const ShellDev* shells, int beg, int n, int nshell, double* Qtab,
                                PairDev* pairsOut, double* diag, size_t room, cudaStream_t st) {
  if (n <= 0) return true;
  bool done = false;
  auto go = [&](auto tag64) {
    using G = decltype(tag64);
    const int slab = (int)std::min<size_t>(n, room / (36 * G::NCHUNK));
    for (int k = 0; k < n; k += slab) {
      const int m = std::min(slab, n - k);
      const long long items = (long long)m * G::NCHUNK * SCHWARZ_LANES;
      schwarz_diag_kernel<G><<<(unsigned)((items + JK_THREADS - 1) / JK_THREADS), JK_THREADS, 0,
                               st>>>(pairs, pp, boys, sph, sphOff, shells, beg + k, m, diag);
      schwarz_finish_kernel<<<(m + 3) / 4, 128, 0, st>>>(pairs, shells, beg + k, m, G::NCHUNK,
                                                         nshell, diag, Qtab, pairsOut);
    }
    done = true;
  };
#define CQF_TRY_SCHWARZ(A_, B_, C_, D_, N64, N32) \
  if (!done && A_ == la && B_ == lb && C_ == la && D_ == lb) go(N64{});
  CQF_GEN_JK_CLASSES(CQF_TRY_SCHWARZ)
#undef CQF_TRY_SCHWARZ
  return done;
}

// Primitive Schwarz bounds of the pairs of one class (LA, LB <= 2):
// Qp = sqrt(max over Cartesian components |(ab|ab)|) of each primitive pair
// alone (contraction coefficients included; the integrals the class kernels
// form), a thread per (pair, chunk of components) and primitive (blockIdx.y);
// ppQ is zero on entry.  (A thread per pair took 235 us for d pairs.)  They
// bound each primitive quartet's integrals by Qp_ab Qp_cd (Cauchy-Schwarz),
// the primitive screen's estimate.
template <class GC>
__global__ void prim_schwarz_kernel(const PairDev* __restrict__ pairs,
                                    const PrimPairDev* __restrict__ pp,
                                    const double* __restrict__ boys, int beg, int n,
                                    double* __restrict__ ppQ) {
  constexpr int NA = ncart(GC::LA), NB = ncart(GC::LB), NCH = GC::NCHUNK;
  constexpr int CS = GC::NI / (NA * NB);
  const int t = blockIdx.x * blockDim.x + threadIdx.x, k = t / NCH, ch = t - k * NCH;
  if (k >= n) return;
  PairDev P1 = pairs[beg + k];
  const int npp = P1.npp, off = P1.pp_off;
  P1.npp = 1;
  for (int ip = blockIdx.y; ip < npp; ip += gridDim.y) {
    P1.pp_off = off + ip;
    double I[GC::NI];
    GC::eri(P1, P1, pp, KetAoS{pp + P1.pp_off, nullptr},
            boys + (size_t)(2 * (GC::LA + GC::LB)) * BOYS_NPTS * BOYS_ROW64, ch, I, nullptr, 0.0);
    double mx = 0.0;
    for (int kk = 0; kk < CS; kk++) {
      const int cd = ch * CS + kk;  // the diagonal element (ab | ab), ab = cd
      if (cd < NA * NB) mx = fmax(mx, fabs(I[cd * CS + kk]));
    }
    // non-negative doubles order as their bits
    atomicMax(reinterpret_cast<unsigned long long*>(ppQ + P1.pp_off),
              (unsigned long long)__double_as_longlong(sqrt(mx)));
  }
}

// Primitive Schwarz bounds of one class with the generated code; false if
// the class has none.
inline bool launch_prim_schwarz(int la, int lb, const PairDev* pairs, const PrimPairDev* pp,
                                const double* boys, int beg, int n, int maxNpp, double* ppQ,
                                cudaStream_t st) {
  if (n <= 0) return true;
  bool done = false;
  auto go = [&](auto tag64) {
    using G = decltype(tag64);
    prim_schwarz_kernel<G><<<dim3((n * G::NCHUNK + 63) / 64, std::min(maxNpp, PRIM_ROWS)), 64, 0, st>>>(
        pairs, pp, boys, beg, n, ppQ);
    done = true;
  };
#define CQF_TRY_PRIM(A_, B_, C_, D_, N64, N32) \
  if (!done && A_ == la && B_ == lb && C_ == la && D_ == lb) go(N64{});
  CQF_GEN_JK_CLASSES(CQF_TRY_PRIM)
#undef CQF_TRY_PRIM
  return done;
}

}  // namespace cqf
