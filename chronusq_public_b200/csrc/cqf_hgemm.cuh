// Hermite-matrix engine: shell quartets of any angular momentum, with plain
// or differentiated pairs, as two dense products on the FP64 matrix
// instructions (mma.sync m16n8k4).
//
// A pair density (times a differential operator acting on it) is a Hermite
// expansion at the product centre; the expansion coefficients of one
// primitive pair are a matrix C[(component pair, operator)][h].  For a
// quartet of primitive pairs
//     G[h][col] = sum_h' K[col][h'] R~[h + h'],    col = (cd, ket operator)
//     M[row][col] = sum_h H[row][h] G[h][col],     row = (ab, bra operator)
// with R~ the Hermite integrals of Q - P (the ket's (-1)^|h'| is moved to
// (-1)^|h| of G).  The tables H and K are built once per basis (hg_ensure);
// they are stored in the order in which a warp's A fragment reads them
// (16 rows x 4 orders = 512 consecutive bytes).
//
// A block takes one bra pair and a batch of its kets from the planning pass's
// masks: the Boys values of a batch of primitive quartets (a lane each; for a
// single one a lane per order), R level by level for the whole batch from a
// table of parents into cubes [t][u][v] (so the index of h + h' is the sum of
// two table entries), G and M in shared memory with the kets' columns side by
// side, then the digestion D::digest of the operator components.  G sums over
// the ket primitives, M over the bra primitives, so a contracted quartet is
// digested once.  The s and p classes batch up to 32 kets and primitives (one
// primitive quartet at a time the barriers and a nearly empty matrix tile
// were most of their time); quartets whose components do not fit in shared
// memory go one ket at a time in chunks of rows and columns.
//
// What bounds it: the per-thread kernels this replaces spent their time on
// integer index work over local arrays at a few percent of the FP64 rate;
// here the products run at the matrix rate and the rest (R, digestion) is
// spread over the block.  Small launches split the primitive quartets of a
// quartet over several blocks (the digestion is linear in the integrals), so
// that a molecule of a few shells with long contractions fills the GPU too.
// Whole builds, with those kernels and with this engine: one uncontracted Ag
// atom (N 152; LLSS, SSSS and the f classes) 495 -> 115 ms, a water molecule
// in 6-31G(d) with SSSS 580 -> 2.3 ms and with Gaunt 651 -> 3.0 ms, J and K of
// 3 waters in cc-pVTZ 141 -> 6.3 ms, the gradient of 4 waters in cc-pVDZ
// 269 -> 11.0 ms; the Ag atom's quartets need 17 ms at the FP64 rate.
#pragma once

#include <algorithm>
#include <atomic>

#include "cqf_eri.cuh"
#include "cqf_hg_items.hpp"
#include "cqf_internal.hpp"

namespace cqf {

// ---------------------------------------------------------------- tables
// Rows of a table: component pair x operators.  PLAIN: none; D6: d/dr of the
// first function (x, y, z), then of the second; D3: of the first only; SPIN:
// dot and cross (x, y, z) of the two gradients.
__host__ __device__ constexpr int hg_ops(int k) {
  return k == HG_PLAIN ? 1 : (k == HG_D6 ? 6 : (k == HG_D3 ? 3 : 4));
}
__host__ __device__ constexpr int hg_rise(int k) { return k == HG_PLAIN ? 0 : (k == HG_SPIN ? 2 : 1); }
__host__ __device__ inline int hg_tiles(int k, int la, int lb) {  // 16-row tiles
  return (ncart(la) * ncart(lb) * hg_ops(k) + 15) / 16;
}
__host__ __device__ inline int hg_ktiles(int k, int la, int lb) {  // 4-order tiles
  return (nherm(la + lb + hg_rise(k)) + 3) / 4;
}
__host__ __device__ inline int hg_size(int k, int la, int lb) {  // doubles per primitive pair
  return hg_tiles(k, la, lb) * hg_ktiles(k, la, lb) * 64;
}

// D(16 x 8) += A(16 x 4) B(4 x 8): lane holds A(lane / 4, lane % 4) and
// A(lane / 4 + 8, lane % 4), B(lane % 4, lane / 4), D(lane / 4 (+ 8),
// 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ void hg_mma(double (&c)[4], double2 a, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3},{%4,%5},{%6},"
               "{%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a.x), "d"(a.y), "d"(b));
}

// ---------------------------------------------------------------- launch
struct HgSide {
  const double* tab;  // table of the class's first primitive pair
  int ppBeg;          // that primitive pair
};
constexpr int HG_MAXPASS = 2;
struct HgLaunch {
  const PairDev* pairs;
  const PrimPairDev* pp;
  const double* boys;
  const float* boys32;
  int la, lb, lc, ld;
  int braBeg, ketBeg, nTiles;      // WTILE-ket words per bra pair
  const uint2* masks;              // .x: FP64 quartets, .y: FP32 ones
  const int* list64;               // words with FP64 quartets, then those with FP32 ones
  const int* list32;
  const unsigned* lcount;          // lengths of the two lists
  unsigned* counter;               // next item
  int nsub;                        // items per word (when items is null)
  const uint2* items;              // or the list hg_expand_kernel made,
  const unsigned* nItems;          // and its length
  int nru, ncu;                    // row / column units per chunk
  int nk, nr;                      // kets and primitive quartets (a power of two) per batch
  HgSide bra[HG_MAXPASS], ket[HG_MAXPASS];
};

// A batch as the digestion sees it: kets Q[0 .. nk), those with pre[q + 1] >
// pre[q] computed; the components of rows [ab0, ab1) and columns [cd0, cd1)
// of ket q are in M[pass] at column q * cw[pass].
struct HgQuartet {
  const PairDev* P;
  const PairDev* Q;
  const int* pre;
  int nk, la, lb, lc, ld;
  int ab0, ab1, cd0, cd1;
  const double* M[HG_MAXPASS];
  int ms[HG_MAXPASS], cw[HG_MAXPASS];  // row strides of M (hg_row), columns per ket
  double* st;                          // D::stage() doubles of shared memory
  __device__ __forceinline__ bool have(int q) const { return pre[q + 1] > pre[q]; }
};

// Row r of M: stride ms (8 modulo 16: the fragments' stores hit every bank
// once) and two more per four rows (the digestion reads M by rows, four per
// component pair, from many threads at once).
__host__ __device__ __forceinline__ int hg_row(int r, int ms) { return r * ms + 2 * (r >> 2); }

// Shared-memory layout (doubles).
struct HgLayout {
  int L, S, FS, NH, RS, CS;        // strides of F, of a recursion buffer and of a cube (odd)
  int oF, oR0, oR1, oCube, oG[HG_MAXPASS], oM[HG_MAXPASS], oSt, oRec, oOff, oKet, oPre, total;
  int ms[HG_MAXPASS], gs[HG_MAXPASS], cw[HG_MAXPASS];
};
template <class D>
__host__ __device__ inline HgLayout hg_layout(int la, int lb, int lc, int ld, int nru, int ncu,
                                              int nk, int nr) {
  HgLayout o;
  const int lab = la + lb, lcd = lc + ld;
  o.L = lab + lcd + hg_rise(D::tb(0)) + hg_rise(D::tk(0));
  o.S = o.L + 1;
  o.FS = (o.L + 5) | 1;  // F_0 .. F_L, X, Y, Z
  o.NH = nherm(o.L);
  o.RS = nherm(o.L - 1) | 1;
  o.CS = o.L * o.S * o.S + 1;  // t = L is the last index; L (L + 1)^2 is even
  int p = 0;
  auto take = [&](int n) { int r = p; p += (n + 1) / 2 * 2; return r; };
  o.oKet = take(32 * (int)(sizeof(PairDev) / sizeof(double)));
  o.oPre = take(34);  // 33 prefix sums, the item, 32 first primitives
  o.oF = take(nr * o.FS);
  o.oR0 = take(nr * o.RS);
  o.oR1 = take(nr * o.RS);
  o.oCube = take(nr * o.CS);
  for (int q = 0; q < D::NP; q++) {
    const int rt = hg_tiles(D::tb(q), la, lb), ct = hg_tiles(D::tk(q), lc, ld);
    const int r = nru * D::rtu(q) < rt ? nru * D::rtu(q) : rt;
    o.cw[q] = ncu * D::ctu(q) < ct ? ncu * D::ctu(q) * 16
                                   : ncart(lc) * ncart(ld) * hg_ops(D::tk(q));
    const int c = (nk * o.cw[q] + 15) / 16;
    // strides free of bank conflicts for the fragments' reads and writes
    o.gs[q] = c * 16 + 4;
    o.ms[q] = c * 16 + 8;
    const int hb = (nherm(lab + hg_rise(D::tb(q))) + 7) / 8 * 8;
    o.oG[q] = take(hb * o.gs[q]);
    o.oM[q] = take(r * 16 * o.ms[q] + r * 8);
  }
  o.oSt = take(D::stage(la, lb, lc, ld, nk));
  o.oRec = take((o.NH + 1) / 2);
  o.oOff = take((o.NH + 1) / 2);
  o.total = p;
  return o;
}

// The parents of Hermite index e in the recursion
// R^(n)_h = X_axis R^(n+1)_p1 + coef R^(n+1)_p2 (p1 = h - 1 on the axis,
// p2 = h - 2, coef = h_axis - 1), and its place in the cube with the parity
// of |h| in bit 30.
__device__ __forceinline__ void hg_index(int e, int S, unsigned& rec, int& off) {
  int n = 0;
  while (nherm(n) <= e) n++;
  const int r = e - nherm(n - 1);
  int k = 0;
  while ((k + 1) * (k + 2) / 2 <= r) k++;
  const int v = r - k * (k + 1) / 2, u = k - v, t = n - k;
  int p1 = 0, p2 = 0, ax = 0, cf = 0;
  if (t > 0) {
    p1 = hidx(t - 1, u, v);
    cf = t - 1;
    if (t > 1) p2 = hidx(t - 2, u, v);
  } else if (u > 0) {
    ax = 1;
    p1 = hidx(0, u - 1, v);
    cf = u - 1;
    if (u > 1) p2 = hidx(0, u - 2, v);
  } else if (v > 0) {
    ax = 2;
    p1 = hidx(0, 0, v - 1);
    cf = v - 1;
    if (v > 1) p2 = hidx(0, 0, v - 2);
  }
  rec = (unsigned)p1 | ((unsigned)p2 << 10) | ((unsigned)ax << 20) | ((unsigned)cf << 22);
  off = (t * S + u) * S + v + ((n & 1) << 30);
}

// Boys values of one primitive quartet, scaled: f[n] = pref (-2 alpha)^n F_n,
// then X, Y, Z of Q - P; T the arithmetic.
template <typename T>
__device__ __forceinline__ void hg_boys(const PrimPairDev& A, const PrimPairDev& B, int L,
                                        double* f, const T* tab) {
  const T X = T(B.P[0] - A.P[0]), Y = T(B.P[1] - A.P[1]), Z = T(B.P[2] - A.P[2]);
  const T pq = T(A.p) + T(B.p), alpha = T(A.p) * T(B.p) / pq;
  T s = T(34.986836655249725693) / sqrt(pq) * T(A.Kp) * T(B.Kp);  // 2 pi^(5/2)
  T F[25];
  boys_rt<T>(L, alpha * (X * X + Y * Y + Z * Z), F, tab);
  const T m2a = T(-2) * alpha;
  for (int n = 0; n <= L; n++) {
    f[n] = double(s * F[n]);
    s *= m2a;
  }
  f[L + 1] = double(X);
  f[L + 2] = double(Y);
  f[L + 3] = double(Z);
}
// the same, the orders spread over the lanes of a warp
template <typename T>
__device__ __forceinline__ void hg_boys_lanes(const PrimPairDev& A, const PrimPairDev& B, int L,
                                              double* f, const T* tab, int lane) {
  const T X = T(B.P[0] - A.P[0]), Y = T(B.P[1] - A.P[1]), Z = T(B.P[2] - A.P[2]);
  const T pq = T(A.p) + T(B.p), alpha = T(A.p) * T(B.p) / pq;
  T s = T(34.986836655249725693) / sqrt(pq) * T(A.Kp) * T(B.Kp);
  T* F = reinterpret_cast<T*>(f);
  boys_lanes<T>(L, alpha * (X * X + Y * Y + Z * Z), F, tab, lane);
  const T v = lane <= L ? F[lane] : T(0);
  __syncwarp();
  const T m2a = T(-2) * alpha;
  for (int n = 0; n < lane; n++) s *= n < L ? m2a : T(1);
  if (lane <= L) f[lane] = double(s * v);
  if (lane == 0) {
    f[L + 1] = double(X);
    f[L + 2] = double(Y);
    f[L + 3] = double(Z);
  }
}

// R~ of nb <= nr primitive quartets (nr = 2^ln) into their cubes, level by
// level over the block, the quartets in the fastest index; ends with a
// barrier.
template <typename T>
__device__ __forceinline__ void hg_R(const HgLayout& o, int ln, int nb, const double* F, T* r0,
                                     T* r1, double* cube, const unsigned* rec, const int* off) {
  const int L = o.L;
  for (int n = L; n >= 0; n--) {
    T* cur = (n & 1) ? r1 : r0;
    const T* prv = (n & 1) ? r0 : r1;
    const int cnt = nherm(L - n) << ln;
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
      const int e = i >> ln, j = i & ((1 << ln) - 1);
      if (j >= nb) continue;
      const double* f = F + j * o.FS;
      T v;
      if (e == 0) {
        v = T(f[n]);
      } else {
        const unsigned w = rec[e];
        const T* p = prv + j * o.RS;
        v = T(f[L + 1 + ((w >> 20) & 3)]) * p[w & 1023] +
            T((int)(w >> 22)) * p[(w >> 10) & 1023];
      }
      if (n > 0) cur[j * o.RS + e] = v;
      else cube[j * o.CS + (off[e] & 0x3fffffff)] = double(v);
    }
    __syncthreads();
  }
}

// G[h][col0 + c] (+)= sum over nj primitive quartets (cubes cs apart, tables
// ksz apart) of sum_h' K[c][h'] R~[h + h'], c < cw, one item: 8 orders h (tile
// nt) and up to two 16-column tiles from tile 2 m0 of ctn.
__device__ __forceinline__ void hg_gemm1(const double* tab, size_t ksz, int nj, int kt, int HK,
                                         int m0, int ctn, int nt, int HB, const double* cube,
                                         int cs, const int* off, double* G, int gs, int cw,
                                         bool first) {
  const int lane = threadIdx.x & 31;
  const int n = nt * 8 + (lane >> 2);
  const double* rn = cube + (n < HB ? (off[n] & 0x3fffffff) : 0);
  const bool two = 2 * m0 + 1 < ctn;
  const double2* a0 = reinterpret_cast<const double2*>(tab) + lane + (size_t)(2 * m0) * kt * 32;
  double c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
  if (two) {
    for (int j = 0; j < nj; j++, a0 += ksz / 2, rn += cs) {
      const double2* a1 = a0 + (size_t)kt * 32;
#pragma unroll 4
      for (int k = 0; k < kt; k++) {
        const int kk = 4 * k + (lane & 3);
        const double b = rn[kk < HK ? (off[kk] & 0x3fffffff) : 0];
        const double2 x = __ldg(a0 + k * 32), y = __ldg(a1 + k * 32);
        hg_mma(c0, x, b);
        hg_mma(c1, y, b);
      }
    }
  } else if (kt == 1) {  // s kets: primitives in the inner loop, two chains
    const double* rk = rn + ((lane & 3) < HK ? (off[lane & 3] & 0x3fffffff) : 0);
    const size_t js = ksz / 2;
    int j = 0;
#pragma unroll 4
    for (; j + 2 <= nj; j += 2) {
      const double2 x = __ldg(a0 + j * js), y = __ldg(a0 + (j + 1) * js);
      const double b0 = rk[j * cs], b1 = rk[(j + 1) * cs];
      hg_mma(c0, x, b0);
      hg_mma(c1, y, b1);
    }
    if (j < nj) hg_mma(c0, __ldg(a0 + j * js), rk[j * cs]);
#pragma unroll
    for (int t = 0; t < 4; t++) c0[t] += c1[t];
  } else {
    for (int j = 0; j < nj; j++, a0 += ksz / 2, rn += cs) {
      int k = 0;
#pragma unroll 2
      for (; k + 2 <= kt; k += 2) {
        const int k0 = 4 * k + (lane & 3), k1 = k0 + 4;
        const double b0 = rn[off[k0] & 0x3fffffff];
        const double b1 = rn[k1 < HK ? (off[k1] & 0x3fffffff) : 0];
        const double2 x = __ldg(a0 + k * 32), y = __ldg(a0 + (k + 1) * 32);
        hg_mma(c0, x, b0);
        hg_mma(c1, y, b1);
      }
      if (k < kt) {
        const int kk = 4 * k + (lane & 3);
        hg_mma(c0, __ldg(a0 + k * 32), rn[kk < HK ? (off[kk] & 0x3fffffff) : 0]);
      }
    }
#pragma unroll
    for (int t = 0; t < 4; t++) c0[t] += c1[t];
  }
  const int c = 32 * m0 + (lane >> 2);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int h = nt * 8 + 2 * (lane & 3) + j;
    const double sg = (h < HB && ((off[h] >> 30) & 1)) ? -1.0 : 1.0;
    double* g = G + (size_t)h * gs + c;
    const double v[4] = {sg * c0[j], sg * c0[2 + j], sg * c1[j], sg * c1[2 + j]};
#pragma unroll
    for (int t = 0; t < 4; t++)
      if (c + 8 * t < cw && (t < 2 || two)) g[8 * t] = first ? v[t] : g[8 * t] + v[t];
  }
}

// M[row][col] (+)= sum_h H[row][h] G[h][col] for rtn tiles of 16 rows of one
// table (tab: its first tile) and ctn tiles of 16 columns.  A warp takes one
// row tile and 16 columns.
__device__ __forceinline__ void hg_gemm2(const double* tab, int kt, int rtn, int ctn,
                                         const double* G, int gs, double* M, int ms, bool first) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const double2* t2 = reinterpret_cast<const double2*>(tab) + lane;
  for (int it = warp; it < rtn * ctn; it += W) {
    const int ct = it / rtn, rt = it - ct * rtn;
    const double2* a = t2 + (size_t)rt * kt * 32;
    const double* g = G + (size_t)(lane & 3) * gs + 16 * ct + (lane >> 2);
    double c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
#pragma unroll 4
    for (int k = 0; k < kt; k++) {
      const double2 x = __ldg(a + k * 32);
      const double b0 = g[(size_t)4 * k * gs], b1 = g[(size_t)4 * k * gs + 8];
      hg_mma(c0, x, b0);
      hg_mma(c1, x, b1);
    }
    double* m = M + hg_row(16 * rt + (lane >> 2), ms) + 16 * ct + 2 * (lane & 3);
    double2* m0 = reinterpret_cast<double2*>(m);
    double2* m1 = reinterpret_cast<double2*>(m + hg_row(8, ms));
    double2 v0 = make_double2(c0[0], c0[1]), v1 = make_double2(c1[0], c1[1]);
    double2 w0 = make_double2(c0[2], c0[3]), w1 = make_double2(c1[2], c1[3]);
    if (!first) {
      v0.x += m0[0].x; v0.y += m0[0].y; v1.x += m0[4].x; v1.y += m0[4].y;
      w0.x += m1[0].x; w0.y += m1[0].y; w1.x += m1[4].x; w1.y += m1[4].y;
    }
    m0[0] = v0;
    m0[4] = v1;
    m1[0] = w0;
    m1[4] = w1;
  }
}

// Items of contracted classes: every listed word cut into parts of about
// `work` primitive quartets, at most `most` of them over both lists (hg_cut).
// Without it the words of the longest contractions (32 x 64 x 64 primitive
// quartets against a mean of a few hundred) were the whole launch's tail: SMs
// were active for 22% of the (ss|ss) gradient launch.
// item = {word | FP32 << 31, b | cb << 8 | k << 16 | ck << 24}.
__global__ static void __launch_bounds__(128)
    hg_expand_kernel(const PairDev* __restrict__ pairs, int braBeg, int ketBeg, int nTiles,
                     const uint2* __restrict__ masks, const int* __restrict__ list64,
                     const int* __restrict__ list32, const unsigned* __restrict__ lcount,
                     int work, int most, uint2* __restrict__ items, unsigned* nItems) {
  const int n64 = (int)lcount[0], n = n64 + (int)lcount[1];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const bool lo = i >= n64;
    const int word = lo ? list32[i - n64] : list64[i];
    const uint2 mk = masks[word];
    const int ib = word / nTiles, jk0 = (word - ib * nTiles) * WTILE;
    // the primitives of the entry's kets and of the word's other ones
    int nk = 0, other = 0;
    for (unsigned b = mk.x | mk.y; b; b &= b - 1u) {
      const int n1 = pairs[ketBeg + jk0 + __ffs(b) - 1].npp;
      if ((lo ? mk.y : mk.x) & (b & -b)) nk += n1;
      else other += n1;
    }
    const HgCut c = hg_cut(pairs[braBeg + ib].npp, nk, other, work, most);
    const int cb = c.cb, ck = c.ck;
    const unsigned at = atomicAdd(nItems, (unsigned)(cb * ck));
    for (int b = 0; b < cb; b++)
      for (int k = 0; k < ck; k++)
        items[at + b * ck + k] =
            make_uint2((unsigned)word | (lo ? 0x80000000u : 0u),
                       (unsigned)b | (cb << 8) | (k << 16) | ((unsigned)ck << 24));
  }
}

template <class D>
__global__ void __launch_bounds__(512, 1)
    hg_kernel(const HgLaunch a, const typename D::Args args) {
  extern __shared__ double sm[];
  const int la = a.la, lb = a.lb, lc = a.lc, ld = a.ld;
  const int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld);
  const HgLayout o = hg_layout<D>(la, lb, lc, ld, a.nru, a.ncu, a.nk, a.nr);
  const int L = o.L, tid = threadIdx.x, nt = blockDim.x, cs = o.CS;
  const int ln = 31 - __clz(a.nr);
  const int warp = tid >> 5, W = nt >> 5;
  double* Fs = sm + o.oF;
  double* cube = sm + o.oCube;
  unsigned* rec = reinterpret_cast<unsigned*>(sm + o.oRec);
  int* off = reinterpret_cast<int*>(sm + o.oOff);
  PairDev* Qs = reinterpret_cast<PairDev*>(sm + o.oKet);
  int* pre = reinterpret_cast<int*>(sm + o.oPre);  // pre[q]: first primitive entry of ket q
  int* sitem = pre + 34;
  int* first = pre + 36;  // first[q]: ket q's first primitive of this item
  for (int e = tid; e < o.NH; e += nt) hg_index(e, o.S, rec[e], off[e]);
  const int n64 = (int)a.lcount[0], n32 = (int)a.lcount[1];
  const int nItems = a.items ? (int)*a.nItems : (n64 + n32) * a.nsub;
  const int abU = a.nru * D::ABU, cdU = a.ncu * D::CDU;  // components per chunk
  for (;;) {
    if (tid == 0) *sitem = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int item = *sitem;
    if (item >= nItems) break;
    uint2 it = make_uint2(0, 0);
    if (a.items) {
      it = __ldg(a.items + item);
    } else {
      const int w = item / a.nsub;
      it.x = w < n64 ? __ldg(a.list64 + w) : (__ldg(a.list32 + (w - n64)) | 0x80000000);
      it.y = (1u << 8) | (1u << 24);
    }
    const bool lo = it.x >> 31;
    const int word = (int)(it.x & 0x7fffffff);
    const uint2 mk = __ldg(a.masks + word);
    unsigned bits = lo ? mk.y : mk.x;
    if (!a.items && a.nsub > 1) {  // a share of the word's kets
      const int span = 32 / a.nsub;
      bits &= ((1u << span) - 1u) << (item % a.nsub * span);
    }
    const int nBits = __popc(bits);
    const int ib = word / a.nTiles, jk0 = (word - ib * a.nTiles) * WTILE;
    const PairDev P = a.pairs[a.braBeg + ib];
    const int cb = (it.y >> 8) & 255, ip0 = P.npp * (int)(it.y & 255) / cb,
              ip1 = P.npp * (int)((it.y & 255) + 1) / cb;
    __syncthreads();  // every thread has read the item
    // the word's kets, and the item's share of their concatenated primitives:
    // ket q computes entries pre[q] .. pre[q + 1] - 1, from primitive first[q]
    if (tid < 32) {
      int n = 0;
      if (tid < nBits) {
        unsigned b = bits;
        for (int q = 0; q < tid; q++) b &= b - 1u;
        const PairDev Q = a.pairs[a.ketBeg + jk0 + __ffs(b) - 1];
        Qs[tid] = Q;
        n = Q.npp;
      }
      int s = n;
      for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, s, d);
        if (tid >= d) s += t;
      }
      const int all = __shfl_sync(0xffffffffu, s, 31);
      const int ck = it.y >> 24, k = (it.y >> 16) & 255;
      const int r0 = all * k / ck, r1 = all * (k + 1) / ck;
      if (tid == 0) pre[0] = 0;
      pre[tid + 1] = min(max(s, r0), r1) - r0;
      first[tid] = max(r0 - (s - n), 0);
    }
    __syncthreads();
    for (int q0 = 0; q0 < nBits; q0 += a.nk) {
      const int q1 = min(q0 + a.nk, nBits), eb0 = pre[q0], eb1 = pre[q1];
      const int total = eb1 - eb0;
      if (total == 0) continue;
      const bool one = total == 1 && ip1 - ip0 == 1;
      bool haveR = false;
      for (int cd0 = 0; cd0 < ncd; cd0 += cdU)
        for (int ab0 = 0; ab0 < nab; ab0 += abU) {
          for (int ip = ip0; ip < ip1; ip++) {
            for (int eb = eb0; eb < eb1; eb += a.nr) {
              const int nb = min(a.nr, eb1 - eb);
              if (!(one && haveR)) {
                const PrimPairDev& A = a.pp[P.pp_off + ip];
                if (nb == 1) {
                  if (tid < 32) {
                    int q = q0;
                    while (pre[q + 1] <= eb) q++;
                    const PrimPairDev& B = a.pp[Qs[q].pp_off + first[q] + eb - pre[q]];
                    if (lo) hg_boys_lanes<float>(A, B, L, Fs, a.boys32, tid);
                    else hg_boys_lanes<double>(A, B, L, Fs, a.boys, tid);
                  }
                } else if (tid < nb) {
                  int q = q0;
                  while (pre[q + 1] <= eb + tid) q++;
                  const PrimPairDev& B = a.pp[Qs[q].pp_off + first[q] + eb + tid - pre[q]];
                  if (lo) hg_boys<float>(A, B, L, Fs + tid * o.FS, a.boys32);
                  else hg_boys<double>(A, B, L, Fs + tid * o.FS, a.boys);
                }
                __syncthreads();
                if (lo)
                  hg_R<float>(o, ln, nb, Fs, reinterpret_cast<float*>(sm + o.oR0),
                              reinterpret_cast<float*>(sm + o.oR1), cube, rec, off);
                else
                  hg_R<double>(o, ln, nb, Fs, sm + o.oR0, sm + o.oR1, cube, rec, off);
                haveR = true;
              }
              if (one && ab0 > 0) continue;  // G is there
              int qa = q0;
              while (pre[qa + 1] <= eb) qa++;
              int qb = qa;
              while (pre[qb + 1] < eb + nb) qb++;
#pragma unroll
              for (int q = 0; q < D::NP; q++) {
                const int TB = D::tb(q), TK = D::tk(q);
                const int HB = nherm(la + lb + hg_rise(TB)), HK = nherm(lc + ld + hg_rise(TK));
                const int ktk = (HK + 3) / 4, ksz = hg_size(TK, lc, ld);
                const int ct0 = cd0 / D::CDU * D::ctu(q);
                const int ctn = min(a.ncu * D::ctu(q), hg_tiles(TK, lc, ld) - ct0);
                const int nn = (HB + 7) / 8, per = nn * ((ctn + 1) / 2);
                for (int it = warp; it < (qb - qa + 1) * per; it += W) {
                  const int k = qa + it / per, r = it % per;
                  const int j0 = max(pre[k], eb), j1 = min(pre[k + 1], eb + nb);
                  if (j0 >= j1) continue;
                  const int iq = first[k] + j0 - pre[k];
                  const double* tk = a.ket[q].tab +
                                     (size_t)(Qs[k].pp_off + iq - a.ket[q].ppBeg) * ksz +
                                     (size_t)ct0 * ktk * 64;
                  hg_gemm1(tk, ksz, j1 - j0, ktk, HK, r / nn, ctn, r % nn, HB,
                           cube + (j0 - eb) * cs, cs, off, sm + o.oG[q] + (k - q0) * o.cw[q], o.gs[q],
                           o.cw[q], j0 == pre[k]);
                }
              }
              __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < D::NP; q++) {
              const int TB = D::tb(q);
              const int ktb = (nherm(la + lb + hg_rise(TB)) + 3) / 4;
              const int rt0 = ab0 / D::ABU * D::rtu(q);
              const int rtn = min(a.nru * D::rtu(q), hg_tiles(TB, la, lb) - rt0);
              const double* tb = a.bra[q].tab +
                                 (size_t)(P.pp_off + ip - a.bra[q].ppBeg) * hg_size(TB, la, lb) +
                                 (size_t)rt0 * ktb * 64;
              hg_gemm2(tb, ktb, rtn, ((q1 - q0) * o.cw[q] + 15) / 16, sm + o.oG[q], o.gs[q],
                       sm + o.oM[q], o.ms[q], ip == ip0);
            }
            __syncthreads();
          }
          HgQuartet z;
          z.P = &P;
          z.Q = Qs + q0;
          z.pre = pre + q0;
          z.nk = q1 - q0;
          z.la = la; z.lb = lb; z.lc = lc; z.ld = ld;
          z.ab0 = ab0;
          z.ab1 = min(nab, ab0 + abU);
          z.cd0 = cd0;
          z.cd1 = min(ncd, cd0 + cdU);
#pragma unroll
          for (int q = 0; q < D::NP; q++) {
            z.M[q] = sm + o.oM[q];
            z.ms[q] = o.ms[q];
            z.cw[q] = o.cw[q];
          }
          z.st = sm + o.oSt;
          D::digest(args, z);
          __syncthreads();
        }
    }
    __syncthreads();  // before the next item is written
  }
}

// Sum over the 2^l lanes of a group (lanes of one group call together).
__device__ __forceinline__ double hg_group_sum(double v, int l) {
  const int lane = threadIdx.x & 31;
  const unsigned mask = (l == 5 ? 0xffffffffu : ((1u << (1 << l)) - 1u)) << (lane & ~((1 << l) - 1));
  for (int o = (1 << l) >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}
// log2 of the lanes that share an exchange unit: enough units for the block,
// at most 8 and not many more than the ni contracted bra components.
__device__ __forceinline__ int hg_share(int units, int ni) {
  int l = 0;
  while (l < 3 && (units << l) < (int)blockDim.x && (1 << l) < ni) l++;
  return l;
}

// The steps k < n at which lo + k step (step > 0) lies in [0, end): [k0, k1).
__device__ __forceinline__ void hg_range(int lo, int step, int n, int end, int& k0, int& k1) {
  k0 = lo < 0 ? (-lo + step - 1) / step : 0;
  k1 = end > lo ? min(n, (end - lo + step - 1) / step) : 0;
}

// Planning pass over the words (bra pair, 32 kets) of nBra x nKet quartets:
// f(ib, jk, work, lo) returns whether quartet (ib, jk) exists and sets
// whether it is computed, and with FP32 Hermite integrals.  Masks, lists of
// non-empty words (lengths in lcount[0 / 1], zero on entry) and the counters
// visited / screened / FP32 / FP64; the layout of jk_plan_kernel.
template <class F>
__device__ __forceinline__ void hg_plan(int nBra, int nKet, uint2* __restrict__ masks,
                                        int* __restrict__ list64, int* __restrict__ list32,
                                        unsigned* __restrict__ lcount,
                                        unsigned long long* counters, F f) {
  const int lane = threadIdx.x & 31;
  const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nw = (int)((gridDim.x * blockDim.x) >> 5);
  const int nTiles = (nKet + WTILE - 1) / WTILE, nWords = nBra * nTiles;
  unsigned long long cVis = 0, cScr = 0, c32 = 0, c64 = 0;
  for (int run = gw; run * 32 < nWords; run += nw) {
    int my64 = -1, my32 = -1, n64 = 0, n32 = 0;
    const int wEnd = min((run + 1) * 32, nWords);
    for (int word = run * 32; word < wEnd; word++) {
      const int ib = word / nTiles, jk = (word - ib * nTiles) * WTILE + lane;
      bool work = false, lo = false;
      const bool visited = jk < nKet && f(ib, jk, work, lo);
      work = work && visited;
      const unsigned bv = __ballot_sync(0xffffffffu, visited);
      const unsigned bw = __ballot_sync(0xffffffffu, work);
      const unsigned b32 = __ballot_sync(0xffffffffu, work && lo), b64 = bw & ~b32;
      cVis += __popc(bv);
      cScr += __popc(bv & ~bw);
      c32 += __popc(b32);
      c64 += __popc(b64);
      if (lane == 0) masks[word] = make_uint2(b64, b32);
      if (b64) {
        if (lane == n64) my64 = word;
        n64++;
      }
      if (b32) {
        if (lane == n32) my32 = word;
        n32++;
      }
    }
    unsigned base64 = 0, base32 = 0;
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
    if (cVis) atomicAdd(counters + 0, cVis);
    if (cScr) atomicAdd(counters + 1, cScr);
    if (c32) atomicAdd(counters + 2, c32);
    if (c64) atomicAdd(counters + 3, c64);
  }
}

// ---------------------------------------------------------- host side
// The engine on nBra x nKet quartets of class pair (cb | ck) in slabs of bra
// pairs whose mask words fit the stream's region (maskWords words of 16 B;
// work: its four counters), and of bra and ket pairs whose tables fit its
// windows where the basis does not hold them.  plan(part, masks, list64,
// list32, lcount, grid) launches the planning pass on a part of the class pair.
struct HgPart {
  int ib0, nBra, k0, nKet;  // bra pairs [ib0, ib0 + nBra) x kets [k0, k0 + nKet)
  // launch arguments of the class pair, narrowed to the part.  braOff is the
  // first bra's place among the kets: of one class, a ket sits at or before its bra
  template <class A>
  A of(A a) const {
    a.braBeg += ib0;
    a.nBra = nBra;
    a.ketBeg += k0;
    a.nKet = nKet;
    a.braOff = ib0 - k0;
    return a;
  }
};
struct HgRegion {
  uint2* masks;
  long long maskWords;
  unsigned* work;
  double* win;  // hg_windows<D> doubles
};
// Chunk of rows and columns, kets and primitive quartets per batch.  A class
// whose components fit whole batches kets (up to 32) and primitives within
// HG_SMEM_BATCH; else one ket at a time and as few chunks as fit in the
// shared memory of two blocks per SM, or of one (the cube and the recursion
// buffers of the f classes take up to 60 KB by themselves).  Returns the
// bytes, 0 when nothing fits.
constexpr size_t HG_SMEM_BATCH = 54 * 1024;  // four blocks of four warps per SM
constexpr int HG_BATCH_WARPS = 4;
constexpr size_t HG_SMEM_TWO = 112 * 1024;
constexpr size_t HG_SMEM_MAX = 224 * 1024;
template <class D>
inline size_t hg_chunk(HgLaunch& a, int nkMax, int nrMax) {
  const int la = a.la, lb = a.lb, lc = a.lc, ld = a.ld;
  const int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld);
  const int ru = (nab + D::ABU - 1) / D::ABU, cu = (ncd + D::CDU - 1) / D::CDU;
  auto bytes = [&](int r, int c, int k, int n) {
    return (size_t)hg_layout<D>(la, lb, lc, ld, r, c, k, n).total * sizeof(double);
  };
  a.nk = a.nr = 1;
  if (bytes(ru, cu, 1, 1) <= HG_SMEM_BATCH) {
    a.nru = ru;
    a.ncu = cu;
    // kets and primitives grow together (a batch has at least one primitive
    // quartet per ket), then the primitives alone, up to a thread each
    for (int n = 2; n <= 32; n *= 2) {
      const int k = std::min(n, nkMax), r = n < 2 * nrMax ? n : a.nr;
      if (bytes(ru, cu, k, r) > HG_SMEM_BATCH) break;
      a.nk = k;
      a.nr = r;
    }
    while (a.nr >= a.nk && 2 * a.nr <= 32 * HG_BATCH_WARPS && 2 * a.nr < 2 * nrMax &&
           bytes(ru, cu, a.nk, 2 * a.nr) <= HG_SMEM_BATCH)
      a.nr *= 2;
    return bytes(ru, cu, a.nk, a.nr);
  }
  // fewest chunks within each limit; one block of 16 warps per SM where that
  // saves chunks (a chunk's digestion keeps only its share of the outputs'
  // threads busy), else two of eight
  int chunks2 = 1 << 30;
  size_t got = 0;
  for (size_t lim : {HG_SMEM_TWO, HG_SMEM_MAX}) {
    double best = 1e30;
    int chunks = 1 << 30, nru = 0, ncu = 0;
    size_t b1 = 0;
    for (int c = 1; c <= cu; c++)
      for (int r = 1; r <= ru; r++) {
        const size_t b = bytes(r, c, 1, 1);
        if (b > lim) break;
        const int n = ((cu + c - 1) / c) * ((ru + r - 1) / r);
        const double cost = n + 0.01 * (r + c);  // the smallest with this chunk count
        if (cost < best) {
          best = cost;
          chunks = n;
          nru = r;
          ncu = c;
          b1 = b;
        }
      }
    if (b1 && (got == 0 || chunks < chunks2)) {
      a.nru = nru;
      a.ncu = ncu;
      got = b1;
      chunks2 = chunks;
    }
  }
  return got;
}

// Warps per block from the products' size (matrix instructions per primitive
// quartet) and the batch.
template <class D>
inline int hg_warps(const HgLaunch& a, size_t smem) {
  if (smem > HG_SMEM_TWO) return 16;  // one block per SM
  long long m = 0;
  for (int q = 0; q < D::NP; q++) {
    const int hb = nherm(a.la + a.lb + hg_rise(D::tb(q)));
    const long long ct = hg_tiles(D::tk(q), a.lc, a.ld), rt = hg_tiles(D::tb(q), a.la, a.lb);
    m += ct * ((hb + 7) / 8) * hg_ktiles(D::tk(q), a.lc, a.ld) + 2 * ct * rt * ((hb + 3) / 4);
  }
  if (a.nr >= 32) return HG_BATCH_WARPS;
  m *= std::max(a.nk, a.nr);
  return m <= 24 ? 1 : (m <= 96 ? 2 : (m <= 400 ? 4 : 8));
}

// Chunk, batch, warps and shared memory of a launch; the search takes tens of
// microseconds for the large classes, so each thread keeps what it found for
// a class pair and batch limits.
struct HgShape {
  int nkMax = 0, nrMax = 0, nru = 0, ncu = 0, nk = 0, nr = 0, W = 0;
  size_t smem = 0;
};
template <class D>
inline const HgShape& hg_shape(HgLaunch a, int nkMax, int nrMax) {
  static thread_local HgShape memo[NCLS][NCLS];
  HgShape& m = memo[class_id(a.la, a.lb)][class_id(a.lc, a.ld)];
  if (m.nkMax != nkMax || m.nrMax != nrMax) {
    m.smem = hg_chunk<D>(a, nkMax, nrMax);
    m.nkMax = nkMax; m.nrMax = nrMax;
    m.nru = a.nru; m.ncu = a.ncu; m.nk = a.nk; m.nr = a.nr;
    m.W = m.smem ? hg_warps<D>(a, m.smem) : 0;
  }
  return m;
}

// Launches the engine on one class pair (la lb | lc ld) whose planning pass
// wrote masks and lists; nItems: items at most.  *counter is zero.
template <class D>
inline cqf_status hg_launch(HgLaunch a, const typename D::Args& args, const HgShape& m,
                            long long nItems, int device, int nsm, cudaStream_t st) {
  if (!m.smem) return fail(CQF_ENOTSUP, "class does not fit in shared memory");
  a.nru = m.nru; a.ncu = m.ncu; a.nk = m.nk; a.nr = m.nr;
  // the shared-memory limit, once per device (always the same value)
  static std::atomic<unsigned> limited{0};
  const unsigned bit = 1u << (device & 31);
  if (device > 31 || !(limited.load() & bit)) {
    if (cudaFuncSetAttribute(hg_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)HG_SMEM_MAX) != cudaSuccess)
      return fail(CQF_ECUDA, "hg_kernel: shared-memory limit");
    limited.fetch_or(bit);
  }
  // resident blocks per SM: shared memory, and the 128 registers per thread
  // of the launch bound
  const int occ = (int)std::max<size_t>(
      1, std::min<size_t>(HG_SMEM_MAX / (m.smem + 1024), (size_t)(16 / m.W)));
  const unsigned grid =
      (unsigned)std::max<long long>(1, std::min((long long)nsm * occ, nItems));
  hg_kernel<D><<<grid, 32 * m.W, m.smem, st>>>(a, args);
  return CQF_OK;
}
// Doubles of a launch stream's windows of the tables that the basis does not
// hold (hg_win), one for each pass and side.
template <class D>
inline size_t hg_windows(const cqf_basis* B) {
  size_t n = 0;
  for (int q = 0; q < D::NP; q++) n += B->hg_win[D::tb(q)] + B->hg_win[D::tk(q)];
  return n;
}
// The pairs from `beg` on, at most n of them and at least one, whose tables of
// `kind` (class c) fit its window; n where the basis holds the table.
inline int hg_fit(const cqf_basis* B, int kind, int c, int beg, int n) {
  if (!B->hg_win[kind]) return n;
  int l1, l2;
  class_ls(c, l1, l2);
  const long long cap = (long long)(B->hg_win[kind] / hg_size(kind, l1, l2));
  const cqf::PairDev* p = B->h_pairs.data() + beg;
  int m = 1;
  while (m < n && (long long)p[m].pp_off + p[m].npp - p[0].pp_off <= cap) m++;
  return m;
}

template <class D, class Plan>
inline cqf_status hg_contract(const cqf_basis* B, int cb, int ck, int braBeg, int nBra, int ketBeg,
                              int nKet, const HgRegion& r, const typename D::Args& args,
                              cudaStream_t st, Plan plan) {
  HgLaunch h{};
  h.pairs = B->d_pairsHg;
  h.pp = B->d_pp;
  h.boys = B->d_boys64;
  h.boys32 = B->d_boys32;
  class_ls(cb, h.la, h.lb);
  class_ls(ck, h.lc, h.ld);
  h.masks = r.masks;
  h.lcount = r.work + 2;
  h.counter = r.work;
  // the tables the basis holds, or windows of them, built for each slab
  double* win[2 * HG_MAXPASS];
  double* next = r.win;
  for (int q = 0; q < D::NP; q++) {
    const int tb = D::tb(q), tk = D::tk(q);
    h.bra[q] = {B->d_hg[tb] + B->hg_beg[tb][cb], B->cls_pp_beg[cb]};
    h.ket[q] = {B->d_hg[tk] + B->hg_beg[tk][ck], B->cls_pp_beg[ck]};
    win[2 * q] = next;
    win[2 * q + 1] = next + B->hg_win[tb];
    next += B->hg_win[tb] + B->hg_win[tk];
  }
  auto window = [&](HgSide& s, double* w, int kind, int c, int beg, int n) {
    if (!B->hg_win[kind]) return;
    s = {w, B->h_pairs[beg].pp_off};
    hg_fill(B, kind, c, beg, n, w, st);
  };
  const int npb = B->cls_npp_max[cb], npk = B->cls_npp_max[ck];
  // items that keep the GPU busy: four for each of an SM's four batch blocks.
  // 4 nsm: gradient of 4 waters in cc-pVDZ 11.0 -> 9.8 ms, four-component
  // builds 3-5% slower; 64 nsm: 13.9 ms and 1-17% slower
  const long long fill = 16LL * B->nsm;
  for (int k0 = 0, nk = 0; k0 < nKet; k0 += nk) {
    nk = nKet - k0;
    for (int q = 0; q < D::NP; q++) nk = std::min(nk, hg_fit(B, D::tk(q), ck, ketBeg + k0, nk));
    for (int q = 0; q < D::NP; q++)
      window(h.ket[q], win[2 * q + 1], D::tk(q), ck, ketBeg + k0, nk);
    h.ketBeg = ketBeg + k0;
    h.nTiles = (nk + WTILE - 1) / WTILE;
    // contracted classes: words are cut by their number of primitive quartets
    const HgSlab sl = npb > 1 || npk > 1 ? hg_slab(2 * r.maskWords, nBra, h.nTiles)
                                         : HgSlab{0, r.maskWords};
    const int most = sl.most;
    const int slab = (int)std::max<long long>(1, sl.words / h.nTiles);
    for (int ib0 = 0, n = 0; ib0 < nBra; ib0 += n) {
      n = std::min(slab, nBra - ib0);
      for (int q = 0; q < D::NP; q++) n = std::min(n, hg_fit(B, D::tb(q), cb, braBeg + ib0, n));
      for (int q = 0; q < D::NP; q++) window(h.bra[q], win[2 * q], D::tb(q), cb, braBeg + ib0, n);
      const long long nWords = (long long)n * h.nTiles;
      int* list64 = reinterpret_cast<int*>(r.masks + nWords);
      int* list32 = list64 + nWords;
      h.list64 = list64;
      h.list32 = list32;
      h.braBeg = braBeg + ib0;
      if (cudaMemsetAsync(r.work, 0, 4 * sizeof(unsigned), st) != cudaSuccess)
        return fail(CQF_ECUDA, "hg_contract: counters");
      const unsigned gp =
          (unsigned)std::min<long long>(((nWords + 31) / 32 + 7) / 8, (long long)B->nsm * 8);
      plan(HgPart{ib0, n, k0, nk}, r.masks, list64, list32, r.work + 2, gp);
      h.nsub = 1;
      long long nItems;
      if (most) {
        uint2* items = r.masks + 2 * nWords;
        h.items = items;
        h.nItems = r.work + 1;
        // a part's primitive quartets: the launch's (unscreened) number over
        // the items that fill the GPU, at least a batch; at most 1024, which
        // bounds the tail of the largest launches (256 and 4096: within 4%)
        const double all = (double)n / nBra * nk / nKet * B->cls_npp_sum[cb] * B->cls_npp_sum[ck];
        const int part = (int)std::min(
            1024.0, std::max((double)hg_shape<D>(h, 32, 32 * npk).nr, all / fill));
        hg_expand_kernel<<<(unsigned)std::min<long long>((nWords + 127) / 128, B->nsm * 8), 128,
                           0, st>>>(h.pairs, h.braBeg, h.ketBeg, h.nTiles, r.masks, list64, list32,
                                    h.lcount, part, most, items, r.work + 1);
        nItems = nWords * most;
      } else {
        h.items = nullptr;
        while (h.nsub < 32 && nWords * h.nsub < fill) h.nsub *= 2;
        nItems = nWords * h.nsub;
      }
      const HgShape& m = hg_shape<D>(h, 32 / h.nsub, 32 / h.nsub * npk);
      const cqf_status s = hg_launch<D>(h, args, m, nItems, B->device, B->nsm, st);
      if (s != CQF_OK) return s;
    }
  }
  return CQF_OK;
}

}  // namespace cqf
