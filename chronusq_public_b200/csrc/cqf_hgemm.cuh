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
// A block takes quartets one after the other from the planning pass's masks:
// Boys values (one lane per primitive quartet, or one lane per order for a
// single one), R level by level from a table of parents into a cube
// [t][u][v] (so the index of h + h' is the sum of two table entries), G and
// M in shared memory, then the digestion D::digest of the operator
// components.  G sums over the ket primitives, M over the bra primitives, so
// a contracted quartet is digested once.  Quartets whose components do not
// fit in shared memory go in chunks of rows and columns.
//
// What bounds it: the per-thread kernels this replaces spent their time on
// integer index work over local arrays at a few percent of the FP64 rate;
// here the products run at the matrix rate and the rest (R, digestion) is
// spread over the block.  Small launches split the primitive quartets of a
// quartet over several blocks (the digestion is linear in the integrals), so
// that a molecule of a few shells with long contractions fills the GPU too.
#pragma once

#include <algorithm>

#include "cqf_eri.cuh"
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
  int nsub, parts;                 // items per word, and parts of a quartet's primitives
  int nru, ncu;                    // row / column units per chunk
  HgSide bra[HG_MAXPASS], ket[HG_MAXPASS];
};

// One quartet's work as the digestion sees it: the components of rows
// [ab0, ab1) and columns [cd0, cd1) are in M.
struct HgQuartet {
  const PairDev* P;
  const PairDev* Q;
  int la, lb, lc, ld;
  int ab0, ab1, cd0, cd1;
  const double* M[HG_MAXPASS];
  int ms[HG_MAXPASS];              // row strides of M
};

// Shared-memory layout (doubles).
struct HgLayout {
  int L, S, FS;
  int oF, oR0, oR1, oCube, oG[HG_MAXPASS], oM[HG_MAXPASS], oRec, oOff, oItem, total;
  int ms[HG_MAXPASS], gs[HG_MAXPASS];
};
template <class D>
__host__ __device__ inline HgLayout hg_layout(int la, int lb, int lc, int ld, int nru, int ncu) {
  HgLayout o;
  const int lab = la + lb, lcd = lc + ld;
  o.L = lab + lcd + hg_rise(D::tb(0)) + hg_rise(D::tk(0));
  o.S = o.L + 1;
  o.FS = (o.L + 5) | 1;  // F_0 .. F_L, X, Y, Z, alpha
  int p = 0;
  auto take = [&](int n) { int r = p; p += (n + 1) / 2 * 2; return r; };
  o.oF = take(32 * o.FS);
  o.oR0 = take(nherm(o.L));
  o.oR1 = take(nherm(o.L));
  o.oCube = take(o.S * o.S * o.S);
  for (int q = 0; q < D::NP; q++) {
    const int rt = hg_tiles(D::tb(q), la, lb), ct = hg_tiles(D::tk(q), lc, ld);
    const int r = nru * D::rtu(q) < rt ? nru * D::rtu(q) : rt;
    const int c = ncu * D::ctu(q) < ct ? ncu * D::ctu(q) : ct;
    // strides free of bank conflicts for the fragments' reads and writes
    o.gs[q] = c * 16 + 4;
    o.ms[q] = c * 16 + 8;
    const int hb = (nherm(lab + hg_rise(D::tb(q))) + 7) / 8 * 8;
    o.oG[q] = take(hb * o.gs[q]);
    o.oM[q] = take(r * 16 * o.ms[q]);
  }
  o.oRec = take((nherm(o.L) + 1) / 2);
  o.oOff = take((nherm(o.L) + 1) / 2);
  o.oItem = take(2);
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

// R~ into the cube, level by level over the block; ends with a barrier.
template <typename T>
__device__ __forceinline__ void hg_R(int L, const double* f, T* r0, T* r1, double* cube,
                                     const unsigned* rec, const int* off) {
  const T X = T(f[L + 1]), Y = T(f[L + 2]), Z = T(f[L + 3]);
  for (int n = L; n >= 0; n--) {
    T* cur = (n & 1) ? r1 : r0;
    const T* prv = (n & 1) ? r0 : r1;
    const int cnt = nherm(L - n);
    for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
      T v;
      if (e == 0) {
        v = T(f[n]);
      } else {
        const unsigned w = rec[e];
        const int ax = (w >> 20) & 3;
        v = (ax == 0 ? X : (ax == 1 ? Y : Z)) * prv[w & 1023] +
            T((int)(w >> 22)) * prv[(w >> 10) & 1023];
      }
      if (n > 0) cur[e] = v;
      else cube[off[e] & 0x3fffffff] = double(v);
    }
    __syncthreads();
  }
}

// G[h][col] (+)= sum_h' K[col][h'] R~[h + h'] for ctn tiles of 16 columns of
// one table (tab: its first tile), HB orders h.  A warp takes 8 orders and
// up to two column tiles.
__device__ __forceinline__ void hg_gemm1(const double* tab, int kt, int HK, int ctn, int HB,
                                         const double* cube, const int* off, double* G, int gs,
                                         bool first) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int nn = (HB + 7) / 8, mg = (ctn + 1) / 2;
  const double2* t2 = reinterpret_cast<const double2*>(tab) + lane;
  for (int it = warp; it < nn * mg; it += W) {
    const int m0 = it / nn, nt = it - m0 * nn;
    const int n = nt * 8 + (lane >> 2);
    const double* rn = cube + (n < HB ? (off[n] & 0x3fffffff) : 0);
    const bool two = 2 * m0 + 1 < ctn;
    const double2* a0 = t2 + (size_t)(2 * m0) * kt * 32;
    const double2* a1 = a0 + (size_t)kt * 32;
    double c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
    if (two) {
#pragma unroll 4
      for (int k = 0; k < kt; k++) {
        const int kk = 4 * k + (lane & 3);
        const double b = rn[kk < HK ? (off[kk] & 0x3fffffff) : 0];
        const double2 x = __ldg(a0 + k * 32), y = __ldg(a1 + k * 32);
        hg_mma(c0, x, b);
        hg_mma(c1, y, b);
      }
    } else {
#pragma unroll 4
      for (int k = 0; k < kt; k++) {
        const int kk = 4 * k + (lane & 3);
        const double b = rn[kk < HK ? (off[kk] & 0x3fffffff) : 0];
        hg_mma(c0, __ldg(a0 + k * 32), b);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int h = nt * 8 + 2 * (lane & 3) + j;
      const double sg = (h < HB && ((off[h] >> 30) & 1)) ? -1.0 : 1.0;
      double* g = G + (size_t)h * gs + 32 * m0 + (lane >> 2);
      if (first) {
        g[0] = sg * c0[j];
        g[8] = sg * c0[2 + j];
        if (two) {
          g[16] = sg * c1[j];
          g[24] = sg * c1[2 + j];
        }
      } else {
        g[0] += sg * c0[j];
        g[8] += sg * c0[2 + j];
        if (two) {
          g[16] += sg * c1[j];
          g[24] += sg * c1[2 + j];
        }
      }
    }
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
    double* m = M + (size_t)(16 * rt + (lane >> 2)) * ms + 16 * ct + 2 * (lane & 3);
    double2* m0 = reinterpret_cast<double2*>(m);
    double2* m1 = reinterpret_cast<double2*>(m + 8 * (size_t)ms);
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

template <class D>
__global__ void __launch_bounds__(256, 2)
    hg_kernel(const HgLaunch a, const typename D::Args args) {
  extern __shared__ double sm[];
  const int la = a.la, lb = a.lb, lc = a.lc, ld = a.ld;
  const int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld);
  const HgLayout o = hg_layout<D>(la, lb, lc, ld, a.nru, a.ncu);
  const int L = o.L, tid = threadIdx.x, nt = blockDim.x;
  double* Fs = sm + o.oF;
  double* cube = sm + o.oCube;
  unsigned* rec = reinterpret_cast<unsigned*>(sm + o.oRec);
  int* off = reinterpret_cast<int*>(sm + o.oOff);
  int* sitem = reinterpret_cast<int*>(sm + o.oItem);
  for (int e = tid; e < nherm(L); e += nt) hg_index(e, o.S, rec[e], off[e]);
  const int n64 = (int)a.lcount[0], n32 = (int)a.lcount[1];
  const int nItems = (n64 + n32) * a.nsub * a.parts;
  const int abU = a.nru * D::ABU, cdU = a.ncu * D::CDU;  // components per chunk
  for (;;) {
    if (tid == 0) *sitem = (int)atomicAdd(a.counter, 1u);
    __syncthreads();
    const int item = *sitem;
    __syncthreads();
    if (item >= nItems) break;
    const int part = item % a.parts, ws = item / a.parts;
    const int sub = ws % a.nsub, w = ws / a.nsub;
    const bool lo = w >= n64;
    const int word = lo ? __ldg(a.list32 + (w - n64)) : __ldg(a.list64 + w);
    const uint2 mk = __ldg(a.masks + word);
    const int span = 32 / a.nsub;
    unsigned bits = (lo ? mk.y : mk.x) >> (sub * span);
    if (span < 32) bits &= (1u << span) - 1u;
    const int ib = word / a.nTiles, jk0 = (word - ib * a.nTiles) * WTILE + sub * span;
    const PairDev P = a.pairs[a.braBeg + ib];
    for (; bits; bits &= bits - 1u) {
      const PairDev Q = a.pairs[a.ketBeg + jk0 + __ffs(bits) - 1];
      const int nq = Q.npp, n = P.npp * nq;
      const int k0 = (int)((long long)n * part / a.parts);
      const int k1 = (int)((long long)n * (part + 1) / a.parts);
      if (k0 == k1) continue;
      const bool one = k1 - k0 == 1;
      bool haveR = false;
      for (int cd0 = 0; cd0 < ncd; cd0 += cdU)
        for (int ab0 = 0; ab0 < nab; ab0 += abU) {
          bool firstM = true;
          for (int kb = k0; kb < k1; kb += 32) {
            const int nb = min(32, k1 - kb);
            if (!(one && haveR)) {
              if (tid < 32) {
                if (one) {
                  const PrimPairDev& A = a.pp[P.pp_off + kb / nq];
                  const PrimPairDev& B = a.pp[Q.pp_off + kb % nq];
                  if (lo) hg_boys_lanes<float>(A, B, L, Fs, a.boys32, tid);
                  else hg_boys_lanes<double>(A, B, L, Fs, a.boys, tid);
                } else if (tid < nb) {
                  const PrimPairDev& A = a.pp[P.pp_off + (kb + tid) / nq];
                  const PrimPairDev& B = a.pp[Q.pp_off + (kb + tid) % nq];
                  if (lo) hg_boys<float>(A, B, L, Fs + tid * o.FS, a.boys32);
                  else hg_boys<double>(A, B, L, Fs + tid * o.FS, a.boys);
                }
              }
              __syncthreads();
            }
            for (int j = 0; j < nb; j++) {
              const int ip = (kb + j) / nq, iq = (kb + j) - ip * nq;
              if (!(one && haveR)) {
                const double* f = Fs + j * o.FS;
                if (lo)
                  hg_R<float>(L, f, reinterpret_cast<float*>(sm + o.oR0),
                              reinterpret_cast<float*>(sm + o.oR1), cube, rec, off);
                else
                  hg_R<double>(L, f, sm + o.oR0, sm + o.oR1, cube, rec, off);
                haveR = true;
              }
              const bool firstG = iq == 0 || kb + j == k0;
              const bool lastG = iq == nq - 1 || kb + j == k1 - 1;
#pragma unroll
              for (int q = 0; q < D::NP; q++) {
                const int TB = D::tb(q), TK = D::tk(q);
                const int HB = nherm(la + lb + hg_rise(TB)), HK = nherm(lc + ld + hg_rise(TK));
                const int ktk = (HK + 3) / 4;
                const int ct0 = cd0 / D::CDU * D::ctu(q);
                const int ctn = min(a.ncu * D::ctu(q), hg_tiles(TK, lc, ld) - ct0);
                double* G = sm + o.oG[q];
                if (!(one && ab0 > 0)) {
                  const double* tk = a.ket[q].tab +
                                     (size_t)(Q.pp_off + iq - a.ket[q].ppBeg) *
                                         hg_size(TK, lc, ld) + (size_t)ct0 * ktk * 64;
                  hg_gemm1(tk, ktk, HK, ctn, HB, cube, off, G, o.gs[q], firstG);
                }
              }
              __syncthreads();
              if (lastG) {
#pragma unroll
                for (int q = 0; q < D::NP; q++) {
                  const int TB = D::tb(q);
                  const int ktb = (nherm(la + lb + hg_rise(TB)) + 3) / 4;
                  const int ct0 = cd0 / D::CDU * D::ctu(q);
                  const int ctn = min(a.ncu * D::ctu(q), hg_tiles(D::tk(q), lc, ld) - ct0);
                  const int rt0 = ab0 / D::ABU * D::rtu(q);
                  const int rtn = min(a.nru * D::rtu(q), hg_tiles(TB, la, lb) - rt0);
                  const double* tb = a.bra[q].tab +
                                     (size_t)(P.pp_off + ip - a.bra[q].ppBeg) *
                                         hg_size(TB, la, lb) + (size_t)rt0 * ktb * 64;
                  hg_gemm2(tb, ktb, rtn, ctn, sm + o.oG[q], o.gs[q], sm + o.oM[q], o.ms[q],
                           firstM);
                }
                firstM = false;
                __syncthreads();
              }
            }
          }
          HgQuartet z;
          z.P = &P;
          z.Q = &Q;
          z.la = la; z.lb = lb; z.lc = lc; z.ld = ld;
          z.ab0 = ab0;
          z.ab1 = min(nab, ab0 + abU);
          z.cd0 = cd0;
          z.cd1 = min(ncd, cd0 + cdU);
#pragma unroll
          for (int q = 0; q < D::NP; q++) {
            z.M[q] = sm + o.oM[q];
            z.ms[q] = o.ms[q];
          }
          D::digest(args, z);
          __syncthreads();
        }
    }
  }
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
// work: its four counters).  plan(ib0, n, masks, list64, list32, lcount,
// grid) launches the planning pass on bra pairs [ib0, ib0 + n) of the class;
// digest arguments may depend on the slab: args(ib0, n).
struct HgRegion {
  uint2* masks;
  long long maskWords;
  unsigned* work;
};
// Chunk of rows and columns: as few chunks as fit in the shared memory of
// two blocks per SM, else of one (the R cube and the recursion buffers of
// the f classes take up to 60 KB by themselves); 0 rows when nothing fits.
constexpr size_t HG_SMEM_TWO = 112 * 1024;
constexpr size_t HG_SMEM_MAX = 224 * 1024;
template <class D>
inline size_t hg_chunk(int la, int lb, int lc, int ld, int& nru, int& ncu) {
  const int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld);
  const int ru = (nab + D::ABU - 1) / D::ABU, cu = (ncd + D::CDU - 1) / D::CDU;
  nru = ncu = 0;
  for (size_t lim : {HG_SMEM_TWO, HG_SMEM_MAX}) {
    double best = 1e30;
    size_t bytes = 0;
    for (int c = 1; c <= cu; c++)
      for (int r = 1; r <= ru; r++) {
        const size_t b = (size_t)hg_layout<D>(la, lb, lc, ld, r, c).total * sizeof(double);
        if (b > lim) break;
        const int nc = (cu + c - 1) / c, nr = (ru + r - 1) / r;
        const double cost = nc * nr + 0.01 * (r + c);  // the smallest with this chunk count
        if (cost < best) {
          best = cost;
          nru = r;
          ncu = c;
          bytes = b;
        }
      }
    // a chunk of a single row tile leaves most warps idle: take one block
    if (bytes && (best < 24.0 || lim == HG_SMEM_MAX)) return bytes;
  }
  return 0;
}

// Warps per block from the products' size (matrix instructions per
// primitive quartet): a warp for the s and p classes, eight from d shells on.
template <class D>
inline int hg_warps(int la, int lb, int lc, int ld) {
  long long m = 0;
  for (int q = 0; q < D::NP; q++) {
    const int hb = nherm(la + lb + hg_rise(D::tb(q)));
    const long long ct = hg_tiles(D::tk(q), lc, ld), rt = hg_tiles(D::tb(q), la, lb);
    m += ct * ((hb + 7) / 8) * hg_ktiles(D::tk(q), lc, ld) + 2 * ct * rt * ((hb + 3) / 4);
  }
  return m <= 48 ? 1 : (m <= 200 ? 2 : (m <= 800 ? 4 : 8));
}

// Launches the engine on one class pair (la lb | lc ld) whose planning pass
// wrote masks and lists of nWords words; nq: quartets at most, npMax: the
// largest product of primitive-pair counts.  *counter is zero.
template <class D>
inline cqf_status hg_launch(HgLaunch a, const typename D::Args& args, long long nWords,
                            long long nq, int npMax, int nsm, cudaStream_t st) {
  const size_t smem = hg_chunk<D>(a.la, a.lb, a.lc, a.ld, a.nru, a.ncu);
  if (!smem) return fail(CQF_ENOTSUP, "class does not fit in shared memory");
  const int W = hg_warps<D>(a.la, a.lb, a.lc, a.ld);
  if (cudaFuncSetAttribute(hg_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)HG_SMEM_MAX) != cudaSuccess)
    return fail(CQF_ECUDA, "hg_kernel: shared-memory limit");
  // resident blocks per SM: shared memory, 2048 threads, 32 blocks, and the
  // 128 registers per thread of the launch bound
  const int occ = (int)std::max<size_t>(
      1, std::min<size_t>(std::min<size_t>(HG_SMEM_MAX / (smem + 1024), 16 / W), 32));
  const long long slots = (long long)nsm * occ;
  // items: enough to fill the GPU four times over, by splitting the words'
  // quartets first and then the quartets' primitives
  a.nsub = 1;
  while (a.nsub < 32 && nWords * a.nsub < 4 * slots) a.nsub *= 2;
  a.parts = 1;
  const long long items = std::min(nq, nWords * a.nsub);
  while (a.parts * 2 <= npMax && items * a.parts < 4 * slots) a.parts *= 2;
  const unsigned grid =
      (unsigned)std::max<long long>(1, std::min(slots, nWords * a.nsub * a.parts));
  hg_kernel<D><<<grid, 32 * W, smem, st>>>(a, args);
  return CQF_OK;
}

template <class D, class Plan>
inline cqf_status hg_contract(const cqf_basis* B, int cb, int ck, int braBeg, int nBra, int ketBeg,
                              int nKet, const HgRegion& r, const typename D::Args& args,
                              cudaStream_t st, Plan plan) {
  HgLaunch h{};
  h.pairs = B->d_pairs;
  h.pp = B->d_pp;
  h.boys = B->d_boys64;
  h.boys32 = B->d_boys32;
  class_ls(cb, h.la, h.lb);
  class_ls(ck, h.lc, h.ld);
  h.ketBeg = ketBeg;
  h.nTiles = (nKet + WTILE - 1) / WTILE;
  h.masks = r.masks;
  h.lcount = r.work + 2;
  h.counter = r.work;
  for (int q = 0; q < D::NP; q++) {
    const int tb = D::tb(q), tk = D::tk(q);
    h.bra[q] = {B->d_hg[tb] + B->hg_beg[tb][cb], B->cls_pp_beg[cb]};
    h.ket[q] = {B->d_hg[tk] + B->hg_beg[tk][ck], B->cls_pp_beg[ck]};
  }
  const int slab = (int)std::max<long long>(1, r.maskWords / h.nTiles);
  for (int ib0 = 0; ib0 < nBra; ib0 += slab) {
    const int n = std::min(slab, nBra - ib0);
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
    plan(ib0, n, r.masks, list64, list32, r.work + 2, gp);
    const cqf_status s = hg_launch<D>(h, args, nWords, (long long)n * nKet,
                                      B->cls_npp_max[cb] * B->cls_npp_max[ck], B->nsm, st);
    if (s != CQF_OK) return s;
  }
  return CQF_OK;
}

}  // namespace cqf
