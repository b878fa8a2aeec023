// Four-component Dirac-Coulomb direct contraction on the device.
//
// Replaces GTODirectRelERIContraction::twoBodyContract -> directScaffoldLibcint
// (include/particleintegrals/contract/direct4C_libcint.hpp:138-2832) and the
// FourCompFock::formGDDirect assembly (include/fockbuilder/fourcompfock/
// impl.hpp:3752-4636).
//
// Small-component functions are the large-component ones differentiated
// (restricted kinetic balance), so the LLSS and SSSS terms need derivative
// ERIs.  A differentiated pair (m, n) acts on the electron's spin as the
// operator P_mn = dm.dn + i sigma.(dm x dn): four real operator components
// (dot, cross x, y, z) per integral.  The reference takes the 9 / 81 raw
// derivative components from libcint and writes each spin product out; here
// the components come from McMurchie-Davidson over the pair's Hermite tables
// raised by one on each centre,
//     d/dx [x^i e^{-a x^2}] = i x^{i-1} e^{-a x^2} - 2a x^{i+1} e^{-a x^2},
// and the digestion is the Pauli algebra of P:
//   Coulomb   J^a(12) += P^a(12|34) rho(43), rho = (Re D^S, -Im D^x, -Im D^y, -Im D^z)
//   LS exchange  K(3,2) -= D(4,1) P_12                          (LLSS)
//   SS exchange  K(1,4) -= P_12 D(2,3) P_34                     (SSSS)
// with the reference's quartet sets, screens and degeneracy factors.
//
// Layout: densities and accumulators live in the Cartesian AO basis (exact
// transforms before and after, as on the 1C path); Coulomb accumulators are
// real, exchange accumulators complex.  The integrals of a shell quartet come
// from the Hermite-matrix engine (cqf_hgemm.cuh), both pairs' operator
// components in its coefficient tables; the digestion reads them from shared
// memory (cqf_hg_digest.cuh) and adds with FP64 atomics.  Hermitian outputs are completed from the
// accumulated half at the back transform (the reference's "upper =
// conj(lower)" after Hermitian digestion).
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "cqf_deriv.cuh"
#include "cqf_eri.cuh"
#include "cqf_hgemm.cuh"
#include "cqf_internal.hpp"

namespace cqf {
namespace {

#define CQF_RCUDA(call)                                                                    \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return fail(e_ == cudaErrorMemoryAllocation ? CQF_ENOMEM : CQF_ECUDA,                \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                     \
  } while (0)

#define CQF_RTRY(expr)           \
  do {                           \
    cqf_status s_ = (expr);      \
    if (s_ != CQF_OK) return s_; \
  } while (0)

unsigned rgrid(size_t n, int b) { return (unsigned)((n + b - 1) / b); }

// max of the six shell-block norms of a quartet in the reference's roles
// (direct4C_libcint.hpp:602-620, :940-948)
__device__ __forceinline__ double sh_max(const double* __restrict__ n, int s1, int s2, int s3,
                                         int s4, int ns) {
  auto B = [&](int a, int b) { return __ldg(n + a + (size_t)b * ns); };
  return fmax(fmax(fmax(B(s1, s2), B(s1, s3)), fmax(B(s2, s3), B(s1, s4))),
              fmax(B(s2, s4), B(s3, s4)));
}

// ------------------------------------------------------------ spin algebra
struct __align__(16) Q4 {  // s + v . sigma, complex components
  double2 s, x, y, z;
};

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 ctimes_i(double2 a) { return make_double2(-a.y, a.x); }

// (p.s + p.v sigma)(q.s + q.v sigma) = p.s q.s + p.v.q.v
//   + (p.s q.v + q.s p.v + i p.v x q.v) . sigma
__device__ __forceinline__ Q4 qmul(const Q4& p, const Q4& q) {
  Q4 r;
  r.s = cadd(cadd(cmul(p.s, q.s), cmul(p.x, q.x)), cadd(cmul(p.y, q.y), cmul(p.z, q.z)));
  r.x = cadd(cadd(cmul(p.s, q.x), cmul(q.s, p.x)),
             ctimes_i(csub(cmul(p.y, q.z), cmul(p.z, q.y))));
  r.y = cadd(cadd(cmul(p.s, q.y), cmul(q.s, p.y)),
             ctimes_i(csub(cmul(p.z, q.x), cmul(p.x, q.z))));
  r.z = cadd(cadd(cmul(p.s, q.z), cmul(q.s, p.z)),
             ctimes_i(csub(cmul(p.x, q.y), cmul(p.y, q.x))));
  return r;
}

// t sigma_k (k = 1, 2, 3): sigma_j sigma_k = delta_jk + i eps_jkl sigma_l, so
// t sigma_x = (t.x, t.s, i t.z, -i t.y), t sigma_y = (t.y, -i t.z, t.s, i t.x),
// t sigma_z = (t.z, i t.y, -i t.x, t.s)
__device__ __forceinline__ Q4 qsig(const Q4& t, int k) {
  auto mi = [](double2 a) { return make_double2(a.y, -a.x); };  // -i a
  if (k == 1) return Q4{t.x, t.s, ctimes_i(t.z), mi(t.y)};
  if (k == 2) return Q4{t.y, mi(t.z), t.s, ctimes_i(t.x)};
  return Q4{t.z, ctimes_i(t.y), mi(t.x), t.s};
}

__device__ __forceinline__ double2 ldz(const double* X, size_t e) {
  return __ldg(reinterpret_cast<const double2*>(X) + e);
}
__device__ __forceinline__ void addz(double* A, size_t e, double2 v, double w) {
  atomicAdd(A + 2 * e, v.x * w);
  atomicAdd(A + 2 * e + 1, v.y * w);
}

struct RelLaunch {
  const PairDev* pairs;
  const float2* pairRange;  // per pair: FP32 range data (fp32_range_ok)
  int mixed;                // 1: quartets with bound < cut take FP32 Hermite integrals
  double cut;
  int braBeg, nBra, braOff, ketBeg, nKet, same, lsum;
  int screen;
  double thresh;
  const double* norms;  // max shell-block norms of the screening matrices
  const double* qLL;
  const double* qSS;
  int nShell, ncart, exchange;
  const double* Xll;     // Cartesian complex X[CLLMS]
  const double* Xss[4];  // Cartesian complex X[CSSM*]
  const double* Xk[4];   // exchange densities: X[XLSM*] (LLSS) / X[XSSM*] (SSSS)
  double* Jll;           // real
  double* Jss[4];        // real
  double* K[4];          // complex
  int shardIdx, shardCnt;  // bra pairs p with p % shardCnt == shardIdx only
  unsigned long long* counters;
};

constexpr int REL_THREADS = 64;

// Planning pass of one class pair: per (bra pair, word of 32 kets) the
// quartets that survive the screen, as FP64 and FP32 lane masks, and the
// lists of non-empty words (the layout of jk_plan_kernel).
// TYPE 1: LLSS (bra = SS pair, differentiated; ket = LL pair), all
// (bra, ket) combinations (direct4C_libcint.hpp:907-929).
// TYPE 2: SSSS, unique quartets of pairs (:2018-2047).
template <int TYPE>
__global__ void __launch_bounds__(256)
    rel_plan_kernel(const RelLaunch a, uint2* __restrict__ masks, int* __restrict__ list64,
                    int* __restrict__ list32, unsigned* __restrict__ lcount) {
  const int ns = a.nShell;
  hg_plan(a.nBra, a.nKet, masks, list64, list32, lcount, a.counters,
          [&](int ib, int jk, bool& work, bool& lo) {
            if ((TYPE == 2 && a.same && jk > ib + a.braOff) ||
                !in_shard(a.braBeg + ib, a.shardIdx, a.shardCnt))
              return false;
            const PairDev P = a.pairs[a.braBeg + ib], Q = a.pairs[a.ketBeg + jk];
            const bool pRef = TYPE == 1 || P.lex >= Q.lex;
            const int s1 = pRef ? P.s1 : Q.s1, s2 = pRef ? P.s2 : Q.s2;
            const int s3 = pRef ? Q.s1 : P.s1, s4 = pRef ? Q.s2 : P.s2;
            // shMax * Q12 * Q34 < thresh (:947-948, :2059-2061)
            const double bound = sh_max(a.norms, s1, s2, s3, s4, ns) *
                                 __ldg(a.qSS + P.s1 + (size_t)P.s2 * ns) *
                                 __ldg((TYPE == 1 ? a.qLL : a.qSS) + Q.s1 + (size_t)Q.s2 * ns);
            work = !a.screen || bound >= a.thresh;
            lo = work && a.mixed && bound < a.cut &&
                 fp32_range_ok(__ldg(a.pairRange + a.braBeg + ib),
                               __ldg(a.pairRange + a.ketBeg + jk),
                               a.lsum + (TYPE == 2 ? 4 : 2), 1, TYPE == 2);
            return true;
          });
}

// left product i^[a > 0] sigma_a d of a Pauli quaternion: a permutation of
// its components with signs
__device__ __forceinline__ Q4 left_sigma(const Q4& d, int a) {
  if (a == 0) return d;
  // sigma_k (s + v.sigma) = v_k + s sigma_k + i (k x v).sigma; times i
  auto neg = [](double2 z) { return make_double2(-z.x, -z.y); };
  if (a == 1) return Q4{ctimes_i(d.x), ctimes_i(d.s), d.z, neg(d.y)};
  if (a == 2) return Q4{ctimes_i(d.y), neg(d.z), ctimes_i(d.s), d.x};
  return Q4{ctimes_i(d.z), d.y, neg(d.x), ctimes_i(d.s)};
}
// sum_b (i f)^[b > 0] t_b sigma_b of four quaternions of 8 reals each
__device__ __forceinline__ Q4 right_sigmas(const double (&t)[4][8], double f) {
  auto q = [&](int b) {
    return Q4{make_double2(t[b][0], t[b][1]), make_double2(t[b][2], t[b][3]),
              make_double2(t[b][4], t[b][5]), make_double2(t[b][6], t[b][7])};
  };
  Q4 r = q(0);
#pragma unroll
  for (int b = 1; b < 4; b++) {
    const Q4 u = qsig(q(b), b);
    r.s = cadd(r.s, make_double2(-f * u.s.y, f * u.s.x));
    r.x = cadd(r.x, make_double2(-f * u.x.y, f * u.x.x));
    r.y = cadd(r.y, make_double2(-f * u.y.y, f * u.y.x));
    r.z = cadd(r.z, make_double2(-f * u.z.y, f * u.z.x));
  }
  return r;
}

// Digestion of one quartet's operator components (TYPE 1: M[(ab, op)][cd],
// TYPE 2: M[(ab, op)][(cd, op')]): the reference's updates with the sums
// over the other two component indices taken before the one atomic of each
// output element (J: over cd or ab; K: over the two contracted indices).
// Work units of the exchange are (target, its bra and ket component), shared
// by a few lanes where there are few; a unit sums m times the density over
// its elements per operator and applies the Pauli matrices once at its end.
// The element-wise digestion this replaces sent up to 36 atomics per element
// (11.7e9 for one Ag atom's LLSS; the L2 takes 185e9 scattered ones per
// second).
template <int TYPE>
__device__ __forceinline__ void rel_digest(const RelLaunch& a, const HgQuartet& z) {
  constexpr int NB = TYPE == 2 ? 4 : 1;
  const PairDev& P = *z.P;
  const int tid = threadIdx.x, nt = blockDim.x, ms = z.ms[0], msab = 4 * ms + 2;
  const size_t nc = a.ncart;
  auto ix = [nc](int r, int c) -> size_t { return (size_t)r + (size_t)c * nc; };
  const int na = ncart(z.la), nb = ncart(z.lb), ncc = ncart(z.lc), nd = ncart(z.ld);
  const int nAB = z.ab1 - z.ab0, nCD = z.cd1 - z.cd0;
  const bool dAB = P.shA == P.shB;
  const double s12d = dAB ? 1.0 : 2.0;
  // the back transform adds the transpose (Hermitian completion): a
  // contribution on a pair's own diagonal block is counted twice there
  const double w12 = dAB ? 0.5 : 1.0;
  // the densities the batch needs, in shared memory: Coulomb vectors in the
  // order of M's rows and columns, exchange blocks (A then B) x (C then D) of
  // each ket, 8 reals an element
  // (two more per bra component: its row starts on another bank)
  const int xrow = (ncc + nd) * 8 + 2, nx = (na + nb) * (ncc + nd);
  double* xk = z.st;
  double* xab = xk + (size_t)z.nk * (na + nb) * xrow;
  double* xcd = xab + 4 * na * nb;
  const double* const* const Xss = a.Xss;
  for (int u = tid; u < nAB * 4; u += nt) {
    const int ab = z.ab0 + (u >> 2), ai = ab / nb, bi = ab - ai * nb, op = u & 3;
    const size_t e = 2 * ix(P.cB + bi, P.cA + ai);
    xab[u] = op == 0 ? __ldg(Xss[0] + e) : -__ldg(Xss[op] + e + 1);
  }
  for (int u = tid; u < z.nk * nCD * NB; u += nt) {
    const int q = u / (nCD * NB), v = u - q * (nCD * NB), op = v % NB;
    const int cd = z.cd0 + v / NB, c = cd / nd, d = cd - c * nd;
    const size_t e = 2 * ix(z.Q[q].cB + d, z.Q[q].cA + c);
    xcd[u] = TYPE == 1 ? __ldg(a.Xll + e)
                       : (op == 0 ? __ldg(Xss[0] + e) : -__ldg(Xss[op] + e + 1));
  }
  if (a.exchange)
    for (int u = tid; u < z.nk * nx * 4; u += nt) {
      const int comp = u & 3, v = u >> 2, q = v / nx, r = v - q * nx;
      const int i = r / (ncc + nd), j = r - i * (ncc + nd);
      const int gB = i < na ? P.cA + i : P.cB + i - na;
      const int gK = j < ncc ? z.Q[q].cA + j : z.Q[q].cB + j - ncc;
      const size_t e = TYPE == 1 ? ix(gK, gB) : ix(gB, gK);
      reinterpret_cast<double2*>(xk + (q * (na + nb) + i) * xrow)[4 * j + comp] =
          ldz(a.Xk[comp], e);
    }
  __syncthreads();
  // Coulomb SS(1,2) from D(4,3) (:1145-1190, :2342-2380): unit (ket, ab, op)
  for (int uu = tid; uu < z.nk * nAB * 4; uu += nt) {
    const int q = uu / (nAB * 4), u = uu - q * (nAB * 4);
    if (!z.have(q)) continue;
    const PairDev& Q = z.Q[q];
    const double* m = z.M[0] + hg_row(u, ms) + q * z.cw[0];
    const double* x = xcd + q * nCD * NB;
    double s = 0.0;
    for (int k = 0; k < nCD * NB; k++) s += m[k] * x[k];
    const int ab = z.ab0 + (u >> 2), ai = ab / nb, bi = ab - ai * nb;
    if (s != 0.0)
      atomicAdd(a.Jss[u & 3] + ix(P.cA + ai, P.cB + bi),
                w12 * (Q.shA == Q.shB ? 1.0 : 2.0) * s);
  }
  // Coulomb LL(3,4) / SS(3,4) from D(2,1) (SSSS: when the pairs differ):
  // unit (ket, cd, op')
  for (int uu = tid; uu < z.nk * nCD * NB; uu += nt) {
    const int q = uu / (nCD * NB), u = uu - q * (nCD * NB);
    const PairDev& Q = z.Q[q];
    if (!z.have(q) || (TYPE == 2 && P.lex == Q.lex)) continue;
    const double* m = z.M[0] + q * z.cw[0] + u;
    double s = 0.0;
    for (int k = 0; k < nAB; k++, m += msab)
      s += m[0] * xab[4 * k] + m[ms] * xab[4 * k + 1] + m[2 * ms] * xab[4 * k + 2] +
           m[3 * ms] * xab[4 * k + 3];
    const int cd = z.cd0 + u / NB, c = cd / nd, d = cd - c * nd;
    if (s != 0.0)
      atomicAdd((TYPE == 1 ? a.Jll : a.Jss[u % NB]) + ix(Q.cA + c, Q.cB + d),
                (Q.shA == Q.shB ? 0.5 : 1.0) * s12d * s);
  }
  if (!a.exchange) return;
  // exchange targets (bra index of the output A or B, ket index C or D):
  // LLSS (:1200-1299) K(c,b) -= D(d,a) P, K(c,a) -= D(d,b) P^(-), ...;
  // SSSS (:2381-2445) K(a,d) -= P D(b,c) P, K(a,c), K(b,d), K(b,c)
  // Units of the four targets side by side, each shared by 2^sh lanes.
  const int both = (na + nb) * (ncc + nd);
  const int sh = hg_share(z.nk * both, na < nb ? na : nb);
  for (int uu = tid; uu < ((z.nk * both) << sh); uu += nt) {
    const int part = uu & ((1 << sh) - 1), v = uu >> sh, q = v / both, r = v - q * both;
    const int kO2 = r / (na + nb), bO2 = r - kO2 * (na + nb);
    const bool outA = bO2 < na, outC = kO2 < ncc;
    const PairDev& Q = z.Q[q];
    if (!z.have(q) || (dAB && outA == (TYPE == 1)) ||
        (Q.shA == Q.shB && outC == (TYPE == 2)))
      continue;
    const int bO = outA ? bO2 : bO2 - na, kO = outC ? kO2 : kO2 - ncc;
    const double f1 = TYPE == 1 ? (outA ? -1.0 : 1.0) : (outA ? 1.0 : -1.0);
    const double f2 = TYPE == 1 ? f1 : (outC ? -1.0 : 1.0);
    const int ni = outA ? nb : na, ki = outC ? nd : ncc;  // contracted components
    const int abI = outA ? 1 : nb, cdI = outC ? 1 : nd;   // their steps in ab and cd
    const int ab0 = (outA ? bO * nb : bO) - z.ab0, cd0 = (outC ? kO * nd : kO) - z.cd0;
    const double* Mq = z.M[0] + q * z.cw[0];
    const double* xq = xk + (q * (na + nb) + (outA ? na : 0)) * xrow + (outC ? ncc : 0) * 8;
    int k0, k1;  // the contracted ket components in the chunk
    hg_range(cd0, cdI, ki, nCD, k0, k1);
    double t[4][8];
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int k = 0; k < 8; k++) t[b][k] = 0.0;
    bool any = false;
#pragma unroll 1
    for (int bI = part; bI < ni; bI += 1 << sh) {
      const int ab = ab0 + bI * abI;
      if (ab < 0 || ab >= nAB) continue;
      const double* m = Mq + ab * msab + NB * (cd0 + k0 * cdI);
      const double* xr = xq + bI * xrow + k0 * 8;
      any = any || k0 < k1;
#pragma unroll 1
      for (int kI = k0; kI < k1; kI++, m += NB * cdI, xr += 8) {
        const double2* x2 = reinterpret_cast<const double2*>(xr);
        const Q4 d{x2[0], x2[1], x2[2], x2[3]};
        if (TYPE == 1) {
          // (D (m0 + i f m.sigma)): per operator m_op D
#pragma unroll
          for (int op = 0; op < 4; op++) {
            const double v = m[op * ms];
            t[op][0] += v * d.s.x; t[op][1] += v * d.s.y;
            t[op][2] += v * d.x.x; t[op][3] += v * d.x.y;
            t[op][4] += v * d.y.x; t[op][5] += v * d.y.y;
            t[op][6] += v * d.z.x; t[op][7] += v * d.z.y;
          }
        } else {
#pragma unroll
          for (int op = 0; op < 4; op++) {
            const Q4 l = left_sigma(d, op);
            const double2 m01 = *reinterpret_cast<const double2*>(m + op * ms);
            const double2 m23 = *reinterpret_cast<const double2*>(m + op * ms + 2);
            const double g = op == 0 ? 1.0 : f1;
            const double v[4] = {g * m01.x, g * m01.y, g * m23.x, g * m23.y};
#pragma unroll
            for (int b = 0; b < 4; b++) {
              t[b][0] += v[b] * l.s.x; t[b][1] += v[b] * l.s.y;
              t[b][2] += v[b] * l.x.x; t[b][3] += v[b] * l.x.y;
              t[b][4] += v[b] * l.y.x; t[b][5] += v[b] * l.y.y;
              t[b][6] += v[b] * l.z.x; t[b][7] += v[b] * l.z.y;
            }
          }
        }
      }
    }
    const Q4 k4 = right_sigmas(t, f2);
    double o8[8] = {k4.s.x, k4.s.y, k4.x.x, k4.x.y, k4.y.x, k4.y.y, k4.z.x, k4.z.y};
    if (sh > 0) {
#pragma unroll
      for (int k = 0; k < 8; k++) o8[k] = hg_group_sum(o8[k], sh);
      any = part == 0;
    }
    if (!any) continue;
    const int gO = (outA ? P.cA : P.cB) + bO, gP = (outC ? Q.cA : Q.cB) + kO;
    const size_t e = 2 * (TYPE == 1 ? ix(gP, gO) : ix(gO, gP));
    const double w = TYPE == 2 && P.lex == Q.lex ? -0.5 : -1.0;
#pragma unroll
    for (int k = 0; k < 8; k++) atomicAdd(a.K[k >> 1] + e + (k & 1), w * o8[k]);
  }
}

template <int TYPE>
struct RelDig {
  using Args = RelLaunch;
  static constexpr int NP = 1;
  static constexpr int ABU = 4, CDU = TYPE == 2 ? 4 : 16;  // components per 16-row tile
  __host__ __device__ static constexpr int tb(int) { return HG_SPIN; }
  __host__ __device__ static constexpr int tk(int) { return TYPE == 2 ? HG_SPIN : HG_PLAIN; }
  __host__ __device__ static constexpr int rtu(int) { return 1; }
  __host__ __device__ static constexpr int ctu(int) { return 1; }
  __host__ __device__ static int stage(int la, int lb, int lc, int ld, int nk) {
    return nk * ((ncart(la) + ncart(lb)) * ((ncart(lc) + ncart(ld)) * 8 + 2) +
                 ncart(lc) * ncart(ld) * (TYPE == 2 ? 4 : 1)) +
           ncart(la) * ncart(lb) * 4;
  }
  static __device__ __forceinline__ void digest(const RelLaunch& a, const HgQuartet& z) {
    rel_digest<TYPE>(a, z);
  }
};

// One class pair: planning pass and engine.
template <int TYPE>
cqf_status launch_rel(cqf_basis* B, const RelLaunch& a, int cb, int ck, const HgRegion& r,
                      cudaStream_t st) {
  return hg_contract<RelDig<TYPE>>(
      B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a, st,
      [&](const HgPart& p, uint2* masks, int* list64, int* list32, unsigned* lcount, unsigned gp) {
        rel_plan_kernel<TYPE><<<gp, 256, 0, st>>>(p.of(a), masks, list64, list32, lcount);
      });
}

// ------------------------------------------------------------------ Gaunt
// The Gaunt term -alpha_1.alpha_2 / r12 (direct4C_libcint.hpp:2833-3907).
// The reference runs over unordered pairs of (differentiated, other) shell
// pairs X = (s2, s1), Y = (s3, s4) with the integrals (m d_j n | d_l k l).
// Here an unordered quartet of unordered significant pairs {P, Q}
// (P = (A, B), Q = (C, D)) gives, per Cartesian element, the 36 blocks (A B with d_j on A or B | C D with d_l on C or D) at once: the
// four (or, for P = Q, three) reference quartets {X, Y} the placements
// make, each screened on its own by shMax Q^G(X) Q^G(Y).  Per element and
// surviving quartet, in the reference's orientation (X >= Y as (deriv,
// other) shell indices), its update sites and conditions with T and, for
// the image, T^T -- the four update kinds as Pauli-algebra maps of the
// invariants t = tr T, tau (cross vector) and S' = T + T^T - t:
//   LL exchange from SS:  3 (d0 t - i d.tau),   -(i d0 tau + S' d)
//   SS exchange from LL:  3 d0 t - i d.tau,     -3 i d0 tau - S' d
//   LS Coulomb from SL (1), LS (2):  (d1_0 - d2_0) t + i (d1 + d2).tau,
//                                     i (d2_0 - d1_0) tau + (T^T - t)(d1 + d2)
//   LS exchange from SL:  d0 t - i d.tau,       i d0 tau + S' d - 4 T^T d
// LL and SS exchange are accumulated in the lower shell triangle (half
// weight on diagonal shell blocks) and completed as B + B^H by the back
// transform, the reference's "upper = conj(lower)" (:3833-3858).  FP64.
struct GauntLaunch {
  const PairDev* pairs;
  const PrimPairDev* pp;
  const ShellDev* shells;
  const double* prim;
  const double* boys;
  int braBeg, nBra, braOff, ketBeg, nKet, same;
  int screen;
  double thresh;
  const double* norms;  // max shell-block norms of the 16 exchange densities
  const double* qG;     // Gaunt Schwarz, qG[deriv + other * nshell]
  int nShell, ncart, exchange;
  const double* Xll[4];  // Cartesian complex densities: XLLM*, XSSM*, CLSM*, CSLM*, XSLM*
  const double* Xss[4];
  const double* Cls[4];
  const double* Csl[4];
  const double* Xsl[4];
  double* Kll[4];  // complex accumulators: LL / SS exchange, LS Coulomb, LS exchange
  double* Kss[4];
  double* Jls[4];
  double* Kls[4];
  int shardIdx, shardCnt;  // bra pairs p with p % shardCnt == shardIdx only
  unsigned long long* counters;
};

struct GInv {
  double T[3][3], t, tau[3], S[3][3];
};
__device__ __forceinline__ void gaunt_inv(const double* v, bool tr, GInv& g) {
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int l = 0; l < 3; l++) g.T[j][l] = tr ? v[3 * l + j] : v[3 * j + l];
  g.t = g.T[0][0] + g.T[1][1] + g.T[2][2];
  g.tau[0] = g.T[1][2] - g.T[2][1];
  g.tau[1] = g.T[2][0] - g.T[0][2];
  g.tau[2] = g.T[0][1] - g.T[1][0];
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int l = 0; l < 3; l++) g.S[j][l] = g.T[j][l] + g.T[l][j] - (j == l ? g.t : 0.0);
}

struct Z4 {  // Pauli components (s, x, y, z), complex
  double2 c[4];
};
__device__ __forceinline__ Z4 ld4(const double* const* X, size_t e) {
  return Z4{{ldz(X[0], e), ldz(X[1], e), ldz(X[2], e), ldz(X[3], e)}};
}
__device__ __forceinline__ void add4(double* const* A, size_t e, const Z4& v, double w) {
#pragma unroll
  for (int k = 0; k < 4; k++) addz(A[k], e, v.c[k], w);
}
__device__ __forceinline__ double2 cscale(double2 a, double f) {
  return make_double2(a.x * f, a.y * f);
}
// sum_x w[x] d_x over the vector part
__device__ __forceinline__ double2 vdot(const Z4& d, const double* w) {
  return make_double2(d.c[1].x * w[0] + d.c[2].x * w[1] + d.c[3].x * w[2],
                      d.c[1].y * w[0] + d.c[2].y * w[1] + d.c[3].y * w[2]);
}
// sum_y M[x][y] d_y (trans: M[y][x])
__device__ __forceinline__ double2 vmat(const Z4& d, const double (*M)[3], int x, bool trans) {
  double2 r = make_double2(0.0, 0.0);
#pragma unroll
  for (int y = 0; y < 3; y++) {
    const double m = trans ? M[y][x] : M[x][y];
    r.x += m * d.c[1 + y].x;
    r.y += m * d.c[1 + y].y;
  }
  return r;
}

__device__ __forceinline__ Z4 gaunt_ll(const GInv& g, const Z4& d) {
  Z4 r;
  r.c[0] = cscale(csub(cscale(d.c[0], g.t), ctimes_i(vdot(d, g.tau))), 3.0);
#pragma unroll
  for (int x = 0; x < 3; x++)
    r.c[1 + x] = cscale(cadd(ctimes_i(cscale(d.c[0], g.tau[x])), vmat(d, g.S, x, false)), -1.0);
  return r;
}
__device__ __forceinline__ Z4 gaunt_ss(const GInv& g, const Z4& d) {
  Z4 r;
  r.c[0] = csub(cscale(d.c[0], 3.0 * g.t), ctimes_i(vdot(d, g.tau)));
#pragma unroll
  for (int x = 0; x < 3; x++)
    r.c[1 + x] = csub(ctimes_i(cscale(d.c[0], -3.0 * g.tau[x])), vmat(d, g.S, x, false));
  return r;
}
__device__ __forceinline__ Z4 gaunt_cls(const GInv& g, const Z4& d1, const Z4& d2) {
  Z4 e;
  e.c[0] = csub(d1.c[0], d2.c[0]);
#pragma unroll
  for (int x = 1; x < 4; x++) e.c[x] = cadd(d1.c[x], d2.c[x]);
  Z4 r;
  r.c[0] = cadd(cscale(e.c[0], g.t), ctimes_i(vdot(e, g.tau)));
#pragma unroll
  for (int x = 0; x < 3; x++)
    r.c[1 + x] = cadd(ctimes_i(cscale(e.c[0], -g.tau[x])),
                      csub(vmat(e, g.T, x, true), cscale(e.c[1 + x], g.t)));
  return r;
}
__device__ __forceinline__ Z4 gaunt_xls(const GInv& g, const Z4& d) {
  Z4 r;
  r.c[0] = csub(cscale(d.c[0], g.t), ctimes_i(vdot(d, g.tau)));
#pragma unroll
  for (int x = 0; x < 3; x++)
    r.c[1 + x] = cadd(ctimes_i(cscale(d.c[0], g.tau[x])),
                      csub(vmat(d, g.S, x, false), cscale(vmat(d, g.T, x, true), 4.0)));
  return r;
}

// The update sites of one reference quartet (s1 s2 | s3 s4) at element
// (m1 m2 | m3 m4) (Cartesian AO indices), T = v (row: the s2 direction).
__device__ __forceinline__ void gaunt_sites(const GauntLaunch& a, const double* v, int s1, int s2,
                                            int s3, int s4, int m1, int m2, int m3, int m4) {
  const size_t nc = a.ncart;
  auto ix = [nc](int r, int c) -> size_t { return (size_t)r + (size_t)c * nc; };
  GInv T, Tt;
  gaunt_inv(v, false, T);
  gaunt_inv(v, true, Tt);
  const bool img = (s1 != s4) || (s2 != s3);
  if (a.exchange) {
    const double w14 = (s1 == s4) ? 0.5 : 1.0, w23 = (s2 == s3) ? 0.5 : 1.0;
    if (s1 >= s4) add4(a.Kll, ix(m1, m4), gaunt_ll(T, ld4(a.Xss, ix(m2, m3))), w14);
    if (s1 < s4 || (s1 == s4 && s2 != s3))
      add4(a.Kll, ix(m4, m1), gaunt_ll(Tt, ld4(a.Xss, ix(m3, m2))), w14);
    add4(a.Kss, ix(m2, m3), gaunt_ss(Tt, ld4(a.Xll, ix(m1, m4))), w23);
    if (s1 != s4 && s2 == s3) add4(a.Kss, ix(m3, m2), gaunt_ss(T, ld4(a.Xll, ix(m4, m1))), 0.5);
  }
  add4(a.Jls, ix(m1, m2), gaunt_cls(T, ld4(a.Csl, ix(m3, m4)), ld4(a.Cls, ix(m4, m3))), 1.0);
  if (img)
    add4(a.Jls, ix(m4, m3), gaunt_cls(Tt, ld4(a.Csl, ix(m2, m1)), ld4(a.Cls, ix(m1, m2))), 1.0);
  if (a.exchange) {
    add4(a.Kls, ix(m1, m3), gaunt_xls(T, ld4(a.Xsl, ix(m2, m4))), 1.0);
    if (img) add4(a.Kls, ix(m4, m2), gaunt_xls(Tt, ld4(a.Xsl, ix(m3, m1))), 1.0);
  }
}

// ------------------------------------------------ gauge (Breit) term
// The gauge part of the Breit interaction (direct4C_libcint.hpp:3908-5160):
// the GAUNT list, quartets and update sites with the kernel
// K_ii' = -r_i r_i' / r12^3 between the densities rho^i, rho^i' in place of
// Gaunt's -delta_ii' / r12.  Per element
//   V[i][i'][j][l] = (m d_j n | K_ii' | d_l k l)
//                  = -delta_ii' T[j][l] + (m d_j n | d_i d_i' r12 | d_l k l)
// (r_i r_i' / r^3 = delta_ii' / r - d_i d_i' r), and with
// W(M, D) = sum_jl M_jl s_j D s_l (the closed form above) the update kinds
// are, Q_ij = s_i s_j:
//   LL exchange from SS:  -sum_ii' s_i W(V^{ii'}, D) s_i'
//   SS exchange from LL:  -sum_jl  s_j W(V_{jl}, D) s_l     (M_ii' = V^{ii'}_jl)
//   LS Coulomb from SL (1), LS (2):  1/2 sum_ij Q_ij sum_i'l V^{ii'}_jl
//                                     (tr[Q_li' D2] - tr[Q_i'l D1])
//   LS exchange from SL:  sum_il s_i W(N_il, D) s_l         (N_ji' = V^{ii'}_jl)
// (for V = -delta T they are the Gaunt maps).  The image takes V with j
// and l exchanged (the kernel is even in r12 and symmetric in i, i').
struct GVd {
  double v[3][3][3][3];  // [i][i'][j][l]
};
__device__ __forceinline__ Q4 qunit(int a) {  // sigma_a
  Q4 r{make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)};
  if (a == 0) r.x = make_double2(1, 0);
  else if (a == 1) r.y = make_double2(1, 0);
  else r.z = make_double2(1, 0);
  return r;
}
__device__ __forceinline__ void zacc(Z4& a, const Q4& b, double f) {
  a.c[0] = cadd(a.c[0], cscale(b.s, f));
  a.c[1] = cadd(a.c[1], cscale(b.x, f));
  a.c[2] = cadd(a.c[2], cscale(b.y, f));
  a.c[3] = cadd(a.c[3], cscale(b.z, f));
}
// W(M, D) = sum_jl M_jl s_j D s_l = d0 t - i d.tau + (i d0 tau + S' d).s
__device__ __forceinline__ Q4 w_map(const double (*M)[3], const Z4& d) {
  GInv g;
  double v[9];
#pragma unroll
  for (int k = 0; k < 9; k++) v[k] = M[k / 3][k % 3];
  gaunt_inv(v, false, g);
  Q4 r;
  r.s = csub(cscale(d.c[0], g.t), ctimes_i(vdot(d, g.tau)));
  double2 w[3];
#pragma unroll
  for (int x = 0; x < 3; x++) w[x] = cadd(ctimes_i(cscale(d.c[0], g.tau[x])), vmat(d, g.S, x, false));
  r.x = w[0];
  r.y = w[1];
  r.z = w[2];
  return r;
}
__device__ Z4 gauge_ll(const GVd& V, const Z4& d) {
  Z4 r{{make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)}};
#pragma unroll 1
  for (int i = 0; i < 3; i++)
#pragma unroll 1
    for (int ip = 0; ip < 3; ip++)
      zacc(r, qmul(qmul(qunit(i), w_map(V.v[i][ip], d)), qunit(ip)), -1.0);
  return r;
}
__device__ Z4 gauge_ss(const GVd& V, const Z4& d) {
  Z4 r{{make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)}};
#pragma unroll 1
  for (int j = 0; j < 3; j++)
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      double M[3][3];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int ip = 0; ip < 3; ip++) M[i][ip] = V.v[i][ip][j][l];
      zacc(r, qmul(qmul(qunit(j), w_map(M, d)), qunit(l)), -1.0);
    }
  return r;
}
__device__ Z4 gauge_xls(const GVd& V, const Z4& d) {
  Z4 r{{make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)}};
#pragma unroll 1
  for (int i = 0; i < 3; i++)
#pragma unroll 1
    for (int l = 0; l < 3; l++) {
      double M[3][3];
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int ip = 0; ip < 3; ip++) M[j][ip] = V.v[i][ip][j][l];
      zacc(r, qmul(qmul(qunit(i), w_map(M, d)), qunit(l)), 1.0);
    }
  return r;
}
// tr[s_a s_b D] = 2 (delta_ab d0 + i eps_abm d_m)
__device__ __forceinline__ double2 tr_qq(int a, int b, const Z4& d) {
  if (a == b) return cscale(d.c[0], 2.0);
  const int m = 3 - a - b;
  const double e = (b == (a + 1) % 3) ? 2.0 : -2.0;
  return ctimes_i(cscale(d.c[1 + m], e));
}
__device__ Z4 gauge_cls(const GVd& V, const Z4& d1, const Z4& d2) {
  double2 sv[3][3];  // [l][i']
#pragma unroll 1
  for (int l = 0; l < 3; l++)
#pragma unroll 1
    for (int ip = 0; ip < 3; ip++) sv[l][ip] = csub(tr_qq(l, ip, d2), tr_qq(ip, l, d1));
  Z4 r{{make_double2(0, 0), make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)}};
#pragma unroll 1
  for (int i = 0; i < 3; i++)
#pragma unroll 1
    for (int j = 0; j < 3; j++) {
      double2 c = make_double2(0, 0);
#pragma unroll
      for (int ip = 0; ip < 3; ip++)
#pragma unroll
        for (int l = 0; l < 3; l++) c = cadd(c, cscale(sv[l][ip], V.v[i][ip][j][l]));
      c = cscale(c, 0.5);
      // Q_ij = delta_ij + i eps_ijm s_m
      if (i == j) r.c[0] = cadd(r.c[0], c);
      else {
        const int m = 3 - i - j;
        const double e = (j == (i + 1) % 3) ? 1.0 : -1.0;
        r.c[1 + m] = cadd(r.c[1 + m], ctimes_i(cscale(c, e)));
      }
    }
  return r;
}

// The gauge update sites of one reference quartet at one element (as
// gaunt_sites), V and its image Vt.
__device__ void gauge_sites(const GauntLaunch& a, const GVd& V, const GVd& Vt, int s1, int s2,
                            int s3, int s4, int m1, int m2, int m3, int m4) {
  const size_t nc = a.ncart;
  auto ix = [nc](int r, int c) -> size_t { return (size_t)r + (size_t)c * nc; };
  const bool img = (s1 != s4) || (s2 != s3);
  if (a.exchange) {
    const double w14 = (s1 == s4) ? 0.5 : 1.0, w23 = (s2 == s3) ? 0.5 : 1.0;
    if (s1 >= s4) add4(a.Kll, ix(m1, m4), gauge_ll(V, ld4(a.Xss, ix(m2, m3))), w14);
    if (s1 < s4 || (s1 == s4 && s2 != s3))
      add4(a.Kll, ix(m4, m1), gauge_ll(Vt, ld4(a.Xss, ix(m3, m2))), w14);
    add4(a.Kss, ix(m2, m3), gauge_ss(V, ld4(a.Xll, ix(m1, m4))), w23);
    if (s1 != s4 && s2 == s3) add4(a.Kss, ix(m3, m2), gauge_ss(Vt, ld4(a.Xll, ix(m4, m1))), 0.5);
  }
  add4(a.Jls, ix(m1, m2), gauge_cls(V, ld4(a.Csl, ix(m3, m4)), ld4(a.Cls, ix(m4, m3))), 1.0);
  if (img)
    add4(a.Jls, ix(m4, m3), gauge_cls(Vt, ld4(a.Csl, ix(m2, m1)), ld4(a.Cls, ix(m1, m2))), 1.0);
  if (a.exchange) {
    add4(a.Kls, ix(m1, m3), gauge_xls(V, ld4(a.Xsl, ix(m2, m4))), 1.0);
    if (img) add4(a.Kls, ix(m4, m2), gauge_xls(Vt, ld4(a.Xsl, ix(m3, m1))), 1.0);
  }
}

// bra component pairs per unit of work of the gauge kernel (its
// accumulator holds 7 x 36 blocks of each)
__host__ __device__ constexpr int gauge_abch(int lm) { return lm <= 2 ? 9 : 4; }

// The reference quartets of {P, Q} that survive their own screen: bit
// 2 pb + pk, derivative on B (pb) / D (pk) instead of A / C.
__device__ __forceinline__ unsigned gaunt_alive(const GauntLaunch& a, const PairDev& P,
                                                const PairDev& Q) {
  const int ns = a.nShell;
  const double shMax = sh_max(a.norms, P.s1, P.s2, Q.s1, Q.s2, ns);
  const bool samePQ = P.lex == Q.lex;
  unsigned alive = 0;
#pragma unroll
  for (int pb = 0; pb < 2; pb++)
#pragma unroll
    for (int pk = 0; pk < 2; pk++) {
      if ((pb && P.shA == P.shB) || (pk && Q.shA == Q.shB) || (samePQ && pb > pk)) continue;
      const int xd = pb ? P.shB : P.shA, xo = pb ? P.shA : P.shB;
      const int yd = pk ? Q.shB : Q.shA, yo = pk ? Q.shA : Q.shB;
      const double bound = shMax * __ldg(a.qG + xd + (size_t)xo * ns) *
                           __ldg(a.qG + yd + (size_t)yo * ns);
      if (!a.screen || bound >= a.thresh) alive |= 1u << (2 * pb + pk);
    }
  return alive;
}

__global__ void __launch_bounds__(256)
    gaunt_plan_kernel(const GauntLaunch a, uint2* __restrict__ masks, int* __restrict__ list64,
                      int* __restrict__ list32, unsigned* __restrict__ lcount) {
  hg_plan(a.nBra, a.nKet, masks, list64, list32, lcount, a.counters,
          [&](int ib, int jk, bool& work, bool&) {
            if ((a.same && jk > ib + a.braOff) ||
                !in_shard(a.braBeg + ib, a.shardIdx, a.shardCnt))
              return false;
            work = gaunt_alive(a, a.pairs[a.braBeg + ib], a.pairs[a.ketBeg + jk]) != 0;
            return true;
          });
}

// Gaunt on the engine: M[(ab, pb, j)][(cd, pk, l)], every surviving reference
// quartet of every element one unit of work.
struct GauntDig {
  using Args = GauntLaunch;
  static constexpr int NP = 1, ABU = 8, CDU = 8;  // 8 component pairs: three row tiles
  __host__ __device__ static constexpr int tb(int) { return HG_D6; }
  __host__ __device__ static constexpr int tk(int) { return HG_D6; }
  __host__ __device__ static constexpr int rtu(int) { return 3; }
  __host__ __device__ static constexpr int ctu(int) { return 3; }
  __host__ __device__ static constexpr int stage(int, int, int, int, int) { return 0; }
  static __device__ __forceinline__ void digest(const GauntLaunch& a, const HgQuartet& z) {
    const PairDev& P = *z.P;
    const int nb = ncart(z.lb), nd = ncart(z.ld), nCD = z.cd1 - z.cd0;
    const int per = (z.ab1 - z.ab0) * nCD * 4;
    for (int uu = threadIdx.x; uu < z.nk * per; uu += blockDim.x) {
      const int q = uu / per, u = uu - q * per;
      const PairDev& Q = z.Q[q];
      const int blk = u & 3, e = u >> 2, r = e / nCD, c = e - r * nCD;
      if (!z.have(q) || !(gaunt_alive(a, P, Q) & (1u << blk))) continue;
      const int pb = blk >> 1, pk = blk & 1;
      const int ab = z.ab0 + r, cd = z.cd0 + c;
      const int gA = P.cA + ab / nb, gB = P.cB + ab % nb;
      const int gC = Q.cA + cd / nd, gD = Q.cB + cd % nd;
      const int xd = pb ? P.shB : P.shA, xo = pb ? P.shA : P.shB;
      const int yd = pk ? Q.shB : Q.shA, yo = pk ? Q.shA : Q.shB;
      const int xdA = pb ? gB : gA, xoA = pb ? gA : gB;
      const int ydA = pk ? gD : gC, yoA = pk ? gC : gD;
      // the reference's orientation: bra X (j on X) or Y (j on Y)
      const bool xb = xd > yd || (xd == yd && xo >= yo);
      const double* m = z.M[0] + q * z.cw[0] + c * 6 + pk * 3;
      const int r0 = r * 6 + pb * 3, ms = z.ms[0];
      double v[9];
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int l = 0; l < 3; l++)
          v[3 * j + l] = xb ? m[hg_row(r0 + j, ms) + l] : m[hg_row(r0 + l, ms) + j];
      if (xb) gaunt_sites(a, v, xo, xd, yd, yo, xoA, xdA, ydA, yoA);
      else gaunt_sites(a, v, yo, yd, xd, xo, yoA, ydA, xdA, xoA);
    }
  }
};

// One thread per (quartet {P, Q}, unit); units = ket component pairs (c, d)
// x slices of bra component pairs, split over nsplit threads.  Seven
// operators -- 1 / r12 and d_i d_i' r12 for the six pairs i <= i' -- each a
// pass over the primitive pairs (the r12 passes on the auxiliary functions
// of r12_aux, the Hermite index shifted by e_i + e_i').
template <int LM>
__global__ void __launch_bounds__(REL_THREADS)
    gauge_kernel(const GauntLaunch a, int la, int lb, int lc, int ld, int nsplit, int nslice) {
  const int ib = blockIdx.x;
  if (!in_shard(a.braBeg + ib, a.shardIdx, a.shardCnt)) return;  // another shard's bra
  const int split = blockIdx.y % nsplit;
  const int jk = (blockIdx.y / nsplit) * REL_THREADS + threadIdx.x;
  const bool visited = jk < a.nKet && !(a.same && jk > ib);
  const PairDev P = a.pairs[a.braBeg + ib];
  PairDev Q = P;
  unsigned alive = 0;
  if (visited) {
    Q = a.pairs[a.ketBeg + jk];
    alive = gaunt_alive(a, P, Q);
  }
  if (split == 0) {
    const unsigned mask = __activemask();
    const unsigned bv = __ballot_sync(mask, visited), bw = __ballot_sync(mask, alive != 0);
    if ((int)(threadIdx.x & 31) == __ffs(mask) - 1) {
      if (bv) atomicAdd(a.counters + 0, (unsigned long long)__popc(bv));
      if (bv & ~bw) atomicAdd(a.counters + 1, (unsigned long long)__popc(bv & ~bw));
      if (bw) atomicAdd(a.counters + 3, (unsigned long long)__popc(bw));
    }
  }
  if (!alive) return;

  constexpr int NOP = 7;
  constexpr int E1 = (LM + 2) * (LM + 2) * (2 * LM + 3);
  constexpr int HB = nherm(2 * LM + 1);
  constexpr int HL = nherm(4 * LM + 4);
  constexpr int FL = 2 * LM + 3;
  constexpr int ABCH = gauge_abch(LM);
  const int na = ncart(la), nb = ncart(lb), ncc = ncart(lc), nd = ncart(ld);
  const int nab = na * nb, ncd = ncc * nd;
  const ShellDev SA = a.shells[P.shA], SB = a.shells[P.shB];
  const ShellDev SC = a.shells[Q.shA], SD = a.shells[Q.shB];
  const int Lb = la + lb + 1, Lk = lc + ld + 1;
  // which placements some surviving quartet needs
  const bool needB[2] = {(alive & 3u) != 0, (alive & 12u) != 0};
  const bool needK[2] = {(alive & 5u) != 0, (alive & 10u) != 0};

  double Ea[3][E1], Ec[3][E1];
  double G[6][HB];  // [pk * 3 + l]
  double Rv[HL];
  double F[4 * LM + 5];
  double acc[ABCH * NOP * 36];
  double fa[3][3][FL], fc[3][3][FL];
  int nfa[3][3], nfc[3][3];

#pragma unroll 1
  for (int u = split; u < ncd * nslice; u += nsplit) {
    const int cd = u / nslice, sl = u % nslice;
    const int ab0 = sl * ABCH, ab1 = min(nab, ab0 + ABCH);
    if (ab0 >= ab1) continue;
    const int c = cd / nd, d = cd % nd;
    const int ci[3] = {cart_lx(lc, c), cart_ly(lc, c), cart_lz(lc, c)};
    const int di[3] = {cart_lx(ld, d), cart_ly(ld, d), cart_lz(ld, d)};
#pragma unroll 1
    for (int k = 0; k < (ab1 - ab0) * NOP * 36; k++) acc[k] = 0.0;
#pragma unroll 1
    for (int op = 0; op < NOP; op++) {
      int oi = -1, oj = -1;
      if (op > 0) op_pair(op - 1, oi, oj);
      const int sx = (oi == 0) + (oj == 0), sy = (oi == 1) + (oj == 1), sz = (oi == 2) + (oj == 2);
      const int L = Lb + Lk + (op > 0 ? 2 : 0);
#pragma unroll 1
      for (int ip = 0; ip < P.npp; ip++) {
        const PrimPairDev& A = a.pp[P.pp_off + ip];
        double ea, eb;
        pair_exps(SA, SB, a.prim, A, ea, eb);
#pragma unroll 1
        for (int x = 0; x < 3; x++)
          hermite_E_rt<double, LM + 1>(la + 1, lb + 1, A.o2p, A.PA[x], A.PB[x], Ea[x]);
#pragma unroll 1
        for (int k = 0; k < 6; k++)
#pragma unroll 1
          for (int h = 0; h < nherm(Lb); h++) G[k][h] = 0.0;
#pragma unroll 1
        for (int iq = 0; iq < Q.npp; iq++) {
          const PrimPairDev& Bq = a.pp[Q.pp_off + iq];
          double ec, ed;
          pair_exps(SC, SD, a.prim, Bq, ec, ed);
#pragma unroll 1
          for (int x = 0; x < 3; x++)
            hermite_E_rt<double, LM + 1>(lc + 1, ld + 1, Bq.o2p, Bq.PA[x], Bq.PB[x], Ec[x]);
          const double X = A.P[0] - Bq.P[0], Y = A.P[1] - Bq.P[1], Z = A.P[2] - Bq.P[2];
          const double pq = A.p + Bq.p, alpha = A.p * Bq.p / pq;
          double pref = PI52X2 / sqrt(pq) * A.Kp * Bq.Kp;
          const double Targ = alpha * (X * X + Y * Y + Z * Z);
          boys_rt<double>(L, Targ, F, a.boys);
          if (op > 0) {
            r12_aux(L, Targ, F);
            pref /= 2.0 * alpha;
          }
          hermite_R_rt<double>(L, alpha, X, Y, Z, F, Rv);
#pragma unroll 1
          for (int x = 0; x < 3; x++)
#pragma unroll 1
            for (int ty = 0; ty < 3; ty++) {
              if (ty > 0 && !needK[ty - 1]) continue;
              nfc[x][ty] = axis_factor<double>(Ec[x], ld + 1, lc + ld + 3, ci[x], di[x], ty,
                                               2.0 * ec, 2.0 * ed, fc[x][ty]);
#pragma unroll 1
              for (int t = 1; t < nfc[x][ty]; t += 2) fc[x][ty][t] = -fc[x][ty][t];
            }
#pragma unroll 1
          for (int pk = 0; pk < 2; pk++) {
            if (!needK[pk]) continue;
#pragma unroll 1
            for (int l = 0; l < 3; l++) {
              const int tx = (l == 0) ? 1 + pk : 0, ty = (l == 1) ? 1 + pk : 0,
                        tz = (l == 2) ? 1 + pk : 0;
              ket_add<double>(G[pk * 3 + l], pref, fc[0][tx], nfc[0][tx], fc[1][ty],
                              nfc[1][ty], fc[2][tz], nfc[2][tz], Lb, Rv, sx, sy, sz);
            }
          }
        }
#pragma unroll 1
        for (int ab = ab0; ab < ab1; ab++) {
          const int ai = ab / nb, bi = ab % nb;
          const int ax[3] = {cart_lx(la, ai), cart_ly(la, ai), cart_lz(la, ai)};
          const int bx[3] = {cart_lx(lb, bi), cart_ly(lb, bi), cart_lz(lb, bi)};
#pragma unroll 1
          for (int x = 0; x < 3; x++)
#pragma unroll 1
            for (int ty = 0; ty < 3; ty++) {
              if (ty > 0 && !needB[ty - 1]) continue;
              nfa[x][ty] = axis_factor<double>(Ea[x], lb + 1, la + lb + 3, ax[x], bx[x], ty,
                                               2.0 * ea, 2.0 * eb, fa[x][ty]);
            }
          double* m = acc + ((ab - ab0) * NOP + op) * 36;
#pragma unroll 1
          for (int pb = 0; pb < 2; pb++) {
            if (!needB[pb]) continue;
#pragma unroll 1
            for (int j = 0; j < 3; j++) {
              const int tx = (j == 0) ? 1 + pb : 0, ty = (j == 1) ? 1 + pb : 0,
                        tz = (j == 2) ? 1 + pb : 0;
#pragma unroll 1
              for (int pk = 0; pk < 2; pk++) {
                if (!(alive & (1u << (2 * pb + pk)))) continue;
#pragma unroll 1
                for (int l = 0; l < 3; l++)
                  m[((pb * 3 + j) * 2 + pk) * 3 + l] +=
                      bra_dot<double>(fa[0][tx], nfa[0][tx], fa[1][ty], nfa[1][ty], fa[2][tz],
                                      nfa[2][tz], G[pk * 3 + l]);
              }
            }
          }
        }
      }
    }
    // digestion: every surviving reference quartet of every element
    const int gC = Q.cA + c, gD = Q.cB + d;
#pragma unroll 1
    for (int ab = ab0; ab < ab1; ab++) {
      const int gA = P.cA + ab / nb, gB = P.cB + ab % nb;
      const double* m = acc + (ab - ab0) * NOP * 36;
#pragma unroll 1
      for (int pb = 0; pb < 2; pb++)
#pragma unroll 1
        for (int pk = 0; pk < 2; pk++) {
          if (!(alive & (1u << (2 * pb + pk)))) continue;
          const int xd = pb ? P.shB : P.shA, xo = pb ? P.shA : P.shB;
          const int yd = pk ? Q.shB : Q.shA, yo = pk ? Q.shA : Q.shB;
          const int xdA = pb ? gB : gA, xoA = pb ? gA : gB;
          const int ydA = pk ? gD : gC, yoA = pk ? gC : gD;
          const bool xb = xd > yd || (xd == yd && xo >= yo);
          // the reference's orientation: bra X (j on X) or Y (j on Y)
          auto comp = [&](int o, int j, int l) -> double {
            return xb ? m[o * 36 + ((pb * 3 + j) * 2 + pk) * 3 + l]
                      : m[o * 36 + ((pb * 3 + l) * 2 + pk) * 3 + j];
          };
          {
            GVd V, Vt;
#pragma unroll 1
            for (int k = 0; k < 6; k++) {
              int i, ip;
              op_pair(k, i, ip);
#pragma unroll 1
              for (int j = 0; j < 3; j++)
#pragma unroll 1
                for (int l = 0; l < 3; l++) {
                  double v = comp(1 + k, j, l), vt = comp(1 + k, l, j);
                  if (i == ip) {
                    v -= comp(0, j, l);
                    vt -= comp(0, l, j);
                  }
                  V.v[i][ip][j][l] = V.v[ip][i][j][l] = v;
                  Vt.v[i][ip][j][l] = Vt.v[ip][i][j][l] = vt;
                }
            }
            if (xb) gauge_sites(a, V, Vt, xo, xd, yd, yo, xoA, xdA, ydA, yoA);
            else gauge_sites(a, V, Vt, yo, yd, xd, xo, yoA, ydA, xdA, xoA);
          }
        }
    }
  }
}

void launch_gauge(const GauntLaunch& a, int la, int lb, int lc, int ld, cudaStream_t st) {
  if (a.nBra == 0 || a.nKet == 0) return;
  const int tiles = (a.nKet + REL_THREADS - 1) / REL_THREADS;
  const int lm = std::max(std::max(la, lb), std::max(lc, ld));
  const int nab = ncart(la) * ncart(lb);
  const int abch = gauge_abch(std::max(lm, 1));
  const int nslice = (nab + abch - 1) / abch;
  const long long quartets = (long long)a.nBra * a.nKet;
  const int units = ncart(lc) * ncart(ld) * nslice;
  int nsplit = (int)std::min<long long>(units, std::max<long long>(1, (1 << 18) / quartets));
  nsplit = std::max(1, std::min(nsplit, 65535 / tiles));
  dim3 grid(a.nBra, tiles * nsplit);
  if (lm <= 1) gauge_kernel<1><<<grid, REL_THREADS, 0, st>>>(a, la, lb, lc, ld, nsplit, nslice);
  else if (lm == 2)
    gauge_kernel<2><<<grid, REL_THREADS, 0, st>>>(a, la, lb, lc, ld, nsplit, nslice);
  else gauge_kernel<3><<<grid, REL_THREADS, 0, st>>>(a, la, lb, lc, ld, nsplit, nslice);
}

// ------------------------------------------------------------ 4C Schwarz
// Q^LL(a,b) = sqrt(max |(ab|ab)|) and Q^SS(a,b) = C2 sqrt(max over the 81
// components of |(dA dB ab|dA dB ab)|), both over every element of the
// spherical quartet block (direct4C_libcint.hpp:341-481).  Every (pair,
// component) is one unit of work for a group of threads, one Cartesian ket
// column per thread (rel_schwarz_kernel).

// Cartesian column out[(a*nb + b) * stride] += w (d ab | K | d cd) of the
// ket component pair (c, d) with derivative directions dir[0..3] (-1:
// none), summed over the bra primitive pairs ip = ip0, ip0 + ipStep, ...
// (shared memory, added atomically: several threads may share a column).
// K = 1 / r12, or d_opi d_opj r12 when opi >= 0.
template <int LM>
__device__ void deriv_column(int la, int lb, int lc, int ld, int c, int d, const int* dir,
                             const PairDev& P, const PairDev& Q, const PrimPairDev* pp,
                             const ShellDev* shells, const double* prim, const double* boys,
                             double* out, int stride, int ip0, int ipStep, int opi = -1,
                             int opj = -1, double w = 1.0) {
  constexpr int E1 = (LM + 2) * (LM + 2) * (2 * LM + 3);
  constexpr int HB = nherm(2 * LM + 2);
  constexpr int HL = nherm(4 * LM + 4);
  constexpr int FL = 2 * LM + 3;
  const int na = ncart(la), nb = ncart(lb);
  const int rb = (dir[0] >= 0 || dir[1] >= 0) ? 1 : 0, rk = (dir[2] >= 0 || dir[3] >= 0) ? 1 : 0;
  const int Lb = la + lb + (dir[0] >= 0) + (dir[1] >= 0);
  const int Lk = lc + ld + (dir[2] >= 0) + (dir[3] >= 0);
  const int sh[3] = {(opi == 0) + (opj == 0), (opi == 1) + (opj == 1), (opi == 2) + (opj == 2)};
  const int L = Lb + Lk + (opi >= 0 ? 2 : 0);
  const ShellDev SA = shells[P.shA], SB = shells[P.shB], SC = shells[Q.shA], SD = shells[Q.shB];
  const int ci[3] = {cart_lx(lc, c), cart_ly(lc, c), cart_lz(lc, c)};
  const int di[3] = {cart_lx(ld, d), cart_ly(ld, d), cart_lz(ld, d)};
  double Ea[3][E1], Ec[3][E1], G[HB], Rv[HL], F[4 * LM + 5], f[3][FL], g[3][FL];
  int nf[3], ng[3];
  for (int ip = ip0; ip < P.npp; ip += ipStep) {
    const PrimPairDev& A = pp[P.pp_off + ip];
    double ea, eb;
    pair_exps(SA, SB, prim, A, ea, eb);
    for (int x = 0; x < 3; x++)
      hermite_E_rt<double, LM + 1>(la + rb, lb + rb, A.o2p, A.PA[x], A.PB[x], Ea[x]);
    for (int h = 0; h < nherm(Lb); h++) G[h] = 0.0;
    for (int iq = 0; iq < Q.npp; iq++) {
      const PrimPairDev& B = pp[Q.pp_off + iq];
      double ec, ed;
      pair_exps(SC, SD, prim, B, ec, ed);
      for (int x = 0; x < 3; x++)
        hermite_E_rt<double, LM + 1>(lc + rk, ld + rk, B.o2p, B.PA[x], B.PB[x], Ec[x]);
      const double X = A.P[0] - B.P[0], Y = A.P[1] - B.P[1], Z = A.P[2] - B.P[2];
      const double pq = A.p + B.p, alpha = A.p * B.p / pq;
      double pref = PI52X2 / sqrt(pq) * A.Kp * B.Kp;
      const double Targ = alpha * (X * X + Y * Y + Z * Z);
      boys_rt<double>(L, Targ, F, boys);
      if (opi >= 0) {
        r12_aux(L, Targ, F);
        pref /= 2.0 * alpha;
      }
      hermite_R_rt<double>(L, alpha, X, Y, Z, F, Rv);
      for (int x = 0; x < 3; x++) {
        const int ty = (dir[2] == x) | ((dir[3] == x) << 1);
        nf[x] = axis_factor(Ec[x], ld + rk, lc + ld + 2 * rk + 1, ci[x], di[x], ty, 2.0 * ec,
                            2.0 * ed, f[x]);
        for (int t = 1; t < nf[x]; t += 2) f[x][t] = -f[x][t];
      }
      ket_add(G, pref, f[0], nf[0], f[1], nf[1], f[2], nf[2], Lb, Rv, sh[0], sh[1], sh[2]);
    }
    for (int ai = 0; ai < na; ai++)
      for (int bi = 0; bi < nb; bi++) {
        const int ax[3] = {cart_lx(la, ai), cart_ly(la, ai), cart_lz(la, ai)};
        const int bx[3] = {cart_lx(lb, bi), cart_ly(lb, bi), cart_lz(lb, bi)};
        for (int x = 0; x < 3; x++) {
          const int ty = (dir[0] == x) | ((dir[1] == x) << 1);
          ng[x] = axis_factor(Ea[x], lb + rb, la + lb + 2 * rb + 1, ax[x], bx[x], ty, 2.0 * ea,
                              2.0 * eb, g[x]);
        }
        atomicAdd(out + (ai * nb + bi) * stride,
                  w * bra_dot(g[0], ng[0], g[1], ng[1], g[2], ng[2], G));
      }
  }
}

// one index of a 4-index block (row-major, index 3 fastest) from Cartesian
// to spherical: out[.. mu ..] = sum_c T[c][mu] in[.. c ..]; the gs threads
// of a group (g0 = this thread's index in it) share the work
__device__ void sph_index(const double* in, double* out, int* dims, int k, const double* T,
                          int nsk, int g0, int gs) {
  int od[4] = {dims[0], dims[1], dims[2], dims[3]};
  od[k] = nsk;
  const int tot = od[0] * od[1] * od[2] * od[3];
  for (int e = g0; e < tot; e += gs) {
    int i[4], r = e;
    for (int q = 3; q >= 0; q--) {
      i[q] = r % od[q];
      r /= od[q];
    }
    const int mu = i[k];
    double s = 0.0;
    for (int c = 0; c < dims[k]; c++) {
      const double t = T[c * nsk + mu];
      if (t == 0.0) continue;
      i[k] = c;
      s += t * in[((i[0] * dims[1] + i[1]) * dims[2] + i[2]) * dims[3] + i[3]];
    }
    out[e] = s;
  }
  dims[k] = nsk;
}

constexpr int SCH_THREADS = 128;

// One (pair, component) per group of gsize threads, SCH_THREADS / gsize
// groups per block, units enumerated pair-major over the components of a
// pair: the plain (ab|ab) block (when lowLL), the 81 blocks
// (dA_i dB_j ab | dA_k dB_l ab) (nSS = 81), the 18 Gaunt blocks
// (dA_i b | dA_k b), (a dB_i | a dB_k) (nG = 18) and the 108 gauge blocks
// (dA_j b | -r_i r_i' / r^3 | dA_l b) and the same on B (nB = 108; i <= i',
// the kernel -delta_ii' / r12 + d_i d_i' r12).  A group builds the
// Cartesian block in shared memory -- thread g0 takes ket column g0 % cpow
// (cpow: the column count rounded up to a power of two) and every
// (gsize / cpow)-th bra primitive pair from g0 / cpow -- transforms it to
// the spherical basis index by index, and folds its largest |element| into
// the pair's maximum (mx[6 pair + 0..5]: plain, SS, Gaunt on A, Gaunt on B,
// gauge on A, gauge on B) with an atomic max on the bit pattern
// (non-negative doubles order as integers).
constexpr int SCH_SLOTS = 6;
template <int LM>
__global__ void __launch_bounds__(SCH_THREADS)
    rel_schwarz_kernel(const PairDev* __restrict__ pairs, const PrimPairDev* __restrict__ pp,
                       const ShellDev* __restrict__ shells, const double* __restrict__ prim,
                       const double* __restrict__ boys, const double* __restrict__ sph,
                       const int* __restrict__ sphOff, int beg, int npair, int la, int lb,
                       int lowLL, int nSS, int nG, int nB, int gsize, int cpow,
                       unsigned long long* mx) {
  extern __shared__ double sm[];
  const int na = ncart(la), nb = ncart(lb);
  const int n4 = na * nb * na * nb;
  const int groups = SCH_THREADS / gsize;
  const int ncomp = lowLL + nSS + nG + nB;
  const int g = threadIdx.x / gsize, g0 = threadIdx.x % gsize;
  const long long unit = (long long)blockIdx.x * groups + g;
  const bool live = unit < (long long)npair * ncomp;
  const int ip = live ? (int)(unit / ncomp) : 0;
  const int comp = live ? (int)(unit % ncomp) : 0;
  const PairDev P = pairs[beg + ip];
  const ShellDev SA = shells[P.shA], SB = shells[P.shB];
  int dir[4] = {-1, -1, -1, -1};
  int slot = 0, opi = -1, opj = -1;
  if (comp >= lowLL + nSS + nG) {  // gauge: one derivative in each pair
    const int gc = comp - lowLL - nSS - nG;
    const int side = gc / 54, r = gc % 54;
    op_pair(r / 9, opi, opj);
    dir[side] = (r % 9) / 3;
    dir[2 + side] = r % 3;
    slot = 4 + side;
  } else if (comp >= lowLL + nSS) {  // Gaunt: one derivative in each pair
    const int gc = comp - lowLL - nSS;
    const int side = gc / 9;  // 0: on A, 1: on B
    dir[side] = (gc % 9) / 3;
    dir[2 + side] = gc % 3;
    slot = 2 + side;
  } else if (comp >= lowLL) {
    const int dc = comp - lowLL;  // derivative component 0..80
    dir[0] = dc / 27;
    dir[1] = (dc / 9) % 3;
    dir[2] = (dc / 3) % 3;
    dir[3] = dc % 3;
    slot = 1;
  }
  double* cur = sm + (size_t)g * 2 * n4;
  double* nxt = cur + n4;
  for (int e = g0; e < n4; e += gsize) cur[e] = 0.0;
  __syncthreads();
  const int col = g0 % cpow, slice = g0 / cpow, nslice = gsize / cpow;
  if (live && col < na * nb) {
    deriv_column<LM>(la, lb, la, lb, col / nb, col % nb, dir, P, P, pp, shells, prim, boys,
                     cur + col, na * nb, slice, nslice, opi, opj);
    if (opi >= 0 && opi == opj)  // the -delta_ii' / r12 part of the gauge kernel
      deriv_column<LM>(la, lb, la, lb, col / nb, col % nb, dir, P, P, pp, shells, prim, boys,
                       cur + col, na * nb, slice, nslice, -1, -1, -1.0);
  }
  __syncthreads();
  int dims[4] = {na, nb, na, nb};
  const ShellDev* S4[4] = {&SA, &SB, &SA, &SB};
  for (int k = 0; k < 4; k++) {  // every thread reaches each barrier
    const ShellDev& S = *S4[k];
    if (live && S.pure) {
      sph_index(cur, nxt, dims, k, sph + sphOff[S.l], nsph(S.l), g0, gsize);
      double* t = cur;
      cur = nxt;
      nxt = t;
    }
    __syncthreads();
  }
  if (!live) return;
  double m = 0.0;
  const int tot = dims[0] * dims[1] * dims[2] * dims[3];
  for (int e = g0; e < tot; e += gsize) m = fmax(m, fabs(cur[e]));
  if (m > 0.0)
    atomicMax(mx + SCH_SLOTS * (size_t)ip + slot, (unsigned long long)__double_as_longlong(m));
}

// Q^LL = sqrt(max), Q^SS = C2 sqrt(max) of each pair of a class into both
// triangles of the nshell x nshell tables (direct4C_libcint.hpp:388-394,
// :464-470); Q^G(d, o) = C1 sqrt(max) with the derivative on shell d
// (SchwarzGaunt, :2910-2955, C1 = 1 / 2c), not symmetric; the same for the
// gauge kernel, Q^B(d, o) (SchwarzGauge, :3960-4005, which maxes over
// libcint's 16 spin components of the operator where this maxes over its
// 81 spatial components).
__global__ void rel_schwarz_finish_kernel(const PairDev* __restrict__ pairs, int beg, int npair,
                                          const unsigned long long* __restrict__ mx,
                                          int needLL, int needSS, int needG, int needB,
                                          int nshell, double* qLL, double* qSS, double* qG,
                                          double* qB) {
  const int ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= npair) return;
  const PairDev P = pairs[beg + ip];
  const size_t e1 = P.s1 + (size_t)P.s2 * nshell, e2 = P.s2 + (size_t)P.s1 * nshell;
  auto v = [&](int k) {
    return sqrt(__longlong_as_double((long long)mx[SCH_SLOTS * ip + k]));
  };
  if (needLL) qLL[e1] = qLL[e2] = v(0);
  if (needSS) {
    const double C2 = 1.0 / (4.0 * SPEED_OF_LIGHT * SPEED_OF_LIGHT);
    qSS[e1] = qSS[e2] = C2 * v(1);
  }
  if (needG) {
    const double C1 = 1.0 / (2.0 * SPEED_OF_LIGHT);
    qG[P.shA + (size_t)P.shB * nshell] = C1 * v(2);
    qG[P.shB + (size_t)P.shA * nshell] = C1 * v(3);
  }
  if (needB) {
    const double C1 = 1.0 / (2.0 * SPEED_OF_LIGHT);
    qB[P.shA + (size_t)P.shB * nshell] = C1 * v(4);
    qB[P.shB + (size_t)P.shA * nshell] = C1 * v(5);
  }
}

cqf_status ensure_rel_schwarz(cqf_basis* B, bool needLL, bool needSS, bool needG,
                              bool needB, cudaStream_t st) {
  needLL = needLL && !B->rel_qLL;
  needSS = needSS && !B->rel_qSS;
  needG = needG && !B->rel_qG;
  needB = needB && !B->rel_qB;
  if (!needLL && !needSS && !needG && !needB) return CQF_OK;
  const size_t ns2 = (size_t)B->nshell * B->nshell;
  // basis-owned, stream-ordered on the basis' stream (freed by free_basis)
  for (double** q : {&B->d_qLL, &B->d_qSS, &B->d_qG, &B->d_qB})
    if (!*q) {
      CQF_RCUDA(cudaMallocAsync(q, ns2 * sizeof(double), B->stream));
      CQF_RCUDA(cudaMemsetAsync(*q, 0, ns2 * sizeof(double), B->stream));
    }
  CQF_RCUDA(cudaStreamSynchronize(B->stream));
  unsigned long long* mx = nullptr;
  const size_t mxn = SCH_SLOTS * (size_t)std::max(1, B->npair);
  CQF_RCUDA(cudaMallocAsync(&mx, mxn * sizeof(unsigned long long), st));
  CQF_RCUDA(cudaMemsetAsync(mx, 0, mxn * sizeof(unsigned long long), st));
  const int nSS = needSS ? 81 : 0, nG = needG ? 18 : 0, nB = needB ? 108 : 0;
  const int ncomp = (needLL ? 1 : 0) + nSS + nG + nB;
  for (int c = 0; c < NCLS; c++) {
    if (B->cls_cnt[c] <= 0) continue;
    int la, lb;
    class_ls(c, la, lb);
    const int n4 = ncart(la) * ncart(lb) * ncart(la) * ncart(lb);
    // threads per (pair, component): at least a warp, and the Cartesian
    // column count rounded up to a power of two (the spare threads split the
    // bra primitive pairs)
    int cpow = 1;
    while (cpow < ncart(la) * ncart(lb)) cpow *= 2;
    const int gsize = std::min(SCH_THREADS, std::max(32, cpow));
    const int groups = SCH_THREADS / gsize;
    const size_t smem = (size_t)groups * 2 * n4 * sizeof(double);
    const long long units = (long long)B->cls_cnt[c] * ncomp;
    const unsigned nblk = (unsigned)((units + groups - 1) / groups);
    unsigned long long* mxc = mx + SCH_SLOTS * (size_t)B->cls_beg[c];
    const int lm = std::max(la, 1);
#define CQF_SCH(LMV)                                                                          \
  if (lm == LMV) {                                                                            \
    CQF_RCUDA(cudaFuncSetAttribute(rel_schwarz_kernel<LMV>,                                   \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));  \
    rel_schwarz_kernel<LMV><<<nblk, SCH_THREADS, smem, st>>>(                                 \
        B->d_pairs, B->d_pp, B->d_shells, B->d_prim, B->d_boys64, B->d_sph, B->d_sphOff,      \
        B->cls_beg[c], B->cls_cnt[c], la, lb, needLL ? 1 : 0, nSS, nG, nB, gsize, cpow, mxc); \
  }
    CQF_SCH(1)
    CQF_SCH(2)
    CQF_SCH(3)
#undef CQF_SCH
    rel_schwarz_finish_kernel<<<(B->cls_cnt[c] + 127) / 128, 128, 0, st>>>(
        B->d_pairs, B->cls_beg[c], B->cls_cnt[c], mxc, needLL, needSS, needG, needB,
        B->nshell, B->d_qLL, B->d_qSS, B->d_qG, B->d_qB);
    CQF_RCUDA(cudaGetLastError());
  }
  cudaFreeAsync(mx, st);
  CQF_RCUDA(cudaStreamSynchronize(st));
  B->rel_qLL = B->rel_qLL || needLL;
  B->rel_qSS = B->rel_qSS || needSS;
  B->rel_qG = B->rel_qG || needG;
  B->rel_qB = B->rel_qB || needB;
  return CQF_OK;
}

// ---------------------------------------------------------- back transform
// AX (complex N x N, assigned) from a Cartesian accumulator, B = T^T Ac T:
//   mode 0: B (complex)             mode 1: B + B^T (real Ac)
//   mode 2: i (B - B^T) (real Ac)   mode 3: B + B^H (complex)
__global__ void rel_from_cart_kernel(const MatList l, int N, int nc,
                                     const ShellDev* __restrict__ sh,
                                     const int* __restrict__ ao2s,
                                     const double* __restrict__ sph,
                                     const int* __restrict__ sphOff) {
  const double* __restrict__ Ac = l.src[blockIdx.y];
  double* AX = l.dst[blockIdx.y];
  const int mode = l.mode[blockIdx.y];
  size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)N * N) return;
  const int i = (int)(k % N), j = (int)(k / N);
  const bool cplx = (mode == 0 || mode == 3);
  auto bval = [&](int r, int c, double& bre, double& bim) {
    const ShellDev A = sh[ao2s[r]], B = sh[ao2s[c]];
    const int mu = r - A.sph_off, nu = c - B.sph_off;
    const double* TA = sph + sphOff[A.l];
    const double* TB = sph + sphOff[B.l];
    bre = 0.0;
    bim = 0.0;
    for (int a = 0; a < ncart(A.l); a++) {
      const double ta = A.pure ? TA[a * nsph(A.l) + mu] : (a == mu);
      if (ta == 0.0) continue;
      for (int b = 0; b < ncart(B.l); b++) {
        const double tb = B.pure ? TB[b * nsph(B.l) + nu] : (b == nu);
        if (tb == 0.0) continue;
        const size_t e = (size_t)(A.cart_off + a) + (size_t)(B.cart_off + b) * nc;
        if (cplx) {
          bre += ta * tb * Ac[2 * e];
          bim += ta * tb * Ac[2 * e + 1];
        } else {
          bre += ta * tb * Ac[e];
        }
      }
    }
  };
  double r1, i1, r2 = 0.0, i2 = 0.0;
  bval(i, j, r1, i1);
  if (mode != 0) bval(j, i, r2, i2);
  double outr, outi;
  if (mode == 0) { outr = r1; outi = i1; }
  else if (mode == 1) { outr = r1 + r2; outi = 0.0; }
  else if (mode == 2) { outr = 0.0; outi = r1 - r2; }
  else { outr = r1 + r2; outi = i1 - i2; }
  AX[2 * k] = outr;
  AX[2 * k + 1] = outi;
}

// imaginary part set to zero (the Coulomb density of the bare term)
__global__ void real_part_kernel(const double* __restrict__ X, size_t n, double* Y) {
  size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  Y[2 * k] = X[2 * k];
  Y[2 * k + 1] = 0.0;
}

// ------------------------------------------------------ 4C assembly kernels
// blk(i, j) = D(ro + i, co + j), N x N out of 2N x 2N
__global__ void get_block_kernel(const double* __restrict__ D, int N, int ro, int co,
                                 double* blk) {
  size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)N * N) return;
  const int i = (int)(k % N), j = (int)(k / N);
  const size_t e = (size_t)(ro + i) + (size_t)(co + j) * 2 * N;
  blk[2 * k] = D[2 * e];
  blk[2 * k + 1] = D[2 * e + 1];
}

// M(ro + i, co + j) += f * src(i, j)
__global__ void add_block_kernel(double* M, int N, int ro, int co, const double* __restrict__ src,
                                 double f) {
  size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)N * N) return;
  const int i = (int)(k % N), j = (int)(k / N);
  const size_t e = (size_t)(ro + i) + (size_t)(co + j) * 2 * N;
  M[2 * e] += f * src[2 * k];
  M[2 * e + 1] += f * src[2 * k + 1];
}

// SL = LS^H (impl.hpp:4560-4575), then G = twoeH - xHFX K
__global__ void finish_gd_kernel(double* twoeH, double* K, int N, double xHFX, int exch,
                                 double* G) {
  const int N2 = 2 * N;
  size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (k >= (size_t)N2 * N2) return;
  const int r = (int)(k % N2), c = (int)(k / N2);
  size_t src = k;
  bool conj = false;
  if (r >= N && c < N) {  // SL block element (N + j, i) = conj(LS(i, N + j))
    src = (size_t)c + (size_t)r * N2;
    conj = true;
  }
  double hr = twoeH[2 * src], hi = twoeH[2 * src + 1];
  double kr = K[2 * src], ki = K[2 * src + 1];
  if (conj) {
    hi = -hi;
    ki = -ki;
  }
  G[2 * k] = hr - (exch ? xHFX * kr : 0.0);
  G[2 * k + 1] = hi - (exch ? xHFX * ki : 0.0);
}

// ------------------------------------------------------------ host driver
cqf_status ensure_relws(cqf_basis* B, size_t bytes) {
  if (bytes <= B->relws_bytes) return CQF_OK;
  if (B->d_relws) CQF_RCUDA(cudaFreeAsync(B->d_relws, B->stream));
  B->d_relws = nullptr;
  B->relws_bytes = 0;
  CQF_RCUDA(cudaMallocAsync(&B->d_relws, bytes, B->stream));
  CQF_RCUDA(cudaStreamSynchronize(B->stream));
  B->relws_bytes = bytes;
  return CQF_OK;
}

size_t align32(size_t n) { return (n + 31) / 32 * 32; }

// One contraction type on device pointers (X, AX: 17 entries, N x N complex).
// ws: device scratch of rel_ws_doubles() doubles.  From opts: screen, and
// precision / fp32_cutoff (CQF_MIXED: quartets whose screening bound is below
// the cutoff run in FP32 arithmetic, the rest in FP64).  cnt: total,
// screened, FP32, FP64 quartet counts, added to.
size_t rel_core_doubles(const cqf_basis* B) {
  const size_t nc2 = (size_t)B->ncart * B->ncart, ns2 = (size_t)B->nshell * B->nshell;
  const size_t dc = align32(9 * 2 * nc2) + align32(13 * nc2) + align32(10 * ns2);
  // Gaunt: 20 Cartesian complex densities | 16 complex accumulators | norms
  const size_t ga = align32(20 * 2 * nc2) + align32(16 * 2 * nc2) + align32(18 * ns2);
  return std::max(dc, ga) + 64;
}
// Mask words of one launch stream's region: the cap, and at least one bra row
// of the widest class.
long long rel_mask_words(const cqf_basis* B) {
  size_t row = 1;
  for (int c = 0; c < NCLS; c++)
    row = std::max(row, ((size_t)B->cls_cnt[c] + WTILE - 1) / WTILE);
  return (long long)std::max(row, MASK_CAP_WORDS);
}
// Table windows of one launch stream (of the kinds that are known not to be
// held: rel_tables first).
size_t rel_window(const cqf_basis* B) {
  return (std::max({hg_windows<RelDig<1>>(B), hg_windows<RelDig<2>>(B),
                    hg_windows<GauntDig>(B)}) + 31) / 32 * 32;
}
// The contraction's arrays, then per launch stream the masks and word lists
// (16 B a word), four counters each, and the table windows.
size_t rel_ws_doubles(const cqf_basis* B) {
  return rel_core_doubles(B) +
         (size_t)(2 * rel_mask_words(B) + 2 + rel_window(B)) * (NAUX + 1);
}
// The engine's tables that a contraction type reads.
cqf_status rel_tables(cqf_basis* B, int type) {
  if (type == CQF_REL_LLSS || type == CQF_REL_SSSS) CQF_RTRY(hg_ensure(B, HG_SPIN));
  if (type == CQF_REL_LLSS) CQF_RTRY(hg_ensure(B, HG_PLAIN));
  if (type == CQF_REL_GAUNT) CQF_RTRY(hg_ensure(B, HG_D6));
  return CQF_OK;
}

// The entries a contraction type writes (the others are neither zeroed nor
// written: the reference's GAUNT list points its CSLM* / XSLM* entries at
// the CLSM* / XLSM* outputs).
std::vector<int> rel_outputs(int type, bool exch) {
  std::vector<int> o;
  auto four = [&](int base) {
    for (int c = 0; c < 4; c++) o.push_back(base + c);
  };
  if (type == CQF_REL_BARE_COULOMB) {
    o.push_back(CQF_CLLMS);
    if (exch) four(CQF_XLLMS);
  } else if (type == CQF_REL_LLSS) {
    o.push_back(CQF_CLLMS);
    four(CQF_CSSMS);
    if (exch) four(CQF_XLSMS);
  } else if (type == CQF_REL_SSSS) {
    four(CQF_CSSMS);
    if (exch) four(CQF_XSSMS);
  } else {
    four(CQF_CLSMS);
    if (exch) {
      four(CQF_XLLMS);
      four(CQF_XSSMS);
      four(CQF_XLSMS);
    }
  }
  return o;
}

cqf_status gaunt_contract_dev(cqf_basis* B, const double* const* X, double* const* AX, int exch,
                              bool gauge, const cqf_opts& opts, cudaStream_t st, double* ws,
                              unsigned long long* cnt);

// A list of (source, destination, mode) collected for one launch of a
// per-matrix kernel.
struct MatJobs {
  std::vector<const double*> src;
  std::vector<double*> dst;
  std::vector<int> mode;
  void add(const double* s, double* d, int m = 0) {
    src.push_back(s);
    dst.push_back(d);
    mode.push_back(m);
  }
  template <class F>
  void run(size_t span, F f) const {
    mat_batches(
        (int)src.size(), span, [&](int m) { return src[m]; }, [&](int m) { return dst[m]; },
        [&](int m) { return mode[m]; }, f);
  }
};
void run_back(const cqf_basis* B, const MatJobs& jobs, cudaStream_t st) {
  const size_t NN = (size_t)B->nbasis * B->nbasis;
  jobs.run(2 * NN, [&](const MatList& l, int n) {
    rel_from_cart_kernel<<<dim3(rgrid(NN, 256), n), 256, 0, st>>>(
        l, B->nbasis, B->ncart, B->d_shells, B->d_ao2shell, B->d_sph, B->d_sphOff);
  });
}

// go(cb, ck, region, stream) for every class pair with quartets (every
// ordered one, or ck <= cb), round-robin over the call's stream and the
// auxiliary ones with a mask region each: the launches only add into the
// accumulators, so one's tail overlaps the next one's start; the largest
// angular momenta first.
template <class Go>
cqf_status for_class_pairs(cqf_basis* B, bool ordered, double* ws, cudaStream_t st, Go go) {
  const long long maskWords = rel_mask_words(B);
  uint2* masks = reinterpret_cast<uint2*>(ws + rel_core_doubles(B));
  unsigned* work = reinterpret_cast<unsigned*>(masks + 2 * maskWords * (NAUX + 1));
  double* win = reinterpret_cast<double*>(work + 4 * (NAUX + 1));
  const size_t winDoubles = rel_window(B);
  CQF_RCUDA(cudaEventRecord(B->evFork, st));
  cudaStream_t lanes[NAUX + 1] = {st};
  for (int i = 0; i < NAUX; i++) {
    lanes[1 + i] = B->aux[i];
    CQF_RCUDA(cudaStreamWaitEvent(B->aux[i], B->evFork, 0));
  }
  int nlaunch = 0;
  cqf_status rc = CQF_OK;
  for (int cb = NCLS - 1; cb >= 0 && rc == CQF_OK; cb--)
    for (int ck = ordered ? NCLS - 1 : cb; ck >= 0 && rc == CQF_OK; ck--) {
      if (!B->cls_cnt[cb] || !B->cls_cnt[ck]) continue;
      const int li = nlaunch++ % (NAUX + 1);
      rc = go(cb, ck,
              HgRegion{masks + 2 * maskWords * li, maskWords, work + 4 * li,
                       win + winDoubles * li},
              lanes[li]);
    }
  for (int i = 0; i < NAUX; i++) {
    CQF_RCUDA(cudaEventRecord(B->evJoin[i], B->aux[i]));
    CQF_RCUDA(cudaStreamWaitEvent(st, B->evJoin[i], 0));
  }
  return rc;
}

cqf_status rel_contract_dev(cqf_basis* B, const double* const* X, double* const* AX, int type,
                            int exch, const cqf_opts& opts, cudaStream_t st, double* ws,
                            unsigned long long* cnt) {
  if (opts.shard_count < 1 || opts.shard_index < 0 || opts.shard_index >= opts.shard_count)
    return fail(CQF_EINVAL, "shard_index must lie in [0, shard_count)");
  const int screen = opts.screen;
  const bool mixed = opts.precision == CQF_MIXED && opts.fp32_cutoff > 0.0;
  const int N = B->nbasis, nc = B->ncart, ns = B->nshell;
  const size_t NN = (size_t)N * N, nc2 = (size_t)nc * nc, ns2 = (size_t)ns * ns;
  for (int m : rel_outputs(type, exch))
    if (AX[m]) CQF_RCUDA(cudaMemsetAsync(AX[m], 0, 2 * NN * sizeof(double), st));
  if (type == CQF_REL_GAUNT || type == CQF_REL_GAUGE)
    return gaunt_contract_dev(B, X, AX, exch, type == CQF_REL_GAUGE, opts, st, ws, cnt);

  if (type == CQF_REL_BARE_COULOMB) {
    // (LL|LL): the 1C engine on J[Re X] and K[X] (the same quartets, screen
    // and digestion as the reference's BARE_COULOMB branch, :514-790)
    if (!X[CQF_CLLMS] || !AX[CQF_CLLMS]) return fail(CQF_EINVAL, "BARE_COULOMB needs CLLMS");
    double* reX = ws;  // N x N complex
    real_part_kernel<<<rgrid(NN, 256), 256, 0, st>>>(X[CQF_CLLMS], NN, reX);
    CQF_RCUDA(cudaGetLastError());
    std::vector<cqf_contraction> list;
    list.push_back({reX, AX[CQF_CLLMS], 1, CQF_COULOMB});
    if (exch)
      for (int c = 0; c < 4; c++) {
        if (!X[CQF_XLLMS + c] || !AX[CQF_XLLMS + c])
          return fail(CQF_EINVAL, "BARE_COULOMB exchange needs XLLM*");
        list.push_back({X[CQF_XLLMS + c], AX[CQF_XLLMS + c], 1, CQF_EXCHANGE});
      }
    cqf_opts o;
    cqf_opts_default(&o);
    o.is_complex = 1;
    o.device_pointers = 1;
    o.screen = screen;
    o.precision = opts.precision;
    o.fp32_cutoff = opts.fp32_cutoff;
    o.stream = st;
    o.shard_index = opts.shard_index;
    o.shard_count = opts.shard_count;
    cqf_stats s1{};
    const int n = (int)list.size();
    if (split_eligible(B, list.data(), n, o)) {
      // Hermitian entries: real and imaginary parts on the real kernels
      CQF_RTRY(basis_workspace(
          B, split_ws_doubles(B, split_real_count(list.data(), n), o) * sizeof(double)));
      CQF_RTRY(split_core(B, list.data(), n, o, &s1, static_cast<double*>(B->d_ws), false,
                          nullptr));
    } else {
      CQF_RTRY(basis_workspace(B, ws_layout(B, n, o).total * sizeof(double)));
      CQF_RTRY(contract_core(B, list.data(), n, o, &s1, static_cast<double*>(B->d_ws), false,
                             nullptr));
    }
    cnt[0] += s1.quartets_total;
    cnt[1] += s1.quartets_screened;
    cnt[2] += s1.quartets_fp32;
    cnt[3] += s1.quartets_fp64;
    return CQF_OK;
  }

  const bool llss = (type == CQF_REL_LLSS);
  CQF_RTRY(ensure_rel_schwarz(B, llss, true, false, false, st));
  // required entries
  std::vector<int> need = {CQF_CSSMS, CQF_CSSMX, CQF_CSSMY, CQF_CSSMZ};
  if (llss) need.push_back(CQF_CLLMS);
  if (exch)
    for (int c = 0; c < 4; c++) need.push_back((llss ? CQF_XLSMS : CQF_XSSMS) + c);
  for (int m : need)
    if (!X[m]) return fail(CQF_EINVAL, "missing X entry for this contraction type");
  std::vector<int> outs = {CQF_CSSMS, CQF_CSSMX, CQF_CSSMY, CQF_CSSMZ};
  if (llss) outs.push_back(CQF_CLLMS);
  if (exch)
    for (int c = 0; c < 4; c++) outs.push_back((llss ? CQF_XLSMS : CQF_XSSMS) + c);
  for (int m : outs)
    if (!AX[m]) return fail(CQF_EINVAL, "missing AX entry for this contraction type");

  // workspace: 9 Cartesian complex densities | 13 real accumulators (Jll,
  // Jss x4, K x4 complex) | norms
  double* xc = ws;
  double* accb = ws + align32(9 * 2 * nc2);
  double* nrm = accb + align32(13 * nc2);
  double* Jll = accb;
  double* Jss[4] = {accb + nc2, accb + 2 * nc2, accb + 3 * nc2, accb + 4 * nc2};
  double* Kc[4] = {accb + 5 * nc2, accb + 7 * nc2, accb + 9 * nc2, accb + 11 * nc2};
  auto XC = [&](int slot) { return xc + (size_t)slot * 2 * nc2; };
  // slots: 0 CLLMS, 1..4 CSSM*, 5..8 exchange densities
  MatJobs cart, norms, backs;
  if (llss) cart.add(X[CQF_CLLMS], XC(0));
  for (int c = 0; c < 4; c++) cart.add(X[CQF_CSSMS + c], XC(1 + c));
  if (exch)
    for (int c = 0; c < 4; c++) cart.add(X[(llss ? CQF_XLSMS : CQF_XSSMS) + c], XC(5 + c));
  cart.run(2 * nc2, [&](const MatList& l, int n) { launch_to_cart(B, l, n, 1, st); });
  // screening norms: max over CLLMS, CSSM*, XLSM* (LLSS) or CSSM* (SSSS)
  std::vector<int> smats = {CQF_CSSMS, CQF_CSSMX, CQF_CSSMY, CQF_CSSMZ};
  if (llss) {
    smats.insert(smats.begin(), CQF_CLLMS);
    for (int c = 0; c < 4; c++)
      if (X[CQF_XLSMS + c]) smats.push_back(CQF_XLSMS + c);
  }
  double* nmAll = nrm + ns2;
  for (size_t i = 0; i < smats.size(); i++) norms.add(X[smats[i]], nmAll + i * ns2);
  norms.run(ns2, [&](const MatList& l, int n) { launch_block_norms(B, l, n, 1, st); });
  launch_max_norms(nmAll, (int)smats.size(), ns2, nrm,
                   reinterpret_cast<unsigned long long*>(nmAll + 9 * ns2), st);
  CQF_RCUDA(cudaMemsetAsync(accb, 0, 13 * nc2 * sizeof(double), st));
  unsigned long long* dcnt = B->d_counters;
  CQF_RCUDA(cudaMemsetAsync(dcnt, 0, 4 * sizeof(unsigned long long), st));
  CQF_RCUDA(cudaGetLastError());

  RelLaunch a{};
  a.pairs = B->d_pairs;
  a.pairRange = B->d_pairRange;
  a.mixed = mixed ? 1 : 0;
  a.cut = opts.fp32_cutoff;
  a.screen = screen;
  a.thresh = B->thresh;
  a.norms = nrm;
  a.qLL = B->d_qLL;
  a.qSS = B->d_qSS;
  a.nShell = ns;
  a.ncart = nc;
  a.exchange = exch;
  a.Xll = XC(0);
  for (int c = 0; c < 4; c++) {
    a.Xss[c] = XC(1 + c);
    a.Xk[c] = XC(5 + c);
    a.Jss[c] = Jss[c];
    a.K[c] = Kc[c];
  }
  a.Jll = Jll;
  a.shardIdx = opts.shard_index;
  a.shardCnt = std::max(1, opts.shard_count);
  a.counters = dcnt;
  CQF_RTRY(for_class_pairs(
      B, llss, ws, st, [&](int cb, int ck, const HgRegion& r, cudaStream_t ls) {
        int la, lb, lc, ld;
        class_ls(cb, la, lb);
        class_ls(ck, lc, ld);
        a.braBeg = B->cls_beg[cb];
        a.nBra = B->cls_cnt[cb];
        a.ketBeg = B->cls_beg[ck];
        a.nKet = B->cls_cnt[ck];
        a.same = (cb == ck);
        a.lsum = la + lb + lc + ld;
        return llss ? launch_rel<1>(B, a, cb, ck, r, ls) : launch_rel<2>(B, a, cb, ck, r, ls);
      }));
  CQF_RCUDA(cudaGetLastError());
  auto back = [&](const double* src, int mode, double* dst) { backs.add(src, dst, mode); };
  if (llss) back(Jll, 1, AX[CQF_CLLMS]);
  back(Jss[0], 1, AX[CQF_CSSMS]);
  for (int c = 1; c < 4; c++) back(Jss[c], 2, AX[CQF_CSSMS + c]);
  if (exch)
    for (int c = 0; c < 4; c++)
      back(Kc[c], llss ? 0 : 3, AX[(llss ? CQF_XLSMS : CQF_XSSMS) + c]);
  run_back(B, backs, st);
  CQF_RCUDA(cudaGetLastError());
  unsigned long long h[4];
  CQF_RCUDA(cudaMemcpyAsync(h, dcnt, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  CQF_RCUDA(cudaStreamSynchronize(st));
  cnt[0] += h[0];
  cnt[1] += h[1];
  cnt[2] += h[2];
  cnt[3] += h[3];
  return CQF_OK;
}


// The GAUNT (or GAUGE) contraction on device pointers (X, AX: 29
// entries).  Needs X[CLSM*], X[CSLM*] and, with exchange, X[XLLM*],
// X[XSSM*], X[XSLM*]; writes AX[CLSM*] and, with exchange, AX[XLLM*],
// AX[XSSM*], AX[XLSM*].  The screening norms are the max over the 16
// exchange densities the reference uses (:2957-3020, :4060-4130), of those
// given.  FP64 (opts.precision is not applied to these terms).
cqf_status gaunt_contract_dev(cqf_basis* B, const double* const* X, double* const* AX, int exch,
                              bool gauge, const cqf_opts& opts, cudaStream_t st, double* ws,
                              unsigned long long* cnt) {
  const int N = B->nbasis, nc = B->ncart, ns = B->nshell;
  const size_t NN = (size_t)N * N, nc2 = (size_t)nc * nc, ns2 = (size_t)ns * ns;
  (void)NN;
  std::vector<int> need;
  for (int c = 0; c < 4; c++) {
    need.push_back(CQF_CLSMS + c);
    need.push_back(CQF_CSLMS + c);
    if (exch) {
      need.push_back(CQF_XLLMS + c);
      need.push_back(CQF_XSSMS + c);
      need.push_back(CQF_XSLMS + c);
    }
  }
  for (int m : need)
    if (!X[m]) return fail(CQF_EINVAL, "missing X entry for the GAUNT / GAUGE contraction");
  for (int m : rel_outputs(CQF_REL_GAUNT, exch))
    if (!AX[m]) return fail(CQF_EINVAL, "missing AX entry for the GAUNT / GAUGE contraction");
  CQF_RTRY(ensure_rel_schwarz(B, false, false, !gauge, gauge, st));

  double* xc = ws;
  double* accb = ws + align32(20 * 2 * nc2);
  double* nrm = accb + align32(16 * 2 * nc2);
  auto XC = [&](int slot) { return xc + (size_t)slot * 2 * nc2; };
  auto AC = [&](int slot) { return accb + (size_t)slot * 2 * nc2; };
  // density slots: 0 XLLM*, 4 XSSM*, 8 CLSM*, 12 CSLM*, 16 XSLM*
  const int src[5] = {CQF_XLLMS, CQF_XSSMS, CQF_CLSMS, CQF_CSLMS, CQF_XSLMS};
  MatJobs cart, norms, backs;
  for (int k = 0; k < 5; k++)
    for (int c = 0; c < 4; c++)
      if (X[src[k] + c]) cart.add(X[src[k] + c], XC(4 * k + c));
  cart.run(2 * nc2, [&](const MatList& l, int n) { launch_to_cart(B, l, n, 1, st); });
  // screening norms: max over XLSM*, XSLM*, XLLM*, XSSM*
  // (without exchange, the LS / SL Coulomb entries stand for the same
  // LS / SL blocks)
  std::vector<int> smats;
  for (int base : {(int)CQF_XLSMS, (int)CQF_XSLMS, (int)CQF_XLLMS, (int)CQF_XSSMS})
    for (int c = 0; c < 4; c++) {
      int m = base + c;
      if (!X[m] && base == CQF_XLSMS) m = CQF_CLSMS + c;
      if (!X[m] && base == CQF_XSLMS) m = CQF_CSLMS + c;
      if (X[m]) smats.push_back(m);
    }
  double* nmAll = nrm + ns2;
  for (size_t i = 0; i < smats.size(); i++) norms.add(X[smats[i]], nmAll + i * ns2);
  norms.run(ns2, [&](const MatList& l, int n) { launch_block_norms(B, l, n, 1, st); });
  launch_max_norms(nmAll, (int)smats.size(), ns2, nrm,
                   reinterpret_cast<unsigned long long*>(nmAll + 16 * ns2), st);
  CQF_RCUDA(cudaMemsetAsync(accb, 0, 16 * 2 * nc2 * sizeof(double), st));
  unsigned long long* dcnt = B->d_counters;
  CQF_RCUDA(cudaMemsetAsync(dcnt, 0, 4 * sizeof(unsigned long long), st));
  CQF_RCUDA(cudaGetLastError());

  GauntLaunch a{};
  a.pairs = B->d_pairs;
  a.pp = B->d_pp;
  a.shells = B->d_shells;
  a.prim = B->d_prim;
  a.boys = B->d_boys64;
  a.screen = opts.screen;
  a.thresh = B->thresh;
  a.norms = nrm;
  a.qG = gauge ? B->d_qB : B->d_qG;
  a.nShell = ns;
  a.ncart = nc;
  a.exchange = exch;
  for (int c = 0; c < 4; c++) {
    a.Xll[c] = XC(0 + c);
    a.Xss[c] = XC(4 + c);
    a.Cls[c] = XC(8 + c);
    a.Csl[c] = XC(12 + c);
    a.Xsl[c] = XC(16 + c);
    a.Kll[c] = AC(0 + c);
    a.Kss[c] = AC(4 + c);
    a.Jls[c] = AC(8 + c);
    a.Kls[c] = AC(12 + c);
  }
  a.shardIdx = opts.shard_index;
  a.shardCnt = std::max(1, opts.shard_count);
  a.counters = dcnt;
  CQF_RTRY(for_class_pairs(
      B, false, ws, st, [&](int cb, int ck, const HgRegion& r, cudaStream_t ls) {
        int la, lb, lc, ld;
        class_ls(cb, la, lb);
        class_ls(ck, lc, ld);
        a.braBeg = B->cls_beg[cb];
        a.nBra = B->cls_cnt[cb];
        a.ketBeg = B->cls_beg[ck];
        a.nKet = B->cls_cnt[ck];
        a.same = (cb == ck);
        if (gauge) {
          launch_gauge(a, la, lb, lc, ld, ls);
          return CQF_OK;
        }
        return hg_contract<GauntDig>(
            B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a, ls,
            [&](const HgPart& p, uint2* masks, int* list64, int* list32, unsigned* lcount,
                unsigned gp) {
              gaunt_plan_kernel<<<gp, 256, 0, ls>>>(p.of(a), masks, list64, list32, lcount);
            });
      }));
  CQF_RCUDA(cudaGetLastError());
  auto back = [&](const double* srcAcc, int mode, double* dst) { backs.add(srcAcc, dst, mode); };
  for (int c = 0; c < 4; c++) {
    back(AC(8 + c), 0, AX[CQF_CLSMS + c]);
    if (exch) {
      back(AC(0 + c), 3, AX[CQF_XLLMS + c]);
      back(AC(4 + c), 3, AX[CQF_XSSMS + c]);
      back(AC(12 + c), 0, AX[CQF_XLSMS + c]);
    }
  }
  run_back(B, backs, st);
  CQF_RCUDA(cudaGetLastError());
  unsigned long long h[4];
  CQF_RCUDA(cudaMemcpyAsync(h, dcnt, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
  CQF_RCUDA(cudaStreamSynchronize(st));
  for (int k = 0; k < 4; k++) cnt[k] += h[k];
  return CQF_OK;
}

}  // namespace
}  // namespace cqf

using namespace cqf;

extern "C" {

cqf_status cqf_rel_two_body_contract(cqf_basis* B, const void* const* X, void* const* AX,
                                     int type, int compute_exchange, const cqf_opts* optsIn,
                                     cqf_stats* stats) {
  if (!B || !X || !AX) return fail(CQF_EINVAL, "cqf_rel_two_body_contract: null argument");
  if (type < CQF_REL_BARE_COULOMB || type > CQF_REL_GAUGE)
    return fail(CQF_EINVAL, "cqf_rel_two_body_contract: unknown contraction type");
  cqf_opts o;
  cqf_opts_default(&o);
  if (optsIn) o = *optsIn;
  std::lock_guard<std::mutex> lk(B->mu);
  CQF_RCUDA(cudaSetDevice(B->device));
  cudaStream_t st = o.stream ? (cudaStream_t)o.stream : B->stream;
  const int nmat = (type >= CQF_REL_GAUNT) ? CQF_REL_NMAT_GAUNT : CQF_REL_NMAT;
  const std::vector<int> outs = rel_outputs(type, compute_exchange != 0);
  const size_t NN = (size_t)B->nbasis * B->nbasis;
  CQF_RTRY(rel_tables(B, type));
  const size_t wsd = rel_ws_doubles(B);
  const size_t hostd = o.device_pointers ? 0 : align32(2 * NN) * 2 * nmat;
  CQF_RTRY(ensure_relws(B, (wsd + hostd) * sizeof(double)));
  double* ws = static_cast<double*>(B->d_relws);
  double* hbuf = ws + wsd;
  const double* Xd[CQF_REL_NMAT_GAUNT] = {};
  double* AXd[CQF_REL_NMAT_GAUNT] = {};
  for (int m = 0; m < nmat; m++) {
    if (o.device_pointers) {
      Xd[m] = static_cast<const double*>(X[m]);
      AXd[m] = static_cast<double*>(AX[m]);
    } else {
      double* xd = hbuf + (size_t)m * align32(2 * NN);
      double* ad = hbuf + (size_t)(nmat + m) * align32(2 * NN);
      Xd[m] = X[m] ? xd : nullptr;
      AXd[m] = AX[m] ? ad : nullptr;
      if (X[m])
        CQF_RCUDA(cudaMemcpyAsync(xd, X[m], 2 * NN * sizeof(double), cudaMemcpyHostToDevice, st));
    }
  }
  CQF_RCUDA(cudaEventRecord(B->ev0, st));
  unsigned long long cnt[4] = {0, 0, 0, 0};
  CQF_RTRY(rel_contract_dev(B, Xd, AXd, type, compute_exchange, o, st, ws, cnt));
  CQF_RCUDA(cudaEventRecord(B->ev1, st));
  // only the entries the type writes come back (a list may alias the others)
  if (!o.device_pointers)
    for (int m : outs)
      if (AX[m])
        CQF_RCUDA(cudaMemcpyAsync(AX[m], AXd[m], 2 * NN * sizeof(double), cudaMemcpyDeviceToHost,
                                  st));
  CQF_RCUDA(cudaStreamSynchronize(st));
  if (stats) {
    stats->quartets_total = (long long)cnt[0];
    stats->quartets_screened = (long long)cnt[1];
    stats->quartets_fp32 = (long long)cnt[2];
    stats->quartets_fp64 = (long long)cnt[3];
    float ms = 0.f;
    cudaEventElapsedTime(&ms, B->ev0, B->ev1);
    stats->device_ms = ms;
  }
  return CQF_OK;
}

void cqf_dc_opts_default(cqf_dc_opts* o) {
  if (!o) return;
  o->bare_coulomb = 1;
  o->dirac_coulomb = 1;
  o->dirac_coulomb_ssss = 1;
  o->libcint = 1;
  o->xHFX = 1.0;
  o->gaunt = 0;
  o->gauge = 0;
}

cqf_status cqf_four_comp_gd(cqf_basis* B, const void* const* D, void* const* G,
                            const cqf_dc_opts* dcIn, const cqf_opts* optsIn, cqf_stats* stats) {
  if (!B || !D || !G) return fail(CQF_EINVAL, "cqf_four_comp_gd: null argument");
  for (int c = 0; c < 4; c++)
    if (!D[c] || !G[c]) return fail(CQF_EINVAL, "cqf_four_comp_gd: null D or G component");
  cqf_dc_opts dc;
  cqf_dc_opts_default(&dc);
  if (dcIn) dc = *dcIn;
  cqf_opts o;
  cqf_opts_default(&o);
  if (optsIn) o = *optsIn;
  std::lock_guard<std::mutex> lk(B->mu);
  CQF_RCUDA(cudaSetDevice(B->device));
  cudaStream_t st = o.stream ? (cudaStream_t)o.stream : B->stream;
  const int N = B->nbasis;
  const size_t NN = (size_t)N * N, NN2 = 4 * NN;
  const double c2 = SPEED_OF_LIGHT * SPEED_OF_LIGHT;
  const double C2 = 1.0 / (4.0 * c2), C4 = 1.0 / (16.0 * c2 * c2);
  const bool exch = std::fabs(dc.xHFX) >= 1e-12;
  // workspace: rel scratch | blocks 16 x N^2 | AX 29 x N^2 | twoeH 4 x 4N^2 |
  // K 4 x 4N^2 | D/G staging (host pointers) 8 x 4N^2, all complex
  if (dc.dirac_coulomb) CQF_RTRY(rel_tables(B, CQF_REL_LLSS));
  if (dc.dirac_coulomb_ssss) CQF_RTRY(rel_tables(B, CQF_REL_SSSS));
  if (dc.gaunt) CQF_RTRY(rel_tables(B, CQF_REL_GAUNT));
  const size_t wsd = rel_ws_doubles(B);
  const size_t blkd = align32(2 * NN), bigd = align32(2 * NN2);
  const size_t total = wsd + 16 * blkd + CQF_REL_NMAT_GAUNT * blkd + 8 * bigd +
                       (o.device_pointers ? 0 : 8 * bigd);
  CQF_RTRY(ensure_relws(B, total * sizeof(double)));
  double* ws = static_cast<double*>(B->d_relws);
  double* blk = ws + wsd;
  double* axb = blk + 16 * blkd;
  double* twoeH = axb + CQF_REL_NMAT_GAUNT * blkd;
  double* Kb = twoeH + 4 * bigd;
  double* stage = Kb + 4 * bigd;
  const double* Dd[4];
  double* Gd[4];
  for (int c = 0; c < 4; c++) {
    if (o.device_pointers) {
      Dd[c] = static_cast<const double*>(D[c]);
      Gd[c] = static_cast<double*>(G[c]);
    } else {
      double* dd = stage + c * bigd;
      Dd[c] = dd;
      Gd[c] = stage + (4 + c) * bigd;
      CQF_RCUDA(cudaMemcpyAsync(dd, D[c], 2 * NN2 * sizeof(double), cudaMemcpyHostToDevice, st));
    }
  }
  CQF_RCUDA(cudaEventRecord(B->ev0, st));
  // LL / SS / LS (/ SL, for Gaunt) blocks of each Pauli component
  // (impl.hpp:3847-3857)
  auto B3 = [&](int k, int c) { return blk + (size_t)(k * 4 + c) * blkd; };
  const int ro[4] = {0, N, 0, N}, co[4] = {0, N, N, 0};
  for (int k = 0; k < (dc.gaunt || dc.gauge ? 4 : 3); k++)
    for (int c = 0; c < 4; c++)
      get_block_kernel<<<rgrid(NN, 256), 256, 0, st>>>(Dd[c], N, ro[k], co[k], B3(k, c));
  CQF_RCUDA(cudaMemsetAsync(twoeH, 0, 8 * bigd * sizeof(double), st));
  CQF_RCUDA(cudaGetLastError());
  const double* X[CQF_REL_NMAT_GAUNT];
  double* AX[CQF_REL_NMAT_GAUNT];
  X[CQF_CLLMS] = B3(0, 0);
  for (int c = 0; c < 4; c++) {
    X[CQF_XLLMS + c] = B3(0, c);
    X[CQF_CSSMS + c] = B3(1, c);
    X[CQF_XSSMS + c] = B3(1, c);
    X[CQF_XLSMS + c] = B3(2, c);
    X[CQF_CLSMS + c] = B3(2, c);
    X[CQF_CSLMS + c] = B3(3, c);
    X[CQF_XSLMS + c] = B3(3, c);
  }
  for (int m = 0; m < CQF_REL_NMAT_GAUNT; m++) AX[m] = axb + (size_t)m * blkd;
  auto H = [&](int c) { return twoeH + (size_t)c * bigd; };
  auto Kk = [&](int c) { return Kb + (size_t)c * bigd; };
  auto add = [&](double* M, int r0, int c0, const double* src, double f) {
    add_block_kernel<<<rgrid(NN, 256), 256, 0, st>>>(M, N, r0, c0, src, f);
  };
  unsigned long long cnt[4] = {0, 0, 0, 0};
  if (dc.bare_coulomb) {  // impl.hpp:3895-3969
    CQF_RTRY(rel_contract_dev(B, X, AX, CQF_REL_BARE_COULOMB, exch, o, st, ws, cnt));
    add(H(0), 0, 0, AX[CQF_CLLMS], dc.libcint ? 2.0 : 1.0);
    if (exch)
      for (int c = 0; c < 4; c++) add(Kk(c), 0, 0, AX[CQF_XLLMS + c], 1.0);
  }
  if (dc.dirac_coulomb) {  // impl.hpp:4003-4147
    CQF_RTRY(rel_contract_dev(B, X, AX, CQF_REL_LLSS, exch, o, st, ws, cnt));
    add(H(0), 0, 0, AX[CQF_CLLMS], 2.0 * C2);
    for (int c = 0; c < 4; c++) add(H(c), N, N, AX[CQF_CSSMS + c], 2.0 * C2);
    if (exch)
      for (int c = 0; c < 4; c++) add(Kk(c), 0, N, AX[CQF_XLSMS + c], -C2);
  }
  if (dc.dirac_coulomb_ssss) {  // impl.hpp:4149-4233
    CQF_RTRY(rel_contract_dev(B, X, AX, CQF_REL_SSSS, exch, o, st, ws, cnt));
    for (int c = 0; c < 4; c++) add(H(c), N, N, AX[CQF_CSSMS + c], 2.0 * C4);
    if (exch)
      for (int c = 0; c < 4; c++) add(Kk(c), N, N, AX[CQF_XSSMS + c], -C4);
  }
  // Gaunt and Gauge (impl.hpp:4228-4540): with the gauge term both are
  // weighted C2 / 2 (their sum is the Breit term)
  const double C2b = dc.gauge ? 0.5 * C2 : C2;
  for (int t : {(int)CQF_REL_GAUNT, (int)CQF_REL_GAUGE}) {
    if (!(t == CQF_REL_GAUNT ? dc.gaunt : dc.gauge)) continue;
    CQF_RTRY(rel_contract_dev(B, X, AX, t, exch, o, st, ws, cnt));
    for (int c = 0; c < 4; c++) add(H(c), 0, N, AX[CQF_CLSMS + c], 2.0 * C2b);
    if (exch)
      for (int c = 0; c < 4; c++) {
        add(Kk(c), 0, 0, AX[CQF_XLLMS + c], -C2b);
        add(Kk(c), N, N, AX[CQF_XSSMS + c], -C2b);
        add(Kk(c), 0, N, AX[CQF_XLSMS + c], -C2b);
      }
  }
  for (int c = 0; c < 4; c++)
    finish_gd_kernel<<<rgrid(NN2, 256), 256, 0, st>>>(H(c), Kk(c), N, dc.xHFX, exch ? 1 : 0,
                                                      Gd[c]);
  CQF_RCUDA(cudaGetLastError());
  CQF_RCUDA(cudaEventRecord(B->ev1, st));
  if (!o.device_pointers)
    for (int c = 0; c < 4; c++)
      CQF_RCUDA(cudaMemcpyAsync(G[c], Gd[c], 2 * NN2 * sizeof(double), cudaMemcpyDeviceToHost,
                                st));
  CQF_RCUDA(cudaStreamSynchronize(st));
  if (stats) {
    stats->quartets_total = (long long)cnt[0];
    stats->quartets_screened = (long long)cnt[1];
    stats->quartets_fp32 = (long long)cnt[2];
    stats->quartets_fp64 = (long long)cnt[3];
    float ms = 0.f;
    cudaEventElapsedTime(&ms, B->ev0, B->ev1);
    stats->device_ms = ms;
  }
  return CQF_OK;
}

}  // extern "C"
