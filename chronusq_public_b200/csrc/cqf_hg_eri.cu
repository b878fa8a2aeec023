// J and K of the class pairs with an f shell on the Hermite-matrix engine
// (cqf_hgemm.cuh): plain pairs on both sides, every matrix of the call
// digested from one quartet's integrals in shared memory.
//
// Quartet set, screen, roles and update formulas are those of the generic
// kernel (cqf_jk_kernels.cuh); the planning pass is the class kernels' one.
#include "cqf_digest.cuh"
#include "cqf_hgemm.cuh"
#include "cqf_jk_plan.cuh"

namespace cqf {
namespace {

// Hermitian real matrices (and the antisymmetric part of a complex split):
// the reference's Hermitian updates (direct.hpp:1858-1918) with the sums over
// the other two components taken before the atomic of each output element.
__device__ __forceinline__ void eri_digest_her(const JKLaunch& a, const HgQuartet& z, bool exch,
                                               const double* __restrict__ X, double* A) {
  const PairDev &P = *z.P, &Q = *z.Q;
  const int tid = threadIdx.x, nt = blockDim.x, ms = z.ms[0];
  const double* M = z.M[0];
  const size_t nc = a.ncart;
  const int na = ncart(z.la), nb = ncart(z.lb), ncc = ncart(z.lc), nd = ncart(z.ld);
  const int nAB = z.ab1 - z.ab0, nCD = z.cd1 - z.cd0;
  const bool pRef = P.lex >= Q.lex;
  const bool swP = P.shA != P.s1, swQ = Q.shA != Q.s1;
  const PairDev &R12 = pRef ? P : Q, &R34 = pRef ? Q : P;
  const double deg = (R12.s1 == R12.s2 ? 1.0 : 2.0) * (R34.s1 == R34.s2 ? 1.0 : 2.0) *
                     (R12.s1 == R34.s1 && R12.s2 == R34.s2 ? 1.0 : 2.0);
  if (!exch) {
    const double v = 0.5 * deg;
    // J(1,2) += X(4,3) I, J(4,3) += X(1,2) I: rows of an output and of its
    // density are the pair's first function (1, 3) or its second
    for (int u = tid; u < nAB + nCD; u += nt) {
      const bool toBra = u < nAB;
      const bool to12 = toBra == pRef;  // the output pair is (1, 2)
      const bool swO = toBra ? swP : swQ, swI = toBra ? swQ : swP;
      const PairDev& O = toBra ? P : Q;
      const PairDev& I = toBra ? Q : P;
      const int nO2 = toBra ? nb : nd, nI2 = toBra ? nd : nb;
      const int base = toBra ? z.cd0 : z.ab0, n = toBra ? nCD : nAB;
      const double* m = toBra ? M + (size_t)u * ms : M + (u - nAB);
      const int st = toBra ? 1 : ms;
      // X's row is the first function of (1, 2) but the second of (4, 3)
      const bool rowFirstI = to12 ? swI : !swI;
      double s = 0.0;
      for (int k = 0; k < n; k++) {
        const int p = base + k, i = p / nI2, j = p - i * nI2;
        const int gi = I.cA + i, gj = I.cB + j;
        s += m[(size_t)k * st] * __ldg(X + (rowFirstI ? gi + (size_t)gj * nc : gj + (size_t)gi * nc));
      }
      const int p = toBra ? z.ab0 + u : z.cd0 + (u - nAB), i = p / nO2, j = p - i * nO2;
      const int gi = O.cA + i, gj = O.cB + j;
      const bool rowFirstO = to12 ? !swO : swO;
      atomicAdd(A + (rowFirstO ? gi + (size_t)gj * nc : gj + (size_t)gi * nc), v * s);
    }
    return;
  }
  const double h = 0.25 * deg;
  const int total = 4 * (na > nb ? na : nb) * (ncc > nd ? ncc : nd);
  for (int up = 0; up < 4; up++) {
    // outputs (1,3), (4,2), (4,1), (2,3) from X(4,2), X(1,3), X(2,3), X(4,1)
    const bool f12 = up == 0 || up == 2, f34 = up == 0 || up == 3;  // first function of the pair
    const bool row12 = up == 0 || up == 3, rowI12 = up == 1 || up == 2;
    const bool outA = (pRef ? f12 : f34) != swP, outC = (pRef ? f34 : f12) != swQ;
    const bool rowBra = row12 == pRef, rowBraI = rowI12 == pRef;
    const int no = outA ? na : nb, ni = outA ? nb : na;
    const int ko = outC ? ncc : nd, ki = outC ? nd : ncc;
    const int gO0 = outA ? P.cA : P.cB, gI0 = outA ? P.cB : P.cA;
    const int hO0 = outC ? Q.cA : Q.cB, hI0 = outC ? Q.cB : Q.cA;
    const int parts = total < nt ? ni : 1;
    for (int u = tid; u < no * ko * parts; u += nt) {
      const int part = u / (no * ko), r = u - part * (no * ko), kO = r / no, bO = r - kO * no;
      double s = 0.0;
#pragma unroll 1
      for (int bI = part; bI < ni; bI += parts) {
        const int ab = (outA ? bO * nb + bI : bI * nb + bO) - z.ab0;
        if (ab < 0 || ab >= nAB) continue;
        const double* m = M + (size_t)ab * ms;
        const int gb = gI0 + bI;
        for (int kI = 0; kI < ki; kI++) {
          const int cd = (outC ? kO * nd + kI : kI * nd + kO) - z.cd0;
          if (cd < 0 || cd >= nCD) continue;
          const int gk = hI0 + kI;
          s += m[cd] * __ldg(X + (rowBraI ? gb + (size_t)gk * nc : gk + (size_t)gb * nc));
        }
      }
      const int go = gO0 + bO, gp = hO0 + kO;
      if (s != 0.0) atomicAdd(A + (rowBra ? go + (size_t)gp * nc : gp + (size_t)go * nc), h * s);
    }
  }
}

// Any matrix: one element per thread, the reference's four branches.
template <bool CPLX>
__device__ __forceinline__ void eri_digest_any(const JKLaunch& a, const HgQuartet& z, int fl,
                                               const double* __restrict__ X, double* A) {
  const PairDev &P = *z.P, &Q = *z.Q;
  const int nb = ncart(z.lb), nd = ncart(z.ld), nCD = z.cd1 - z.cd0;
  const bool pRef = P.lex >= Q.lex;
  const bool swP = P.shA != P.s1, swQ = Q.shA != Q.s1;
  const PairDev &R12 = pRef ? P : Q, &R34 = pRef ? Q : P;
  const double deg = (R12.s1 == R12.s2 ? 1.0 : 2.0) * (R34.s1 == R34.s2 ? 1.0 : 2.0) *
                     (R12.s1 == R34.s1 && R12.s2 == R34.s2 ? 1.0 : 2.0);
  for (int e = threadIdx.x; e < (z.ab1 - z.ab0) * nCD; e += blockDim.x) {
    const int r = e / nCD, c = e - r * nCD, ab = z.ab0 + r, cd = z.cd0 + c;
    const int ga = P.cA + ab / nb, gb = P.cB + ab % nb, gc = Q.cA + cd / nd, gd = Q.cB + cd % nd;
    const int pa = swP ? gb : ga, pb = swP ? ga : gb;
    const int qc = swQ ? gd : gc, qd = swQ ? gc : gd;
    digest_one<CPLX>(fl, X, A, a.ncart, pRef ? pa : qc, pRef ? pb : qd, pRef ? qc : pa,
                     pRef ? qd : pb, 0.5 * deg * z.M[0][(size_t)r * z.ms[0] + c]);
  }
}

template <bool CPLX>
struct EriDig {
  using Args = JKLaunch;
  static constexpr int NP = 1, ABU = 16, CDU = 16;
  __host__ __device__ static constexpr int tb(int) { return HG_PLAIN; }
  __host__ __device__ static constexpr int tk(int) { return HG_PLAIN; }
  __host__ __device__ static constexpr int rtu(int) { return 1; }
  __host__ __device__ static constexpr int ctu(int) { return 1; }
  static __device__ __forceinline__ void digest(const JKLaunch& a, const HgQuartet& z) {
    const size_t stride = (size_t)a.ncart * a.ncart * (CPLX ? 2 : 1);
    for (int m = 0; m < a.nMat; m++) {
      const int fl = __ldg(a.flags + m);
      const double* X = a.Xc + m * stride;
      double* A = a.Ac + m * stride;
      if (!CPLX && (fl & 1)) eri_digest_her(a, z, fl & 2, X, A);
      else eri_digest_any<CPLX>(a, z, fl, X, A);
    }
  }
};

}  // namespace

// Planning pass and engine of one class pair (cb | ck); either side may be
// the engine's bra: the one whose products need fewer matrix instructions.
cqf_status launch_jk_hg(const cqf_basis* B, JKLaunch a, int cb, int ck, uint2* masks,
                        long long maskWords, unsigned* work, cudaStream_t st) {
  if (a.nBra == 0 || a.nKet == 0) return CQF_OK;
  auto cost = [](int b, int k) {
    int la, lb, lc, ld;
    class_ls(b, la, lb);
    class_ls(k, lc, ld);
    const int rt = hg_tiles(HG_PLAIN, la, lb), ct = hg_tiles(HG_PLAIN, lc, ld);
    const int hb = nherm(la + lb);
    return ct * ((hb + 7) / 8) * hg_ktiles(HG_PLAIN, lc, ld) + 2 * ct * rt * ((hb + 3) / 4);
  };
  if (cost(ck, cb) < cost(cb, ck)) {
    std::swap(cb, ck);
    std::swap(a.braBeg, a.ketBeg);
    std::swap(a.nBra, a.nKet);
  }
  int la, lb, lc, ld;
  class_ls(cb, la, lb);
  class_ls(ck, lc, ld);
  a.lsum = la + lb + lc + ld;
  const bool mixed = a.precision == 1 && a.fp32_cut > 0.0;
  auto plan = [&](int ib0, int n, uint2* mk, int* list64, int* list32, unsigned* lcount,
                  unsigned) {
    JKLaunch c = a;
    c.braBeg = a.braBeg + ib0;
    c.nBra = n;
    c.braOff = ib0;
    launch_jk_plan(c, mixed, mk, list64, list32, lcount, B->nsm, st);
  };
  const HgRegion r{masks, maskWords, work};
  return a.cplx ? hg_contract<EriDig<true>>(B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a,
                                            st, plan)
                : hg_contract<EriDig<false>>(B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a,
                                             st, plan);
}

}  // namespace cqf
