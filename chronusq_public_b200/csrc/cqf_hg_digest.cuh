// Hermitian digestion of one quartet on the Hermite-matrix engine, shared by
// the J/K and gradient contractions.
#pragma once

#include "cqf_hgemm.cuh"

namespace cqf {

// The reference's Hermitian updates of a real matrix (direct.hpp:1858-1918,
// :2470-2520) with the sums over the other two components taken before the
// atomic of each output element:
//   J(1,2) += X(4,3) I, J(4,3) += X(1,2) I;
//   K(1,3), (4,2), (4,1), (2,3) += h X(4,2), X(1,3), X(2,3), X(4,1) I,
// in the reference's roles of the four functions.  nCombo integrals per
// element (derivative components), val(k, ab, cd) (components counted from
// the chunk's first) into the accumulator acc(k); work units are (combo,
// output element, a share of the contracted bra components when the outputs
// alone do not fill the block).  xT: exchange densities are read with rows
// and columns exchanged in the updates whose row is function 1 or 2 (the
// gradient's orientation).
template <class V, class Acc>
__device__ __forceinline__ void hg_digest_her(const HgQuartet& z, size_t nc, bool exch, double f,
                                              bool xT, const double* __restrict__ X, int nCombo,
                                              V val, Acc acc) {
  const PairDev &P = *z.P, &Q = *z.Q;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int na = ncart(z.la), nb = ncart(z.lb), ncc = ncart(z.lc), nd = ncart(z.ld);
  const int nAB = z.ab1 - z.ab0, nCD = z.cd1 - z.cd0;
  const bool pRef = P.lex >= Q.lex;
  const bool swP = P.shA != P.s1, swQ = Q.shA != Q.s1;
  const PairDev &R12 = pRef ? P : Q, &R34 = pRef ? Q : P;
  const double deg = (R12.s1 == R12.s2 ? 1.0 : 2.0) * (R34.s1 == R34.s2 ? 1.0 : 2.0) *
                     (R12.s1 == R34.s1 && R12.s2 == R34.s2 ? 1.0 : 2.0);
  if (!exch) {
    const double v = 0.5 * f * deg;
    // rows of an output and of its density are the pair's first function
    // (1, 3) or its second
    for (int uu = tid; uu < nCombo * (nAB + nCD); uu += nt) {
      const int k0 = uu / (nAB + nCD), u = uu - k0 * (nAB + nCD);
      const bool toBra = u < nAB;
      const bool to12 = toBra == pRef;  // the output pair is (1, 2)
      const bool swO = toBra ? swP : swQ, swI = toBra ? swQ : swP;
      const PairDev& O = toBra ? P : Q;
      const PairDev& I = toBra ? Q : P;
      const int nO2 = toBra ? nb : nd, nI2 = toBra ? nd : nb;
      const int base = toBra ? z.cd0 : z.ab0, n = toBra ? nCD : nAB;
      // X's row is the first function of (1, 2) but the second of (4, 3)
      const bool rowFirstI = to12 ? swI : !swI;
      double s = 0.0;
      for (int k = 0; k < n; k++) {
        const int p = base + k, i = p / nI2, j = p - i * nI2;
        const int gi = I.cA + i, gj = I.cB + j;
        s += (toBra ? val(k0, u, k) : val(k0, k, u - nAB)) *
             __ldg(X + (rowFirstI ? gi + (size_t)gj * nc : gj + (size_t)gi * nc));
      }
      const int p = toBra ? z.ab0 + u : z.cd0 + (u - nAB), i = p / nO2, j = p - i * nO2;
      const int gi = O.cA + i, gj = O.cB + j;
      const bool rowFirstO = to12 ? !swO : swO;
      if (s != 0.0)
        atomicAdd(acc(k0) + (rowFirstO ? gi + (size_t)gj * nc : gj + (size_t)gi * nc), v * s);
    }
    return;
  }
  const double h = 0.25 * f * deg;
  const int total = 4 * nCombo * (na > nb ? na : nb) * (ncc > nd ? ncc : nd);
  for (int up = 0; up < 4; up++) {
    const bool f12 = up == 0 || up == 2, f34 = up == 0 || up == 3;  // first function of the pair
    const bool row12 = up == 0 || up == 3, rowI12 = !xT && (up == 1 || up == 2);
    const bool outA = (pRef ? f12 : f34) != swP, outC = (pRef ? f34 : f12) != swQ;
    const bool rowBra = row12 == pRef, rowBraI = rowI12 == pRef;
    const int no = outA ? na : nb, ni = outA ? nb : na;
    const int ko = outC ? ncc : nd, ki = outC ? nd : ncc;
    const int gO0 = outA ? P.cA : P.cB, gI0 = outA ? P.cB : P.cA;
    const int hO0 = outC ? Q.cA : Q.cB, hI0 = outC ? Q.cB : Q.cA;
    const int parts = total < nt ? ni : 1;
    for (int uu = tid; uu < nCombo * no * ko * parts; uu += nt) {
      const int k0 = uu / (no * ko * parts), u = uu - k0 * (no * ko * parts);
      const int part = u / (no * ko), r = u - part * (no * ko), kO = r / no, bO = r - kO * no;
      double s = 0.0;
#pragma unroll 1
      for (int bI = part; bI < ni; bI += parts) {
        const int ab = (outA ? bO * nb + bI : bI * nb + bO) - z.ab0;
        if (ab < 0 || ab >= nAB) continue;
        const int gb = gI0 + bI;
        for (int kI = 0; kI < ki; kI++) {
          const int cd = (outC ? kO * nd + kI : kI * nd + kO) - z.cd0;
          if (cd < 0 || cd >= nCD) continue;
          const int gk = hI0 + kI;
          s += val(k0, ab, cd) *
               __ldg(X + (rowBraI ? gb + (size_t)gk * nc : gk + (size_t)gb * nc));
        }
      }
      const int go = gO0 + bO, gp = hO0 + kO;
      if (s != 0.0)
        atomicAdd(acc(k0) + (rowBra ? go + (size_t)gp * nc : gp + (size_t)go * nc), h * s);
    }
  }
}

}  // namespace cqf
