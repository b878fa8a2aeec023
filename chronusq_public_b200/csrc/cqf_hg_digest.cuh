// Hermitian digestion of one quartet on the Hermite-matrix engine, shared by
// the J/K and gradient contractions.
#pragma once

#include "cqf_hgemm.cuh"

namespace cqf {

// The reference's Hermitian updates of a real matrix (direct.hpp:1858-1918,
// :2470-2520) with the sums over the other two components taken before the
// atomics of each output element:
//   J(1,2) += X(4,3) I, J(4,3) += X(1,2) I;
//   K(1,3), (4,2), (4,1), (2,3) += h X(4,2), X(1,3), X(2,3), X(4,1) I,
// in the reference's roles of the four functions.  An element has NV
// integrals (derivative components), val(q, ab, cd, v) of ket q (components
// counted from the chunk's first); out(q, element, s) adds their sums, scaled.
// The density blocks are read once into shared memory, in the orientation
// their update wants.  Work units are (ket, output element), shared by a few
// lanes where there are few.
// xT: exchange densities are read with rows and columns exchanged in the
// updates whose row is function 1 or 2 (the gradient's orientation).
struct HgRoles {
  bool pRef, swP, swQ;
  double deg;
};
__device__ __forceinline__ HgRoles hg_roles(const PairDev& P, const PairDev& Q) {
  HgRoles r;
  r.pRef = P.lex >= Q.lex;
  r.swP = P.shA != P.s1;
  r.swQ = Q.shA != Q.s1;
  const PairDev &R12 = r.pRef ? P : Q, &R34 = r.pRef ? Q : P;
  r.deg = (R12.s1 == R12.s2 ? 1.0 : 2.0) * (R34.s1 == R34.s2 ? 1.0 : 2.0) *
          (R12.s1 == R34.s1 && R12.s2 == R34.s2 ? 1.0 : 2.0);
  return r;
}
__host__ __device__ inline int hg_her_stage(int la, int lb, int lc, int ld, int nk) {
  const int nx = (ncart(la) + ncart(lb)) * (ncart(lc) + ncart(ld));
  const int nj = ncart(la) * ncart(lb) + ncart(lc) * ncart(ld);
  return nk * (nx > nj ? nx : nj);
}
template <int NV, class V, class Out>
__device__ __forceinline__ void hg_digest_her(const HgQuartet& z, int nc, bool exch, double f,
                                              bool xT, const double* __restrict__ X, V val,
                                              Out out) {
  const PairDev& P = *z.P;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int na = ncart(z.la), nb = ncart(z.lb), ncc = ncart(z.lc), nd = ncart(z.ld);
  const int nAB = z.ab1 - z.ab0, nCD = z.cd1 - z.cd0;
  double* xs = z.st;
  if (!exch) {
    // rows of an output and of its density are the pair's first function
    // (1, 3) or its second; X's row is the first function of (1, 2) but the
    // second of (4, 3).  Per ket: X over ab (orders J(cd)), X over cd
    const int per = nAB + nCD;
    for (int uu = tid; uu < z.nk * per; uu += nt) {
      const int q = uu / per, u = uu - q * per;
      const PairDev& Q = z.Q[q];
      const HgRoles ro = hg_roles(P, Q);
      const bool bra = u < nAB;
      const bool is12 = bra == ro.pRef, sw = bra ? ro.swP : ro.swQ;
      const int p = bra ? z.ab0 + u : z.cd0 + u - nAB, n2 = bra ? nb : nd;
      const int i = p / n2, j = p - i * n2;
      const int gi = (bra ? P.cA : Q.cA) + i, gj = (bra ? P.cB : Q.cB) + j;
      const bool rowFirst = is12 ? !sw : sw;
      xs[uu] = __ldg(X + (rowFirst ? gi + (size_t)gj * nc : gj + (size_t)gi * nc));
    }
    __syncthreads();
    for (int uu = tid; uu < z.nk * per; uu += nt) {
      const int q = uu / per, u = uu - q * per;
      if (!z.have(q)) continue;
      const PairDev& Q = z.Q[q];
      const HgRoles ro = hg_roles(P, Q);
      const bool bra = u < nAB;
      const double* x = xs + q * per + (bra ? nAB : 0);
      double s[NV];
#pragma unroll
      for (int k = 0; k < NV; k++) s[k] = 0.0;
      for (int k = 0; k < (bra ? nCD : nAB); k++) {
        double v[NV];
        val(q, bra ? u : k, bra ? k : u - nAB, v);
#pragma unroll
        for (int t = 0; t < NV; t++) s[t] += v[t] * x[k];
      }
      const bool is12 = bra == ro.pRef, sw = bra ? ro.swP : ro.swQ;
      const int p = bra ? z.ab0 + u : z.cd0 + u - nAB, n2 = bra ? nb : nd;
      const int i = p / n2, j = p - i * n2;
      const int gi = (bra ? P.cA : Q.cA) + i, gj = (bra ? P.cB : Q.cB) + j;
      const bool rowFirst = is12 ? !sw : sw;
#pragma unroll
      for (int k = 0; k < NV; k++) s[k] *= 0.5 * f * ro.deg;
      out(q, rowFirst ? gi + (size_t)gj * nc : gj + (size_t)gi * nc, s);
    }
    return;
  }
  // (output A or B) x (output C or D): from the roles, whether the output's
  // row and the density's row are the bra's function.  (1,3), (2,3) have row
  // (1,2) and read X with row (3,4); (4,2), (4,1) the reverse
  const int nx = (na + nb) * (ncc + nd);
  for (int uu = tid; uu < z.nk * nx; uu += nt) {
    const int q = uu / nx, r = uu - q * nx, i = r / (ncc + nd), j = r - i * (ncc + nd);
    const PairDev& Q = z.Q[q];
    const HgRoles ro = hg_roles(P, Q);
    const bool inA = i < na, inC = j < ncc;
    // the output holds the first function of (3, 4): it has the other bra
    // and the other ket function
    const bool f34 = ro.pRef ? (!inC != ro.swQ) : (!inA != ro.swP);
    const bool rowBra = (!xT && !f34) == ro.pRef;
    const int gb = inA ? P.cA + i : P.cB + i - na, gk = inC ? Q.cA + j : Q.cB + j - ncc;
    xs[uu] = __ldg(X + (rowBra ? gb + (size_t)gk * nc : gk + (size_t)gb * nc));
  }
  __syncthreads();
  const int sh = hg_share(z.nk * nx, na < nb ? na : nb);
  for (int uu = tid; uu < ((z.nk * nx) << sh); uu += nt) {
    const int part = uu & ((1 << sh) - 1), w = uu >> sh, q = w / nx, r = w - q * nx;
    if (!z.have(q)) continue;
    const int kO2 = r / (na + nb), bO2 = r - kO2 * (na + nb);
    const bool outA = bO2 < na, outC = kO2 < ncc;
    const int bO = outA ? bO2 : bO2 - na, kO = outC ? kO2 : kO2 - ncc;
    const int ni = outA ? nb : na, ki = outC ? nd : ncc;
    const int abI = outA ? 1 : nb, cdI = outC ? 1 : nd;
    const int ab0 = (outA ? bO * nb : bO) - z.ab0, cd0 = (outC ? kO * nd : kO) - z.cd0;
    const PairDev& Q = z.Q[q];
    const HgRoles ro = hg_roles(P, Q);
    const double* xq = xs + q * nx + (outA ? na : 0) * (ncc + nd) + (outC ? ncc : 0);
    int k0, k1;  // the contracted ket components in the chunk
    hg_range(cd0, cdI, ki, nCD, k0, k1);
    double s[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) s[k] = 0.0;
#pragma unroll 1
    for (int bI = part; bI < ni; bI += 1 << sh) {
      const int ab = ab0 + bI * abI;
      if (ab < 0 || ab >= nAB) continue;
      const double* x = xq + bI * (ncc + nd);
      for (int kI = k0; kI < k1; kI++) {
        double v[NV];
        val(q, ab, cd0 + kI * cdI, v);
#pragma unroll
        for (int t = 0; t < NV; t++) s[t] += v[t] * x[kI];
      }
    }
    if (sh > 0) {
#pragma unroll
      for (int k = 0; k < NV; k++) s[k] = hg_group_sum(s[k], sh);
      if (part) continue;
    }
    const bool f34 = ro.pRef ? (outC != ro.swQ) : (outA != ro.swP);
    const bool rowBra = f34 == ro.pRef;
    const int go = (outA ? P.cA : P.cB) + bO, gp = (outC ? Q.cA : Q.cB) + kO;
#pragma unroll
    for (int k = 0; k < NV; k++) s[k] *= 0.25 * f * ro.deg;
    out(q, rowBra ? go + (size_t)gp * nc : gp + (size_t)go * nc, s);
  }
}

}  // namespace cqf
