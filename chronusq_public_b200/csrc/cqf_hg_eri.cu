// J and K of the class pairs with an f shell on the Hermite-matrix engine
// (cqf_hgemm.cuh): plain pairs on both sides, every matrix of the call
// digested from one quartet's integrals in shared memory.
//
// Quartet set, screen, roles and update formulas are those of the generic
// kernel (cqf_jk_kernels.cuh); the planning pass is the class kernels' one.
#include "cqf_digest.cuh"
#include "cqf_hg_digest.cuh"
#include "cqf_jk_plan.cuh"

namespace cqf {
namespace {

// Any matrix: one element per thread, the reference's four branches.
template <bool CPLX>
__device__ __forceinline__ void eri_digest_any(const JKLaunch& a, const HgQuartet& z, int fl,
                                               const double* __restrict__ X, double* A) {
  const PairDev& P = *z.P;
  const int nb = ncart(z.lb), nd = ncart(z.ld), nCD = z.cd1 - z.cd0;
  const int per = (z.ab1 - z.ab0) * nCD;
  for (int uu = threadIdx.x; uu < z.nk * per; uu += blockDim.x) {
    const int q = uu / per, e = uu - q * per;
    if (!z.have(q)) continue;
    const PairDev& Q = z.Q[q];
    const bool pRef = P.lex >= Q.lex;
    const bool swP = P.shA != P.s1, swQ = Q.shA != Q.s1;
    const PairDev &R12 = pRef ? P : Q, &R34 = pRef ? Q : P;
    const double deg = (R12.s1 == R12.s2 ? 1.0 : 2.0) * (R34.s1 == R34.s2 ? 1.0 : 2.0) *
                       (R12.s1 == R34.s1 && R12.s2 == R34.s2 ? 1.0 : 2.0);
    const int r = e / nCD, c = e - r * nCD, ab = z.ab0 + r, cd = z.cd0 + c;
    const int ga = P.cA + ab / nb, gb = P.cB + ab % nb, gc = Q.cA + cd / nd, gd = Q.cB + cd % nd;
    const int pa = swP ? gb : ga, pb = swP ? ga : gb;
    const int qc = swQ ? gd : gc, qd = swQ ? gc : gd;
    digest_one<CPLX>(fl, X, A, a.ncart, pRef ? pa : qc, pRef ? pb : qd, pRef ? qc : pa,
                     pRef ? qd : pb,
                     0.5 * deg * z.M[0][hg_row(r, z.ms[0]) + q * z.cw[0] + c]);
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
  __host__ __device__ static int stage(int la, int lb, int lc, int ld, int nk) {
    return CPLX ? 0 : hg_her_stage(la, lb, lc, ld, nk);
  }
  static __device__ __forceinline__ void digest(const JKLaunch& a, const HgQuartet& z) {
    const size_t stride = (size_t)a.ncart * a.ncart * (CPLX ? 2 : 1);
    for (int m = 0; m < a.nMat; m++) {
      const int fl = __ldg(a.flags + m);
      const double* X = a.Xc + m * stride;
      double* A = a.Ac + m * stride;
      if (!CPLX && (fl & 1)) {
        if (m > 0) __syncthreads();  // the last matrix's densities are done with
        hg_digest_her<1>(
            z, a.ncart, fl & 2, 1.0, false, X,
            [&](int q, int ab, int cd, double (&v)[1]) {
              v[0] = z.M[0][hg_row(ab, z.ms[0]) + q * z.cw[0] + cd];
            },
            [&](int, size_t e, const double (&s)[1]) {
              if (s[0] != 0.0) atomicAdd(A + e, s[0]);
            });
      } else {
        eri_digest_any<CPLX>(a, z, fl, X, A);
      }
    }
  }
};

}  // namespace

// Planning pass and engine of one class pair (cb | ck); either side may be
// the engine's bra: the one whose products need fewer matrix instructions.
cqf_status launch_jk_hg(const cqf_basis* B, JKLaunch a, int cb, int ck, uint2* masks,
                        long long maskWords, unsigned* work, double* win, cudaStream_t st) {
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
  auto plan = [&](const HgPart& p, uint2* mk, int* list64, int* list32, unsigned* lcount,
                  unsigned) {
    launch_jk_plan(p.of(a), mixed, false, mk, list64, list32, lcount, B->nsm, st);
  };
  const HgRegion r{masks, maskWords, work, win};
  return a.cplx ? hg_contract<EriDig<true>>(B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a,
                                            st, plan)
                : hg_contract<EriDig<false>>(B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a,
                                             st, plan);
}

}  // namespace cqf
