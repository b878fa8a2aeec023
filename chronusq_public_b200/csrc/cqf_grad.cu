// Nuclear-gradient contraction on the device.
//
// Replaces DirectGradContraction::gradTwoBodyContract (include/
// particleintegrals/gradints.hpp:278-283) -> directScaffoldGrad
// (include/particleintegrals/contract/direct.hpp:2198-2571): for Hermitian
// real densities X, the J- and K-type contractions of the first derivatives
// of the ERIs with respect to every nuclear coordinate,
//   AX[atom, xyz] += 1/2 (A + A^T),  A = sum over quartets of
//   d(12|34)/dR_{atom,xyz} at the COULOMB / EXCHANGE update sites,
// over the reference's quartet set (unordered pairs of significant shell
// pairs, no screening: the reference's loop has none) with its degeneracy
// factors.  The derivative of a quartet with respect to the centre of one of
// its shells is minus the d/dr of that shell's functions; each of the 12
// (4 centres x 3 axes) goes to the component of the shell's atom.
//
// Quartets run on the Hermite-matrix engine (cqf_hgemm.cuh): the first
// derivatives on A and B against the plain ket, and the plain bra against
// those on C, are two matrix products per primitive quartet; those on D are
// minus the sum (translational invariance: against 50-digit integrals of an O
// and an H with s functions it is off by 1.4e-15 of the largest element, where
// the four centres' own derivatives, whose tight primitives amplify the rounding
// of P - A, were off by 4e-13).  The derivatives of one atom are
// summed before the digestion, and a quartet on a single atom, whose
// derivatives cancel, is dropped by the planning pass.  Accumulators are
// Cartesian, one per (component, matrix); the back transform symmetrises.
// FP64.  The kernel this replaces (one thread per quartet and ket component,
// 12 x 6 atomics per element) took 268 ms for (H2O)4 / cc-pVDZ.
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "cqf_hg_digest.cuh"
#include "cqf_internal.hpp"

namespace cqf {
namespace {

#define CQF_GCUDA(call)                                                                    \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return fail(e_ == cudaErrorMemoryAllocation ? CQF_ENOMEM : CQF_ECUDA,                \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                     \
  } while (0)

constexpr int GRAD_MAXMAT = 8;  // matrices per call

struct GradLaunch {
  const PairDev* pairs;
  int braBeg, nBra, braOff, ketBeg, nKet, same;
  int ncart, nMat;
  int type[GRAD_MAXMAT];  // COULOMB / EXCHANGE
  const int* shellAtom;   // per shell (device)
  const double* Xc;       // nMat Cartesian real densities
  double* Ac;             // (3 natom) x nMat Cartesian accumulators
  int shardIdx, shardCnt;
  unsigned long long* counters;
};

__global__ void __launch_bounds__(256)
    grad_plan_kernel(const GradLaunch a, uint2* __restrict__ masks, int* __restrict__ list64,
                     int* __restrict__ list32, unsigned* __restrict__ lcount) {
  hg_plan(a.nBra, a.nKet, masks, list64, list32, lcount, a.counters,
          [&](int ib, int jk, bool& work, bool&) {
            if ((a.same && jk > ib + a.braOff) ||
                !in_shard(a.braBeg + ib, a.shardIdx, a.shardCnt))
              return false;
            const PairDev P = a.pairs[a.braBeg + ib], Q = a.pairs[a.ketBeg + jk];
            const int t = __ldg(a.shellAtom + P.shA);
            work = __ldg(a.shellAtom + P.shB) != t || __ldg(a.shellAtom + Q.shA) != t ||
                   __ldg(a.shellAtom + Q.shB) != t;
            return true;
          });
}

struct GradDig {
  using Args = GradLaunch;
  static constexpr int NP = 2, ABU = 16, CDU = 16;
  __host__ __device__ static constexpr int tb(int q) { return q == 0 ? HG_D6 : HG_PLAIN; }
  __host__ __device__ static constexpr int tk(int q) { return q == 0 ? HG_PLAIN : HG_D3; }
  __host__ __device__ static constexpr int rtu(int q) { return q == 0 ? 6 : 1; }
  __host__ __device__ static constexpr int ctu(int q) { return q == 0 ? 1 : 3; }
  __host__ __device__ static int stage(int la, int lb, int lc, int ld, int nk) {
    return hg_her_stage(la, lb, lc, ld, nk);
  }
  static __device__ __forceinline__ void digest(const GradLaunch& a, const HgQuartet& z) {
    const PairDev& P = *z.P;
    const int aA = __ldg(a.shellAtom + P.shA), aB = __ldg(a.shellAtom + P.shB);
    const double *M0 = z.M[0], *M1 = z.M[1];
    const int m0 = z.ms[0], m1 = z.ms[1];
    const size_t nc2 = (size_t)a.ncart * a.ncart;
    // the nine derivatives on A, B and C; the one on D is minus their sum.
    // Each atom gets the sum of its functions' (d/dR = -d/dr is the factor -1
    // below)
    auto val = [&](int q, int ab, int cd, double (&v)[9]) {
#pragma unroll
      for (int k = 0; k < 6; k++) v[k] = M0[hg_row(6 * ab + k, m0) + q * z.cw[0] + cd];
#pragma unroll
      for (int x = 0; x < 3; x++) v[6 + x] = M1[hg_row(ab, m1) + q * z.cw[1] + 3 * cd + x];
    };
    for (int mt = 0; mt < a.nMat; mt++) {
      if (mt > 0) __syncthreads();  // the last matrix's densities are done with
      hg_digest_her<9>(
          z, a.ncart, a.type[mt] != CQF_COULOMB, -1.0, true, a.Xc + mt * nc2, val,
          [&](int q, size_t e, const double (&s)[9]) {
            const int aC = __ldg(a.shellAtom + z.Q[q].shA), aD = __ldg(a.shellAtom + z.Q[q].shB);
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const int t = k == 0 ? aA : (k == 1 ? aB : (k == 2 ? aC : aD));
              if ((k > 0 && t == aA) || (k > 1 && t == aB) || (k > 2 && t == aC)) continue;
              const double w = t == aD ? -1.0 : 0.0;
              const double wa = w + (t == aA), wb = w + (t == aB), wc = w + (t == aC);
#pragma unroll
              for (int x = 0; x < 3; x++) {
                const double v = wa * s[x] + wb * s[3 + x] + wc * s[6 + x];
                if (v != 0.0) atomicAdd(a.Ac + ((size_t)(t * 3 + x) * a.nMat + mt) * nc2 + e, v);
              }
            }
          });
    }
  }
};

}  // namespace
}  // namespace cqf

using namespace cqf;

extern "C" {

cqf_status cqf_grad_two_body_contract(cqf_basis* B, const int* shell_atom, int natom,
                                      const cqf_contraction* list, int nMat, void* const* AX,
                                      const cqf_opts* optsIn, cqf_stats* stats) {
  if (!B || !shell_atom || !list || !AX || natom < 1 || nMat < 1)
    return fail(CQF_EINVAL, "cqf_grad_two_body_contract: null or empty argument");
  if (nMat > GRAD_MAXMAT)
    return fail(CQF_EINVAL, "cqf_grad_two_body_contract: at most 8 matrices per call");
  cqf_opts o;
  cqf_opts_default(&o);
  if (optsIn) o = *optsIn;
  if (o.is_complex)
    return fail(CQF_EINVAL, "cqf_grad_two_body_contract: complex densities are not built");
  if (o.shard_count < 1 || o.shard_index < 0 || o.shard_index >= o.shard_count)
    return fail(CQF_EINVAL, "shard_index must lie in [0, shard_count)");
  for (int m = 0; m < nMat; m++) {
    if (!list[m].X) return fail(CQF_EINVAL, "cqf_grad_two_body_contract: null X");
    // the reference stops on non-Hermitian gradient contractions (:2539-2541)
    if (!list[m].hermitian)
      return fail(CQF_EINVAL, "cqf_grad_two_body_contract: non-Hermitian X is not built");
    if (list[m].type != CQF_COULOMB && list[m].type != CQF_EXCHANGE)
      return fail(CQF_EINVAL, "cqf_grad_two_body_contract: COULOMB or EXCHANGE only");
  }
  const int nGrad = 3 * natom;
  for (int k = 0; k < nGrad * nMat; k++)
    if (!AX[k]) return fail(CQF_EINVAL, "cqf_grad_two_body_contract: null AX");
  for (int s = 0; s < B->nshell; s++)
    if (shell_atom[s] < 0 || shell_atom[s] >= natom)
      return fail(CQF_EINVAL, "cqf_grad_two_body_contract: shell_atom outside [0, natom)");
  std::lock_guard<std::mutex> lk(B->mu);
  CQF_GCUDA(cudaSetDevice(B->device));
  cudaStream_t st = o.stream ? (cudaStream_t)o.stream : B->stream;
  const int N = B->nbasis, nc = B->ncart;
  const size_t NN = (size_t)N * N, nc2 = (size_t)nc * nc;
  // scratch (stream-ordered): shell atoms | Cartesian X | Cartesian
  // accumulators | host staging of X and AX
  const size_t host = o.device_pointers ? 0 : (size_t)nMat * NN + (size_t)nGrad * nMat * NN;
  // then, per launch stream, the planning pass's masks and lists, four
  // counters, and windows of the tables that the basis does not hold
  size_t row = 1;
  for (int c = 0; c < NCLS; c++)
    row = std::max(row, ((size_t)B->cls_cnt[c] + WTILE - 1) / WTILE);
  const size_t maskWords = std::max(row, MASK_CAP_WORDS);
  const size_t lists = (2 * maskWords + 2) * (NAUX + 1);
  const size_t fixed = ((size_t)nMat * nc2 + (size_t)nGrad * nMat * nc2 + host + 1) / 2 * 2;
  for (int k : {(int)HG_PLAIN, (int)HG_D6, (int)HG_D3}) {
    const cqf_status s = hg_ensure(B, k);
    if (s != CQF_OK) return s;
  }
  const size_t winDoubles = hg_windows<GradDig>(B);
  const size_t doubles = fixed + lists + winDoubles * (NAUX + 1);
  double* ws = nullptr;
  int* dAtom = nullptr;
  CQF_GCUDA(cudaMallocAsync(&ws, doubles * sizeof(double), st));
  CQF_GCUDA(cudaMallocAsync(&dAtom, (size_t)B->nshell * sizeof(int), st));
  double* Xc = ws;
  double* Ac = Xc + (size_t)nMat * nc2;
  double* hX = Ac + (size_t)nGrad * nMat * nc2;
  double* hAX = hX + (size_t)nMat * NN;
  CQF_GCUDA(cudaMemcpyAsync(dAtom, shell_atom, (size_t)B->nshell * sizeof(int),
                            cudaMemcpyHostToDevice, st));
  if (!o.device_pointers)
    for (int m = 0; m < nMat; m++)
      CQF_GCUDA(cudaMemcpyAsync(hX + (size_t)m * NN, list[m].X, NN * sizeof(double),
                                cudaMemcpyHostToDevice, st));
  auto noMode = [](int) { return 0; };
  mat_batches(
      nMat, nc2,
      [&](int m) {
        return o.device_pointers ? static_cast<const double*>(list[m].X) : hX + (size_t)m * NN;
      },
      [&](int m) { return Xc + (size_t)m * nc2; }, noMode,
      [&](const MatList& l, int n) { launch_to_cart(B, l, n, 0, st); });
  CQF_GCUDA(cudaMemsetAsync(Ac, 0, (size_t)nGrad * nMat * nc2 * sizeof(double), st));
  CQF_GCUDA(cudaMemsetAsync(B->d_counters, 0, 4 * sizeof(unsigned long long), st));
  CQF_GCUDA(cudaEventRecord(B->ev0, st));

  GradLaunch a{};
  a.pairs = B->d_pairs;
  a.ncart = nc;
  a.nMat = nMat;
  for (int m = 0; m < nMat; m++) a.type[m] = list[m].type;
  a.shellAtom = dAtom;
  a.Xc = Xc;
  a.Ac = Ac;
  a.shardIdx = o.shard_index;
  a.shardCnt = o.shard_count;
  a.counters = B->d_counters;
  // class pairs round-robin over the call's stream and the auxiliary ones
  // (they only add into the accumulators), the largest first
  uint2* masks = reinterpret_cast<uint2*>(ws + fixed);
  unsigned* work = reinterpret_cast<unsigned*>(masks + 2 * maskWords * (NAUX + 1));
  double* win = ws + fixed + lists;
  CQF_GCUDA(cudaEventRecord(B->evFork, st));
  cudaStream_t lanes[NAUX + 1] = {st};
  for (int i = 0; i < NAUX; i++) {
    lanes[1 + i] = B->aux[i];
    CQF_GCUDA(cudaStreamWaitEvent(B->aux[i], B->evFork, 0));
  }
  int nlaunch = 0;
  cqf_status rc = CQF_OK;
  for (int cb = NCLS - 1; cb >= 0; cb--)
    for (int ck = cb; ck >= 0 && rc == CQF_OK; ck--) {
      if (!B->cls_cnt[cb] || !B->cls_cnt[ck]) continue;
      a.braBeg = B->cls_beg[cb];
      a.nBra = B->cls_cnt[cb];
      a.ketBeg = B->cls_beg[ck];
      a.nKet = B->cls_cnt[ck];
      a.same = (cb == ck);
      const int li = nlaunch++ % (NAUX + 1);
      const cudaStream_t ls = lanes[li];
      const HgRegion r{masks + 2 * maskWords * li, (long long)maskWords, work + 4 * li,
                       win + winDoubles * li};
      rc = hg_contract<GradDig>(
          B, cb, ck, a.braBeg, a.nBra, a.ketBeg, a.nKet, r, a, ls,
          [&](const HgPart& p, uint2* mk, int* list64, int* list32, unsigned* lcount,
              unsigned gp) {
            grad_plan_kernel<<<gp, 256, 0, ls>>>(p.of(a), mk, list64, list32, lcount);
          });
    }
  for (int i = 0; i < NAUX; i++) {
    CQF_GCUDA(cudaEventRecord(B->evJoin[i], B->aux[i]));
    CQF_GCUDA(cudaStreamWaitEvent(st, B->evJoin[i], 0));
  }
  if (rc != CQF_OK) {
    cudaFreeAsync(ws, st);
    cudaFreeAsync(dAtom, st);
    return rc;
  }
  CQF_GCUDA(cudaGetLastError());
  // AX += 1/2 (A + A^T) per component and matrix (:2550-2560)
  if (!o.device_pointers)
    for (int k = 0; k < nGrad * nMat; k++)
      CQF_GCUDA(cudaMemcpyAsync(hAX + (size_t)k * NN, AX[k], NN * sizeof(double),
                                cudaMemcpyHostToDevice, st));
  mat_batches(
      nGrad * nMat, NN, [&](int k) { return Ac + (size_t)k * nc2; },
      [&](int k) {
        return o.device_pointers ? static_cast<double*>(AX[k]) : hAX + (size_t)k * NN;
      },
      [](int) { return 1; },
      [&](const MatList& l, int n) { launch_from_cart(B, l, n, 0, st); });
  CQF_GCUDA(cudaGetLastError());
  CQF_GCUDA(cudaEventRecord(B->ev1, st));
  if (!o.device_pointers)
    for (int k = 0; k < nGrad * nMat; k++)
      CQF_GCUDA(cudaMemcpyAsync(AX[k], hAX + (size_t)k * NN, NN * sizeof(double),
                                cudaMemcpyDeviceToHost, st));
  unsigned long long h[4];
  CQF_GCUDA(cudaMemcpyAsync(h, B->d_counters, sizeof(h), cudaMemcpyDeviceToHost, st));
  cudaFreeAsync(ws, st);
  cudaFreeAsync(dAtom, st);
  CQF_GCUDA(cudaStreamSynchronize(st));
  if (stats) {
    stats->quartets_total = (long long)h[0];
    stats->quartets_screened = (long long)h[1];  // on one atom: the derivatives cancel
    stats->quartets_fp32 = 0;
    stats->quartets_fp64 = (long long)h[3];
    float ms = 0.f;
    cudaEventElapsedTime(&ms, B->ev0, B->ev1);
    stats->device_ms = ms;
  }
  return CQF_OK;
}

}  // extern "C"
