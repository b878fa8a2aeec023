// Coefficient tables of the Hermite-matrix engine (cqf_hgemm.cuh).
#include <string>

#include "cqf_deriv.cuh"
#include "cqf_hgemm.cuh"
#include "cqf_once.hpp"

namespace cqf {
namespace {

constexpr int HT_THREADS = 128;

// Hermite length bound of one axis' factor (both derivatives)
__host__ __device__ inline int ht_fl(int la, int lb) { return la + lb + 3; }
__host__ __device__ inline int ht_e1(int la, int lb) { return (la + 2) * (lb + 2) * (la + lb + 3); }

// One block per primitive pair (pair beg + blockIdx.x, primitives from blockIdx.y on):
// the 1D tables raised by one on both centres, the factors of every axis,
// exponent pair and derivative type, then every entry of the table in
// fragment order.
__global__ void __launch_bounds__(HT_THREADS)
    hg_table_kernel(const PairDev* __restrict__ pairs, const PrimPairDev* __restrict__ pp,
                    const ShellDev* __restrict__ shells, const double* __restrict__ prim, int beg,
                    int ppBeg, int kind, int la, int lb, double* __restrict__ tab) {
  extern __shared__ double sm[];
  const PairDev P = pairs[beg + blockIdx.x];
  const int tid = threadIdx.x;
  for (int ip = blockIdx.y; ip < P.npp; ip += gridDim.y) {
    const PrimPairDev A = pp[P.pp_off + ip];
    double ea, eb;
    pair_exps(shells[P.shA], shells[P.shB], prim, A, ea, eb);
    const int E1 = ht_e1(la, lb), FL = ht_fl(la, lb);
    double* E = sm;
    double* fa = sm + 3 * E1;
    if (tid < 3)
      hermite_E_rt<double, LMAX + 1>(la + 1, lb + 1, A.o2p, A.PA[tid], A.PB[tid], E + tid * E1);
    __syncthreads();
    for (int it = tid; it < 3 * (la + 1) * (lb + 1) * 4; it += HT_THREADS) {
      const int ty = it % 4, j = (it / 4) % (lb + 1), i = (it / 4 / (lb + 1)) % (la + 1),
                x = it / 4 / (lb + 1) / (la + 1);
      double* f = fa + (size_t)it * FL;
      const int n = axis_factor<double>(E + x * E1, lb + 1, la + lb + 3, i, j, ty, 2.0 * ea,
                                        2.0 * eb, f);
      for (int t = n; t < FL; t++) f[t] = 0.0;
    }
    __syncthreads();
    const int nb = ncart(lb), nab = ncart(la) * nb, nop = hg_ops(kind);
    const int H = nherm(la + lb + hg_rise(kind)), kt = hg_ktiles(kind, la, lb);
    const int size = hg_size(kind, la, lb);
    double* out = tab + (size_t)(P.pp_off + ip - ppBeg) * size;
    for (int e = tid; e < size; e += HT_THREADS) {
      // [row tile][order tile][lane][half]
      const int half = e & 1, lane = (e >> 1) & 31, k = (e >> 6) % kt, rt = (e >> 6) / kt;
      const int row = rt * 16 + half * 8 + (lane >> 2), h = k * 4 + (lane & 3);
      double v = 0.0;
      if (row < nab * nop && h < H) {
        const int ab = row / nop, op = row % nop, a = ab / nb, b = ab % nb;
        int n = 0;
        while (nherm(n) <= h) n++;
        const int r = h - nherm(n - 1);
        int kk = 0;
        while ((kk + 1) * (kk + 2) / 2 <= r) kk++;
        const int hv = r - kk * (kk + 1) / 2, hu = kk - hv, ht = n - kk;
        const int ax[3] = {cart_lx(la, a), cart_ly(la, a), cart_lz(la, a)};
        const int bx[3] = {cart_lx(lb, b), cart_ly(lb, b), cart_lz(lb, b)};
        auto f = [&](int x, int ty, int t) {
          return t < FL ? fa[(size_t)(((x * (la + 1) + ax[x]) * (lb + 1) + bx[x]) * 4 + ty) * FL + t]
                        : 0.0;
        };
        if (kind == HG_SPIN) {
          for (int mu = 0; mu < 3; mu++)
            for (int nu = 0; nu < 3; nu++) {
              int o2;
              double sg;
              op_of(mu, nu, o2, sg);
              if (o2 != op) continue;
              v += sg * f(0, (mu == 0) | ((nu == 0) << 1), ht) *
                   f(1, (mu == 1) | ((nu == 1) << 1), hu) * f(2, (mu == 2) | ((nu == 2) << 1), hv);
            }
        } else {
          const int dir = kind == HG_PLAIN ? -1 : op % 3, ty = op < 3 ? 1 : 2;
          v = f(0, dir == 0 ? ty : 0, ht) * f(1, dir == 1 ? ty : 0, hu) *
              f(2, dir == 2 ? ty : 0, hv);
        }
      }
      out[e] = v;
    }
    __syncthreads();  // before the next one's factors
  }
}

// The pairs with npp cut to the primitive pairs that can contribute: they are
// sorted by their Schwarz bound, and one below 1e-34 (a tight primitive on
// another centre, exp(-mu R^2) = 0) stays below rounding against any partner
// and through four derivatives.
__global__ void hg_pairs_kernel(const PairDev* __restrict__ in, const double* __restrict__ ppQ,
                                int n, PairDev* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  PairDev P = in[i];
  while (P.npp > 1 && ppQ[P.pp_off + P.npp - 1] < 1e-34) P.npp--;
  out[i] = P;
}

// Window of a table that is not held: doubles for one side of a launch.
// 64 MiB hold some 110 primitive pairs of two f functions with all six
// derivatives, so that a window's building stays small beside its quartets.
constexpr size_t HG_WINDOW = size_t(8) << 20;

}  // namespace

cqf_status hg_ensure(cqf_basis* B, int kind) {
  auto status = [](cudaError_t e) {
    if (e == cudaSuccess) return CQF_OK;
    return fail(e == cudaErrorMemoryAllocation ? CQF_ENOMEM : CQF_ECUDA,
                std::string("hg_ensure: ") + cudaGetErrorString(e));
  };
  // build_once with memory of the basis' stream; fill enqueues
  auto build = [&](auto*& slot, size_t n, auto fill) {
    return status(build_once(
        slot, cudaSuccess,
        [&](auto** p) { return cudaMallocAsync((void**)p, std::max<size_t>(1, n) * sizeof(**p), B->stream); },
        [&](auto* p) {
          fill(p);
          const cudaError_t e = cudaGetLastError();
          return e != cudaSuccess ? e : cudaStreamSynchronize(B->stream);
        },
        [&](auto* p) { cudaFreeAsync(p, B->stream); }));
  };
  const cqf_status s = build(B->d_pairsHg, B->npair, [&](PairDev* p) {
    hg_pairs_kernel<<<std::max(1, (B->npair + 127) / 128), 128, 0, B->stream>>>(
        B->d_pairs, B->d_ppQ, B->npair, p);
  });
  if (s != CQF_OK || B->d_hg[kind]) return s;
  if (B->hg_win[kind]) return CQF_OK;
  size_t total = 0, pair = 0;  // doubles of the table, and of the largest pair in it
  for (int c = 0; c < NCLS; c++) {
    B->hg_beg[kind][c] = total;
    if (!B->cls_cnt[c]) continue;
    int la, lb;
    class_ls(c, la, lb);
    total += (size_t)B->cls_npp_sum[c] * hg_size(kind, la, lb);
    pair = std::max(pair, (size_t)B->cls_npp_max[c] * hg_size(kind, la, lb));
  }
  if (B->hg_bytes + total * sizeof(double) <= B->hg_limit) {
    const cqf_status t = build(B->d_hg[kind], total, [&](double* d) {
      for (int c = 0; c < NCLS; c++)
        if (B->cls_cnt[c])
          hg_fill(B, kind, c, B->cls_beg[c], B->cls_cnt[c], d + B->hg_beg[kind][c], B->stream);
    });
    if (t == CQF_OK) B->hg_bytes += total * sizeof(double);
    if (t != CQF_ENOMEM) return t;
    cudaGetLastError();
    fail(CQF_OK, "");
  }
  // (a table's tiles are 64 doubles; a small limit means small windows)
  B->hg_win[kind] = std::max(pair, std::min(HG_WINDOW, B->hg_limit / 4096 * 64));
  return CQF_OK;
}

void hg_fill(const cqf_basis* B, int kind, int c, int beg, int n, double* tab, cudaStream_t st) {
  int la, lb;
  class_ls(c, la, lb);
  const size_t smem =
      (3 * ht_e1(la, lb) + (size_t)12 * (la + 1) * (lb + 1) * ht_fl(la, lb)) * sizeof(double);
  hg_table_kernel<<<dim3(n, std::min(B->cls_npp_max[c], PRIM_ROWS)), HT_THREADS, smem, st>>>(
      B->d_pairs, B->d_pp, B->d_shells, B->d_prim, beg, B->h_pairs[beg].pp_off, kind, la, lb, tab);
}

}  // namespace cqf
