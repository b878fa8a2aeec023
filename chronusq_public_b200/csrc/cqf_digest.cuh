// The reference's four digestion branches for one integral (HER / non-HER x
// COULOMB / EXCHANGE), real and complex matrices.
#pragma once

#include <cuda_runtime.h>

namespace cqf {

template <bool CPLX>
struct Mat;

template <>
struct Mat<false> {
  static __device__ __forceinline__ double ld(const double* X, size_t i) { return __ldg(X + i); }
  static __device__ __forceinline__ double ldc(const double* X, size_t i) { return __ldg(X + i); }
  static __device__ __forceinline__ double ldre(const double* X, size_t i) { return __ldg(X + i); }
  static __device__ __forceinline__ void add(double* A, size_t i, double v, double w) {
    atomicAdd(A + i, v * w);
  }
  static __device__ __forceinline__ void addre(double* A, size_t i, double v) {
    atomicAdd(A + i, v);
  }
};

template <>
struct Mat<true> {
  static __device__ __forceinline__ double2 ld(const double* X, size_t i) {
    return __ldg(reinterpret_cast<const double2*>(X) + i);
  }
  static __device__ __forceinline__ double2 ldc(const double* X, size_t i) {
    double2 z = __ldg(reinterpret_cast<const double2*>(X) + i);
    z.y = -z.y;
    return z;
  }
  static __device__ __forceinline__ double ldre(const double* X, size_t i) {
    return __ldg(X + 2 * i);
  }
  static __device__ __forceinline__ void add(double* A, size_t i, double2 v, double w) {
    atomicAdd(A + 2 * i, v.x * w);
    atomicAdd(A + 2 * i + 1, v.y * w);
  }
  static __device__ __forceinline__ void addre(double* A, size_t i, double v) {
    atomicAdd(A + 2 * i, v);
  }
};

__device__ __forceinline__ double2 operator+(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}

// Digest one integral v (already x 0.5 deg) with role indices i1..i4 into
// matrix m (direct.hpp:1858-2002).
template <bool CPLX>
__device__ __forceinline__ void digest_one(int flags, const double* __restrict__ X, double* A,
                                           size_t nc, int i1, int i2, int i3, int i4, double v) {
  using M = Mat<CPLX>;
  const bool her = flags & 1, exch = flags & 2;
  auto ix = [nc](int r, int c) -> size_t { return (size_t)r + (size_t)c * nc; };
  if (her) {
    if (!exch) {
      // J(1,2) += X(4,3) I ; J(4,3) += X(1,2) I   (real parts)
      M::addre(A, ix(i1, i2), M::ldre(X, ix(i4, i3)) * v);
      M::addre(A, ix(i4, i3), M::ldre(X, ix(i1, i2)) * v);
    } else {
      // (bit 2, the antisymmetric part of a split complex Hermitian density,
      // needs nothing here: these four updates read X in the orientation
      // the antisymmetric back transform expects, as the class kernels' do)
      const double h = 0.5 * v;
      M::add(A, ix(i1, i3), M::ldc(X, ix(i4, i2)), h);
      M::add(A, ix(i4, i2), M::ldc(X, ix(i1, i3)), h);
      M::add(A, ix(i4, i1), M::ldc(X, ix(i2, i3)), h);
      M::add(A, ix(i2, i3), M::ldc(X, ix(i4, i1)), h);
    }
  } else {
    const double h = 0.5 * v;
    if (!exch) {
      auto x34 = M::ld(X, ix(i4, i3)) + M::ld(X, ix(i3, i4));
      auto x12 = M::ld(X, ix(i2, i1)) + M::ld(X, ix(i1, i2));
      M::add(A, ix(i1, i2), x34, h);
      M::add(A, ix(i3, i4), x12, h);
      M::add(A, ix(i2, i1), x34, h);
      M::add(A, ix(i4, i3), x12, h);
    } else {
      M::add(A, ix(i3, i1), M::ld(X, ix(i4, i2)), h);
      M::add(A, ix(i4, i2), M::ld(X, ix(i3, i1)), h);
      M::add(A, ix(i4, i1), M::ld(X, ix(i3, i2)), h);
      M::add(A, ix(i3, i2), M::ld(X, ix(i4, i1)), h);
      M::add(A, ix(i1, i3), M::ld(X, ix(i2, i4)), h);
      M::add(A, ix(i2, i4), M::ld(X, ix(i1, i3)), h);
      M::add(A, ix(i1, i4), M::ld(X, ix(i2, i3)), h);
      M::add(A, ix(i2, i3), M::ld(X, ix(i1, i4)), h);
    }
  }
}

}  // namespace cqf
