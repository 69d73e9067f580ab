// kf_solve6.cuh — FP64 solve of the ICP's 6x6 normal equations.  Host code can include it as
// well: the tests compare it with exact arithmetic there and on the device.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define KF_SOLVE_FN __host__ __device__ __forceinline__
#define KF_SOLVE_UNROLL _Pragma("unroll")
#else
#define KF_SOLVE_FN inline
#define KF_SOLVE_UNROLL
#endif

// 1 / d of a normal d to FP64 precision without a divide: an estimate whose error e is at most
// 2^-20 (the host's form: the quotient cut to 20 bits), then y (1 + e + e^2), which leaves e^3.
KF_SOLVE_FN double kf_reciprocal(double d) {
  double y;
#ifdef __CUDA_ARCH__
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
#else
  y = 1.0 / d;
  uint64_t bits;
  std::memcpy(&bits, &y, 8);
  bits &= ~0xffffffffull;
  std::memcpy(&y, &bits, 8);
#endif
  const double e = std::fma(-d, y, 1.0);
  return std::fma(std::fma(e, e, e), y, y);
}

// C x = b by Cholesky's factorisation without square roots (C = L D L^T); C as the 21
// upper-triangular values of reduce.cs rows 7..27 (row-major).  For a C that passed the rank
// check (its pivots are positive; the result for another C is not used).  By one thread, all in
// registers.  What bounds it is the chain of six pivots, each a reciprocal and a multiply-add, and
// the substitution behind them.  Relative error against exact arithmetic, median / worst, over
// 270,000 systems with tilted normals that pass the check, by trace(C) trace(C^-1): below 250
// 2.5e-16 / 6.3e-15, to 1,600 8.5e-16 / 6.3e-14, to 10,000 4.4e-15 / 4.2e-13, to 50,000 2.2e-14 /
// 1.5e-12; Cholesky with reciprocal square roots 3.9e-16 / 9.5e-15 .. 3.8e-14 / 3.4e-12.  3x3 blocks
// inverted by their cofactors lose the square of the condition (2.1e-13 / 1.9e-8 in the last
// range) and are no faster: 512^3 frame 281 us against 279, 128^3 177 against 177; those blocks
// with a step of refinement 284 and 178, reciprocals from an FP32 estimate 288 and 184.
KF_SOLVE_FN void kf_solve6(const double* c21, const double* b, double* x) {
  double l[6][6], u[6][6], inv[6], y[6];  // u[i][j] = l[i][j] d[j]
  KF_SOLVE_UNROLL
  for (int j = 0; j < 6; ++j) {
    const double* row = c21 + 6 * j - j * (j - 1) / 2;
    double d = row[0];
    KF_SOLVE_UNROLL
    for (int k = 0; k < j; ++k) d = std::fma(-l[j][k], u[j][k], d);
    inv[j] = kf_reciprocal(d);
    KF_SOLVE_UNROLL
    for (int i = j + 1; i < 6; ++i) {
      double v = row[i - j];
      KF_SOLVE_UNROLL
      for (int k = 0; k < j; ++k) v = std::fma(-l[i][k], u[j][k], v);
      u[i][j] = v;
      l[i][j] = v * inv[j];
    }
  }
  KF_SOLVE_UNROLL
  for (int i = 0; i < 6; ++i) {
    y[i] = b[i];
    KF_SOLVE_UNROLL
    for (int k = 0; k < i; ++k) y[i] = std::fma(-l[i][k], y[k], y[i]);
  }
  KF_SOLVE_UNROLL
  for (int i = 5; i >= 0; --i) {
    double v = y[i] * inv[i];
    KF_SOLVE_UNROLL
    for (int k = i + 1; k < 6; ++k) v = std::fma(-l[k][i], x[k], v);
    x[i] = v;
  }
}
