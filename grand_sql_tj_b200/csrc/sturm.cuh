// Sturm counts of a symmetric tridiagonal matrix, shared by the truncation's
// eigenvalues and the Ritz value of the Lanczos iteration.
#pragma once
#include <cuda_runtime.h>

namespace tjb {

// The power of two that scales T's largest row sum tnorm into [1/2, 1); 1 where
// T is zero (or out of range).
__device__ __forceinline__ double tridiag_scale(double tnorm) {
  const int te = __double2hiint(tnorm) >> 20 & 2047;
  return te > 0 && te < 2045 ? __hiloint2double((2045 - te) << 20, 0) : 1.0;
}

// Number of eigenvalues of the scaled T (diagonal ds, squared off-diagonal e2)
// below x: the sign changes along the leading principal minors of T - x I,
// p_{i+1} = (d_i - x) p_i - e_{i-1}^2 p_{i-1}.  The pivots of LDL^T, the ratios
// of consecutive minors, would cost a division a step; the minors take three
// operations and a rescaling by a power of two every eight steps.  A zero
// minor between others needs no care (its neighbours have opposite signs, so
// either sign of it makes one change); only where eight steps shrink the
// minors below 2^-500 (a zero pivot at a zero off-diagonal, or entries far
// under the accuracy asked for) are they repeated with every pivot below 2^-60
// taken as -2^-60, as LAPACK's dstebz does with its pivmin.
__device__ __forceinline__ int sturm1(const double *__restrict__ ds, const double *__restrict__ e2, int n, double x) {
  double p0 = 1.0, p1 = ds[0] - x;
  if (fabs(p1) < 0x1p-60) p1 = -0x1p-60;
  int c = __double2hiint(p1) >> 31;   // minus the count
  auto step = [&](double di, double ei, bool careful) {
    double p = fma(di - x, p1, -(ei * p0));
    // |p| < 2^-60 |p1| by the exponents
    if (careful && (__double2hiint(p) & 0x7ff00000) + (60 << 20) < (__double2hiint(p1) & 0x7ff00000)) p = -0x1p-60 * p1;
    c += (__double2hiint(p) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p;
  };
  // the larger exponent of the two last minors
  auto expo = [&]() { return max(__double2hiint(p0) >> 20 & 2047, __double2hiint(p1) >> 20 & 2047); };
  int i = 1;
  for (; i + 8 <= n; i += 8) {
    double dv[8], ev[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      dv[u] = ds[i + u];
      ev[u] = e2[i + u - 1];
    }
    const double b0 = p0, b1 = p1;
    const int bc = c;
#pragma unroll
    for (int u = 0; u < 8; ++u) step(dv[u], ev[u], false);
    if (expo() < 1023 - 500) {
      p0 = b0;
      p1 = b1;
      c = bc;
#pragma unroll 1
      for (int u = 0; u < 8; ++u) step(ds[i + u], e2[i + u - 1], true);
    }
    // the larger of the two to about one
    const double f = __hiloint2double(min(max(2046 - expo(), 1), 2045) << 20, 0);
    p0 *= f;
    p1 *= f;
  }
#pragma unroll 1
  for (; i < n; ++i) step(ds[i], e2[i - 1], true);
  return -c;
}

}  // namespace tjb
