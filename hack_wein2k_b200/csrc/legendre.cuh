// legendre.cuh -- explicit polynomials of (2l+1) P_l(x), l < SPH_LMAX.
//
// P_l is x^(l odd) times a polynomial of degree l/2 in x^2.  It is summed in
// y = x^2 - 1/2, |y| <= 1/2: the coefficients, multiples of powers of two, are
// exact in FP64, and at l = 12 the terms sum to at most 903 in magnitude (343 at
// l = 10) where in powers of x^2 they reach 1.5e5 (2.3e4).  Largest error over
// [-1, 1], absolute: 5.6e-14 at l = 12 and 3.0e-14 at l = 10; the three-term
// recursion of hamilt.F:250-281 5.8e-14 and 3.7e-14; in powers of x^2 3.8e-12 and
// 6.7e-13.  Both bases take one operation for their argument (x^2, or x^2 - 1/2 as
// one FMA) and l/2 FMAs.
#pragma once
#include <cmath>

struct LegCoef {
  double c[SPH_LMAX][(SPH_LMAX + 1) / 2];  // by descending power of y
};
__host__ __device__ constexpr LegCoef leg_make() {
  LegCoef t{};
  for (int l = 0; l < SPH_LMAX; l++) {
    const int d = l / 2;
    // (2l+1) P_l = x^(l odd) sum_m a_m (x^2)^m, with k = d - m:
    // P_l = 2^-l sum_k (-1)^k C(l,k) C(2l-2k,l) x^(l-2k)
    double a[(SPH_LMAX + 1) / 2] = {};
    for (int k = 0; k <= d; k++) {
      double v = 1.0;
      for (int i = 1; i <= k; i++) v = v * (l - k + i) / i;      // C(l,k)
      double w = 1.0;
      for (int i = 1; i <= l; i++) w = w * (l - 2 * k + i) / i;  // C(2l-2k,l)
      double q = (k & 1) ? -v * w : v * w;
      for (int i = 0; i < l; i++) q *= 0.5;
      a[d - k] = q * (2 * l + 1);
    }
    // (y + 1/2)^m = sum_j C(m,j) 2^-(m-j) y^j
    for (int j = 0; j <= d; j++) {
      double s = 0.0;
      for (int m = j; m <= d; m++) {
        double q = a[m];
        for (int i = 1; i <= j; i++) q = q * (m - j + i) / i;  // C(m,j)
        for (int i = 0; i < m - j; i++) q *= 0.5;
        s += q;
      }
      t.c[l][d - j] = s;
    }
  }
  return t;
}
template <int l, int N>
__host__ __device__ __forceinline__ void leg_poly(const double (&x)[N], double (&w)[N]) {
  constexpr LegCoef K = leg_make();
#pragma unroll
  for (int u = 0; u < N; u++) {
    const double y = fma(x[u], x[u], -0.5);
    double p = K.c[l][0];
#pragma unroll
    for (int k = 1; k <= l / 2; k++) p = fma(p, y, K.c[l][k]);
    w[u] = (l & 1) ? p * x[u] : p;
  }
}
