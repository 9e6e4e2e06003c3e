// Elementary functions of the FP64 likelihood kernels: polynomials and iterations that need no division, for
// several arguments side by side (U), so that a constant is read once for all of them.  Only IEEE operations, so a
// host build gives the same bits (tests/test_device_math.py checks them there against a wider type).
#pragma once
#include <cuda_runtime.h>

namespace qcbc {

// 1/x from an approximation r of it, by two steps of Newton's iteration r <- r + r (1 - x r) (Newton-Raphson
// division; J.-M. Muller et al., Handbook of Floating-Point Arithmetic, ch. 4): a relative error of 2^-18 goes to
// 2^-36 and then to the last step's rounding, one unit in the last place.  x and 1/x finite and normal.
__device__ __forceinline__ double recip_newton(double x, double r) {
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

// sin and cos of 2 pi t, |t| <= 1/8, and atan(w)/w, |w| <= 0.2645: polynomials in t^2 and w^2,
// interpolated at Chebyshev nodes in 60-digit arithmetic and rounded; relative errors 3.9e-17, 2.1e-17
// and 2.5e-17.
static __constant__ double c_sin2pi[7] = {6.283185307179586, -41.341702240399634, 81.60524927594804, -76.70585970427454,
                                   42.058685020160894, -15.093804209987114, 3.7808689593022957};
static __constant__ double c_cos2pi[8] = {1.0, -19.739208802178716, 64.93939402266795, -85.45681720652271,
                                   60.244641328867296, -26.426250908622137, 7.903091687751697, -1.6968494702918826};
static __constant__ double c_atan64[9] = {1.0, -0.33333333333330495, 0.19999999998915635, -0.14285714126071508,
                                   0.11111099310073162, -0.09090417358899357, 0.07680201267088747,
                                   -0.06490960023860128, 0.04468242583532965};
constexpr double kAtanRange = 0.2645;

// sin and cos of 2 pi cyc of U values.  Any: cyc may be beyond 2^45, infinite or NaN (the tile's bound on
// its phase, Tile64, keeps the others below).
template <int U, bool Any>
__device__ __forceinline__ void sincos_cycles(const double (&cyc)[U], double (&sv)[U], double (&cv)[U]) {
  constexpr double kMagic = 6755399441055744.0;         // 1.5 2^52: the add rounds to an integer
  int k[U];                                             // quadrant
  double t[U], z[U], s[U], c[U];
#pragma unroll
  for (int j = 0; j < U; j++) {
    double x = cyc[j];
    if (Any && (__double2hiint(x) & 0x7fffffff) > 0x42c00000) x -= rint(x);
    const double q = fma(x, 4.0, kMagic);
    k[j] = __double2loint(q);
    t[j] = fma(q - kMagic, -0.25, x);
    z[j] = t[j] * t[j];
    s[j] = c_sin2pi[6];
    c[j] = c_cos2pi[7];
  }
#pragma unroll
  for (int m = 6; m >= 0; m--) {
    const double b = c_cos2pi[m];
#pragma unroll
    for (int j = 0; j < U; j++) c[j] = fma(z[j], c[j], b);
    if (m < 6) {
      const double a = c_sin2pi[m];
#pragma unroll
      for (int j = 0; j < U; j++) s[j] = fma(z[j], s[j], a);
    }
  }
#pragma unroll
  for (int j = 0; j < U; j++) {
    const double st = s[j] * t[j];
    const double a = (k[j] & 1) ? c[j] : st, d = (k[j] & 1) ? st : c[j];
    sv[j] = __hiloint2double(__double2hiint(a) ^ ((k[j] & 2) << 30), __double2loint(a));
    cv[j] = __hiloint2double(__double2hiint(d) ^ (((k[j] + 1) & 2) << 30), __double2loint(d));
  }
}
__device__ __forceinline__ void sincos_cycles(double cyc, double& sv, double& cv) {
  const double x[1] = {cyc};
  double s[1], c[1];
  sincos_cycles<1, true>(x, s, c);
  sv = s[0];
  cv = c[0];
}

// atan(w)/w from w^2
template <int U>
__device__ __forceinline__ void atan_ratio(const double (&w2)[U], double (&p)[U]) {
#pragma unroll
  for (int j = 0; j < U; j++) p[j] = c_atan64[8];
#pragma unroll
  for (int k = 7; k >= 0; k--) {
    const double a = c_atan64[k];
#pragma unroll
    for (int j = 0; j < U; j++) p[j] = fma(w2[j], p[j], a);
  }
}

}  // namespace qcbc
