"""The FP64 likelihood's own elementary functions (csrc/qcbc_math.cuh), built for the host, against long double over
the ranges that the kernels call them on.

Bounds: recip_newton's last step rounds once and its argument's residual is exact but for one rounding, so one unit
in the last place; the sine and cosine polynomials are within 2^-54 of their functions and Horner's last two
roundings act on at most one, so 1.5 2^-52 absolute near one quadrant's ends plus the argument's reduction, which is
exact; the arctangent's last multiply-add and product round once each, two units."""
import ctypes as C

import numpy as np

from hostcc import compile_host

CODE = r"""
#include "qcbc_math.cuh"
extern "C" void recip(const double* x, const double* r, double* y, int n) {
  for (int k = 0; k < n; k++) y[k] = qcbc::recip_newton(x[k], r[k]);
}
extern "C" void sc(const double* x, double* s, double* c, int n, int any) {
  for (int k = 0; k < n; k++) {
    const double a[1] = {x[k]};
    double u[1], v[1];
    if (any) qcbc::sincos_cycles<1, true>(a, u, v);
    else qcbc::sincos_cycles<1, false>(a, u, v);
    s[k] = u[0];
    c[k] = v[0];
  }
}
extern "C" void at(const double* w, double* y, int n) {
  for (int k = 0; k < n; k++) {
    const double a[1] = {w[k] * w[k]};
    double p[1];
    qcbc::atan_ratio<1>(a, p);
    y[k] = w[k] * p[0];
  }
}
"""
LD = np.longdouble


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _ulps(got, want):
    return np.max(np.abs((got.astype(LD) - want) / np.spacing(np.abs(want).astype(float)).astype(LD)))


def test_reciprocal(tmp_path):
    L = compile_host(str(tmp_path), CODE)
    rng = np.random.default_rng(1)
    n = 200000
    # the Lorentzian times 1 + z z_c: from (fDM g3)^2 at fDM = 60 Msec df of a neutron star up to a few thousand, and
    # far beyond on either side; the starting value off by up to 2^-18
    for lo, hi in ((-45, 12), (-300, 300)):
        x = rng.uniform(1, 2, n) * 2.0 ** rng.integers(lo, hi, n)
        r = (1 / x) * (1 + rng.choice([-1.0, 1.0], n) * 2.0 ** rng.uniform(-40, -18, n))
        y = np.empty(n)
        L.recip(_p(x), _p(r), _p(y), n)
        assert _ulps(y, 1 / x.astype(LD)) <= 1.0


def test_sine_and_cosine_of_cycles(tmp_path):
    L = compile_host(str(tmp_path), CODE)
    rng = np.random.default_rng(2)
    pi2 = LD("6.283185307179586476925286766559005768")
    eighths = np.concatenate([np.arange(-64, 65) / 8.0 + d for d in (0.0, 1e-16, -1e-16, 1e-9, -1e-9)])
    for any_, scale in ((0, 1.0), (0, 1e6), (0, 2.0 ** 44), (1, 1.0), (1, 1e18)):
        x = np.concatenate([eighths, rng.uniform(-1, 1, 100000) * scale, rng.uniform(-1, 1, 1000) * 1e-9])
        s, c = np.empty(len(x)), np.empty(len(x))
        L.sc(_p(x), _p(s), _p(c), len(x), any_)
        frac = (x - np.rint(x)).astype(LD)                     # exact
        assert np.max(np.abs(s - np.sin(pi2 * frac))) <= 1.5 * 2.0 ** -52
        assert np.max(np.abs(c - np.cos(pi2 * frac))) <= 1.5 * 2.0 ** -52
    bad = np.array([np.inf, -np.inf, np.nan])
    s, c = np.empty(3), np.empty(3)
    L.sc(_p(bad), _p(s), _p(c), 3, 1)
    assert np.all(np.isnan(s)) and np.all(np.isnan(c))


def test_arctangent(tmp_path):
    L = compile_host(str(tmp_path), CODE)
    rng = np.random.default_rng(3)
    w = np.concatenate([rng.uniform(-0.2645, 0.2645, 200000), [0.2645, -0.2645], 10.0 ** rng.uniform(-12, -1, 1000)])
    y = np.empty(len(w))
    L.at(_p(w), _p(y), len(w))
    assert _ulps(y, np.arctan(w.astype(LD))) <= 2.0
