"""The FP64 likelihood's own elementary functions (csrc/qcbc_math.cuh), built for the host, against long double over
the ranges that the kernels call them on.

Bounds: recip_newton's last step rounds once and its argument's residual is exact but for one rounding, so one unit
in the last place; the sine and cosine polynomials are within 2^-54 of their functions and Horner's last two
roundings act on at most one, so 1.5 2^-52 absolute near one quadrant's ends plus the argument's reduction, which is
exact; the arctangent's last multiply-add and product round once each, two units."""
import ctypes as C
from fractions import Fraction

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


PHASE = r"""
#include "qcbc_device.cuh"
extern "C" void lin(double df, double t, double slope, const double* n, double* y, int k) {
  const qcbc::LinPhase p(df, t, slope);
  for (int j = 0; j < k; j++) y[j] = p.cycles(n[j]);
}
extern "C" void fold(const double* q, const double* ql, const double* f, const double* t, double* y, int n) {
  for (int k = 0; k < n; k++) {
    const double r = 1.0 / t[k];
    double lo;
    const double hi = qcbc::fold_r5(q[k], ql[k], r, qcbc::rthird_eps(f[k], 1.0 / f[k], t[k], r), lo);
    y[2 * k] = hi;
    y[2 * k + 1] = lo;
  }
}
"""


def test_linear_phase_is_reduced_exactly(tmp_path):
    """Against exact fractions: the slope's last part, n lo and the sum are rounded, 2^-52 of a cycle together."""
    L = compile_host(str(tmp_path), PHASE)
    n = np.concatenate([[0, 1, (1 << 20) - 1], np.random.default_rng(4).integers(0, 1 << 20, 500)]).astype(float)
    for df, t, slope in ((1 / 128.0, 126.3, 1.7e-5), (1 / 7.3, 5.1, 2e-3), (0.25, 2.0, -0.4), (1 / 64.0, 61.99, 0.0)):
        y = np.empty(len(n))
        L.lin(C.c_double(df), C.c_double(t), C.c_double(slope), _p(n), _p(y), len(n))
        step = Fraction(df) * Fraction(t) - Fraction(slope)
        for k, got in zip(n, y):
            d = Fraction(got) - int(k) * step
            assert abs(d - round(d)) <= Fraction(1, 2 ** 52)


def test_newtonian_coefficient(tmp_path):
    """q f^{-5/3} / 2 pi from a cube root that is a unit in the last place off: to 2^-63 as hi + lo."""
    L = compile_host(str(tmp_path), PHASE)
    rng = np.random.default_rng(5)
    n = 20000
    f, q = 10.0 ** rng.uniform(-8, -1, n), rng.uniform(0.01, 5.0, n)
    ql = q * rng.uniform(-1, 1, n) * 2.0 ** -53
    t = np.cbrt(f) * (1 + rng.integers(-1, 2, n) * 2.0 ** -52)
    y = np.empty(2 * n)
    L.fold(_p(q), _p(ql), _p(f), _p(t), _p(y), n)
    got = y[0::2].astype(LD) + y[1::2].astype(LD)
    want = (q.astype(LD) + ql) * f.astype(LD) ** (LD(-5) / LD(3)) / LD("6.283185307179586476925286766559005768")
    assert np.max(np.abs(got / want - 1)) <= 2.0 ** -60       # long double's own power has a few bits of its 64
    assert np.max(np.abs(y[0::2] / want.astype(float) - 1)) > 2.0 ** -52        # the one-term product is not enough
