"""The heterodyne grid search on the device against a serial restatement on the CPU oracle's waveforms:
band limits, Fisher matrix, efix, grid walk and flattening (QuickCBC.c:4275-4910, 2449-2530, 2695-2817), one to
three detectors and 4 to 16 s, so that the walk's windows, ratio pieces and block sums end at different places.
The grids are whole numbers and are equal: FP64 rounding (1e-12 in a ratio) moves a grid point only if the
interpolation error of a bin meets the tolerance to that precision."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template, prior_bounds
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu
TPI, PI = 6.2831853071795862319959269370884, 3.1415926535897931159979634685442


def fqnm(p):
    Mc, M = (np.exp(p[k]) / synth.MSUN_SI * 4.92569043916e-6 for k in (0, 1))
    eta = min((Mc / M) ** (5.0 / 3.0), 0.25)
    dm = np.sqrt(1 - 4 * eta)
    m1, m2, c1, c2 = M * (1 + dm) / 2, M * (1 - dm) / 2, p[2], p[3]
    r = m1 / m2 if m1 < m2 else m2 / m1
    eta = r / (1 + r) ** 2
    atot = (c1 + r * r * c2) / (1 + r) ** 2
    ae = atot + 0.41616 * eta * (c1 + c2)
    Z1 = 1 + (1 - ae * ae) ** (1 / 3.) * ((1 + ae) ** (1 / 3.) + (1 - ae) ** (1 / 3.))
    Z2 = np.sqrt(3 * ae * ae + Z1 * Z1)
    ri = 3 + Z2 - ae / (abs(ae) + 1e-20) * np.sqrt((3 - Z1) * (3 + Z1 + 2 * Z2))
    E, L = np.sqrt(1 - 2 / (3 * ri)), 2 / (3 * np.sqrt(3)) * (1 + 2 * np.sqrt(3 * ri - 2))
    Mf = (1 - eta * (1 - E) - 4 * eta * eta * (4 * 0.04827 + 16 * 0.01707 * atot * (atot + 1) + E - 1)) * (m1 + m2)
    af = (atot + eta * (L - 2 * atot * (E - 1)) - 3.82 * eta ** 2 - 1.2019 * eta ** 2 * ae - 1.20764 * eta ** 2 * ae ** 2 +
          3.79245 * eta ** 3 + 1.18385 * eta ** 3 * ae + 4.90494 * eta ** 3 * ae ** 2)
    return (1.5251 - 1.1568 * (1 - af) ** 0.1292) / (TPI * Mf)


def jacobi(F):
    """Cyclic Jacobi rotations (Golub & Van Loan 8.5): with one detector the matrix is singular, and the basis of
    its null space is the one this sequence of rotations leaves."""
    A, V = F.copy(), np.eye(11)
    for _ in range(100):
        off = np.sum(A * A) - np.sum(np.diag(A) ** 2)
        if off <= 1e-30 * np.sum(A * A):
            break
        for a in range(10):
            for b in range(a + 1, 11):
                if A[a, b] == 0.0:
                    continue
                th = (A[b, b] - A[a, a]) / (2 * A[a, b])
                t = (1.0 if th >= 0 else -1.0) / (abs(th) + np.sqrt(th * th + 1))
                c = 1 / np.sqrt(t * t + 1)
                G = np.array([[c, t * c], [-t * c, c]])
                A[:, [a, b]] = A[:, [a, b]] @ G
                A[[a, b]] = G.T @ A[[a, b]]
                V[:, [a, b]] = V[:, [a, b]] @ G
    return np.diag(A).copy(), V


def step(p, a, e, lo, hi):
    x = p + a * e
    if np.exp(5 / 3. * (x[0] - x[1])) > 0.25:
        x = p - a * e
    for k, T in ((4, TPI), (7, TPI), (9, PI)):
        y = x[k] / T
        x[k] = (y - np.floor(y)) * T + (1.0 if y < 0 else 0.0)
        while x[k] > T:
            x[k] -= T
        while x[k] < 0:
            x[k] += T
    x = np.maximum(np.minimum(x, hi), lo)
    eta = np.exp(5 / 3. * (x[0] - x[1]))
    if eta > 0.25:
        x[0] = x[1] + 0.6 * np.log(0.2499)
    if eta < 0.05:
        x[0] = x[1] + 0.6 * np.log(0.05)
    return x


def serial_het_space(ora, ev, p, lo, hi):
    nh, T, S = ev.N // 2, ev.Tobs, ev.SN
    wave = lambda x: ora.fullphaseamp(ev.labels, ev.GMST, T, ev.freq, x, ev.N)     # noqa: E731
    Ar, Pr = wave(p)
    M = min(int(max(2 * fqnm(p), 64.0) * T), nh)
    fs = ora.fbegin(p)
    jmin = int(T * ev.fmin) if ev.fmin > fs else int(T * fs)
    d = np.zeros(M)
    d[jmin:] = (4 * Ar[:, jmin:M] ** 2 / S[:, jmin:M]).sum(0)
    acc = np.cumsum(d)
    MN = jmin + int(np.argmax(acc[jmin:] > 0.001))
    MM = jmin + int(np.argmax(acc[-1] - acc[jmin:] < 0.001))
    x = acc[-1] / (MM - MN)
    ratio = np.where(d > 0, 1.0 / np.where(d > 0, d / x, 1.0), 1.0)
    k = np.arange(int(T * ev.fmin), min(int(T * 1024), nh))
    dA, dP = [], []
    for i in range(11):
        u, v = p.copy(), p.copy()
        u[i] += 1e-5
        v[i] -= 1e-5
        (Au, Pu), (Av, Pv) = wave(u), wave(v)
        dA.append((Au - Av)[:, k] / 2e-5)
        dP.append((Pu - Pv)[:, k] / 2e-5)
    F = np.array([[np.sum(4 * (dA[i] * dA[j] + Ar[:, k] ** 2 * dP[i] * dP[j]) / S[:, k]) for j in range(11)]
                  for i in range(11)])
    val, V = jacobi(F)
    order = np.argsort(np.abs(val), kind="stable")
    ev_, ej = V.T[order], 1 / np.sqrt(np.maximum(val[order], 10.0))

    def dist(y):
        A, P = wave(y)
        s = slice(jmin, M)
        c = Ar[:, s] - A[:, s] * np.cos(Pr[:, s] - P[:, s])
        return np.sum(4 * (c ** 2 + (A[:, s] * np.sin(Pr[:, s] - P[:, s])) ** 2) / S[:, s])
    zs, rows = 30.0, []
    for i in range(11):
        e, dz_min, am, a0, n = ej[i] * ev_[i], 1e20, 1.0, 1.0, 0
        while True:
            z0 = dist(step(p, a0, e, lo, hi))
            if abs(z0 - zs) < dz_min:
                dz_min, am = abs(z0 - zs), a0
            if z0 < zs / 2:
                a0 *= 2.0
            if z0 > zs * 2:
                a0 /= 1.9
            n += 1
            if not ((z0 > 2 * zs or z0 < zs / 2) and n < 15 and a0 < 1e4):
                break
        a, n = a0 * 1.1, 0
        while True:
            z = dist(step(p, a, e, lo, hi))
            new = a0 + (zs - z0) / (z - z0) * (a - a0) if a > a0 else a + (zs - z) / (z0 - z) * (a0 - a)
            if abs(z - zs) < dz_min:
                dz_min, am = abs(z - zs), a
            z0, a0, a = z, a, new
            n += 1
            if not (abs(z - zs) > 0.2 and n < 10 and a < 1e4):
                break
        A, P = wave(step(p, 1.0, (0.0 if dz_min / zs > 1 else am) * e, lo, hi))
        C = 1 - A / np.where(Ar > 0, Ar, 1) * np.cos(Pr - P)
        Sn = A / np.where(Ar > 0, Ar, 1) * np.sin(Pr - P)
        rows += [C, Sn, C * C + Sn * Sn]
    R = np.concatenate(rows)
    grid, j0 = [MN], MN
    while True:
        j = np.arange(j0 + 1, MM)
        if not len(j):
            break
        jm = (j + j0) // 2
        mid = (R[:, [j0]] * (j - jm) + R[:, j] * (jm - j0)) / (j - j0)
        bad = (np.abs(R[:, jm] - mid) > np.maximum(0.003 * ratio[j], 0.003)).any(0) | (j - j0 > int(100 * T))
        if not bad.any():
            break
        j0 = int(j[np.argmax(bad)])
        grid.append(j0)
    dfa = np.full(nh, 100)
    for a, b in zip(grid, grid[1:]):
        dfa[a:b] = b - a
    dfa[grid[-1]:MM] = MM - grid[-1]
    out, j = [MN], MN
    while True:
        jm = dfa[j]
        while True:
            kk = j + 2 * jm
            m = min(jm, dfa[j:kk + 1].min())
            again = m < jm and kk < nh
            jm = m
            if not again:
                break
        j = kk
        out += [out[-1] + jm, out[-1] + 2 * jm]
        if j >= MM:
            break
    jm = (MM - out[-3]) // 2
    if jm >= 1:
        out[-2:] = [out[-3] + jm, out[-3] + 2 * jm]
    return np.array(out), MN, MM


@pytest.mark.parametrize("Tobs,fs,labels,m1,m2,seed", [(4.0, 2048.0, [0, 1], 36.0, 29.0, 5), (8.0, 4096.0, [2], 12.0, 8.0, 6),
                                                       (16.0, 2048.0, [1, 0, 2], 10.0, 6.0, 7)])
def test_grid_equals_serial_search(ora, Tobs, fs, labels, m1, m2, seed):
    ev = synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=fs, fmin=16.0, m1=m1, m2=m2, chi1=0.2,
                          chi2=-0.1, snr=20.0, seed=seed)
    lo, hi = prior_bounds(Tobs)
    want, MN, MM = serial_het_space(ora, ev, ev.inj, lo, hi)
    e = q.Event.from_synthetic(ev)
    g, mn, mm = e.het_space(ev.inj, lo, hi)
    assert (mn, mm) == (MN, MM)
    assert np.array_equal(g, want)
    e.close()
