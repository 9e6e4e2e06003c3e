"""The likelihood setup (8 lanes per set, four sets per block) against the CPU oracle at the edges of its
blocks, with rejected sets between good ones, for one to three detectors and the intrinsic model, and with a
QNM table whose spacing is too fine for the one-row lookup (the binary search takes its place).

Tolerance: the FP64 likelihood's 1e-8 absolute bound against the reference (phases of ~1e4 rad in FP64)."""
import ctypes as C

import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import _lib, qnm, synth

pytestmark = pytest.mark.gpu


def make(ora, labels, seed=3):
    return synth.make_event(oracle_template(ora), labels=labels, Tobs=4.0, fs=2048.0, fmin=16.0, m1=36.0, m2=29.0,
                            chi1=0.3, chi2=-0.1, snr=20.0, seed=seed)


@pytest.mark.parametrize("labels", [[0], [2, 1], [0, 1, 2]])
@pytest.mark.parametrize("B", [1, 3, 4, 5, 9])
def test_block_edges_and_rejected_sets(ora, labels, B):
    ev = make(ora, labels)
    rng = np.random.default_rng(B)
    P = np.vstack([synth.draw_params(rng, B, ev.inj), synth.jitter_params(rng, 1, ev.inj)])[:max(B, 1)]
    want, _ = ora.lnl_full_batch(ev, P)
    bad = B // 2 if B > 1 else -1
    if bad >= 0:
        P[bad, 2] = 1.5                              # outside the spin range
    e = q.Event.from_synthetic(ev)
    got = e.lnl_full(P, q.FP64, allow_invalid=True)
    mixed = e.lnl_full(P, q.MIXED, allow_invalid=True)
    ok = np.arange(len(P)) != bad
    np.testing.assert_allclose(got[ok], want[ok], rtol=1e-10, atol=1e-8)
    assert np.all(np.isfinite(mixed)) and np.all(mixed[ok] > -1e20)
    if bad >= 0:
        assert got[bad] == -1e20 and mixed[bad] == -1e20
    e.close()


@pytest.mark.parametrize("change", [dict(k=0, v=-800.0), dict(k=1, v=800.0), dict(k=6, v=-800.0), dict(k=3, v=np.nan),
                                    dict(k=0, v=np.nan)])
def test_extreme_parameters_leave_their_neighbours_alone(ora, change):
    ev = make(ora, [0, 1])
    P = synth.jitter_params(np.random.default_rng(1), 6, ev.inj)
    want, _ = ora.lnl_full_batch(ev, P)
    P[2, change["k"]] = change["v"]
    e = q.Event.from_synthetic(ev)
    got = e.lnl_full(P, q.FP64, allow_invalid=True)
    ok = np.arange(6) != 2
    np.testing.assert_allclose(got[ok], want[ok], rtol=1e-10, atol=1e-8)
    assert not (np.isfinite(got[2]) and got[2] > want.max())
    e.close()


def test_fine_qnm_table_same_likelihood(ora):
    """Knots added on the natural spline itself leave the spline as it is."""
    from scipy.interpolate import CubicSpline
    a, fr, fd = (np.array(v) for v in qnm.table())
    splines = [CubicSpline(a, y, bc_type="natural") for y in (fr, fd)]
    fine = np.sort(np.concatenate([a, np.linspace(-0.4004, 0.95003, 1500)]))
    fine = fine[np.concatenate([[True], np.diff(fine) > 1e-7])]
    pd = C.POINTER(C.c_double)

    def install(x, u, v):
        arr = [np.ascontiguousarray(w, dtype=np.float64) for w in (x, u, v)]
        _lib.check(_lib.lib().qcbc_set_qnm_table(*[w.ctypes.data_as(pd) for w in arr], len(arr[0])))
    ev = make(ora, [0, 1])
    P = synth.draw_params(np.random.default_rng(2), 9, ev.inj)
    want, _ = ora.lnl_full_batch(ev, P)
    e = q.Event.from_synthetic(ev)
    try:
        install(fine, splines[0](fine), splines[1](fine))
        np.testing.assert_allclose(e.lnl_full(P, q.FP64), want, rtol=1e-10, atol=1e-8)
    finally:
        install(a, fr, fd)
    np.testing.assert_allclose(e.lnl_full(P, q.FP64), want, rtol=1e-10, atol=1e-8)
    e.close()
