"""Calls that reach the same result by two routes, and results that only one test would notice.

* mixed precision: the kernel that makes the records itself and the launch after a setup of its own (forced by results
  that overlap the parameters) give the same bits at the same launch shape, at the edge of the rule (296 blocks);
* the heterodyned likelihood with its results in its parameters' memory;
* rho of a multi-event call, written by the set's last tile or, for a rejected set, with the work list;
* what each kind of unusable parameter gives.

Tolerances: 1e-3 in lnL for mixed against the oracle and 1e-8 / 1e-10 for FP64, as elsewhere; the rest is equality."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def make(ora, labels, Tobs=4.0, seed=5):
    return synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=2048.0, fmin=16.0, m1=36.0, m2=29.0,
                            chi1=0.3, chi2=-0.1, snr=20.0, seed=seed)


def on_device(call, e, P, precision, in_place, *outs):
    dP = q.DeviceBuffer(P.nbytes)
    dP.upload(P)
    dL = dP if in_place else q.DeviceBuffer(8 * len(P))
    assert call(e.handle, dP.ptr, len(P), dL.ptr, *outs, precision, None) == 0, _lib.last_error()
    assert _lib.lib().qcbc_synchronize() == 0
    return dL.download((len(P),))


@pytest.mark.parametrize("labels", [[0], [2, 1], [0, 1, 2]])
@pytest.mark.parametrize("B,tiles,threads", [(1, 7, 128), (17, 1, 256), (98, 3, 128), (148, 2, 256)])
def test_mixed_one_launch_equals_two(ora, labels, B, tiles, threads):
    ev = make(ora, labels)
    P = synth.jitter_params(np.random.default_rng(B), B, ev.inj)
    e = q.Event.from_synthetic(ev)
    e.set_launch(tiles, threads)
    one = e.lnl_full(P, q.MIXED)
    dev = on_device(_lib.lib().qcbc_lnl_full_dev, e, P, q.MIXED, False, None)
    two = on_device(_lib.lib().qcbc_lnl_full_dev, e, P, q.MIXED, True, None)
    assert np.array_equal(one, dev) and np.array_equal(one, two)
    want, _ = ora.lnl_full_batch(ev, P)
    np.testing.assert_allclose(one, want, rtol=0, atol=1e-3)
    e.close()


@pytest.mark.parametrize("precision", [q.FP64, q.MIXED])
@pytest.mark.parametrize("B", [1, 17, 128, 129])
def test_heterodyned_in_place(ora, B, precision):
    ev = make(ora, [0, 1, 2], Tobs=8.0)
    g = np.arange(160, 160 + 64 * 41, 64, dtype=np.int32)
    e = q.Event.from_synthetic(ev)
    e.het_setup(ev.inj, g, int(g[0]), int(g[-1]), 2)
    P = synth.jitter_params(np.random.default_rng(B), B, ev.inj)
    want = e.lnl_het(P, precision)
    for in_place in (False, True):
        assert np.array_equal(on_device(_lib.lib().qcbc_lnl_het_dev, e, P, precision, in_place), want), in_place
    e.close()


@pytest.mark.parametrize("precision,tol", [(q.FP64, 1e-9), (q.MIXED, 1e-4)])
def test_rho_of_many_events(ora, precision, tol):
    evs = [make(ora, lab, T, 5 + k) for k, (lab, T) in enumerate([([1], 4.0), ([0, 2], 8.0), ([2, 0, 1], 16.0)])]
    hs = [q.Event.from_synthetic(ev) for ev in evs]
    b = q.Batch(hs)
    rng = np.random.default_rng(3)
    eo = np.repeat(np.arange(3, dtype=np.int32), 12)
    P = np.vstack([synth.jitter_params(rng, 12, ev.inj) for ev in evs])
    P[14, 2] = 1.5                                    # rejected
    eo[30] = 7                                        # no such event
    bad = np.isin(np.arange(36), (14, 30))
    lnl, rho = b.lnl(eo, P, precision, rho=True, allow_invalid=True)
    assert np.all(lnl[bad] == -1e20) and np.all(rho[bad] == 0.0) and np.all(lnl[~bad] > -1e20)
    for k, (ev, e) in enumerate(zip(evs, hs)):
        at = (eo == k) & ~bad
        L, r = e.lnl_full(P[at], precision, rho=True)
        np.testing.assert_allclose(rho[at][:, :ev.nifo], r, rtol=0, atol=tol)
        assert np.all(rho[at][:, ev.nifo:] == 0.0)
        h = np.array([ora.lnl_full(ev, p)[1] for p in P[at]])
        np.testing.assert_allclose(r, h, rtol=0, atol=1e-9 if precision == q.FP64 else 1e-3)
    b.close()
    for e in hs:
        e.close()


# parameter, value -> rejected (masses, spins or distance that no system has), nan, or the oracle's likelihood (equal
# masses stand in for a chirp mass that is too large; a NaN or negative merger time leaves no bin, an infinite
# distance no signal)
OUTCOMES = [(k, v, "rejected") for k in range(4) for v in (np.nan, -800.0, 800.0) if (k, v) != (0, 800.0)]
OUTCOMES += [(0, 800.0, "oracle"), (4, np.nan, "nan"), (4, -800.0, "oracle"), (4, 800.0, "oracle"), (5, np.nan, 0.0),
             (5, -800.0, 0.0), (5, 800.0, "oracle"), (6, np.nan, "rejected"), (6, -800.0, "rejected"), (6, 800.0, 0.0)]


@pytest.mark.parametrize("k,v,what", OUTCOMES)
def test_unusable_parameters(ora, k, v, what):
    ev = make(ora, [0, 1])
    P = synth.jitter_params(np.random.default_rng(1), 6, ev.inj)
    P[2, k] = v
    e = q.Event.from_synthetic(ev)
    big = np.vstack([P] * 80)                         # several waves: two launches
    for prec, tol in ((q.FP64, 1e-8), (q.MIXED, 1e-3)):
        for got in (e.lnl_full(P, prec, allow_invalid=True)[2], e.lnl_full(big, prec, allow_invalid=True)[2]):
            if what == "rejected":
                assert got == -1e20
            elif what == "nan":
                assert np.isnan(got)
            else:
                want = ora.lnl_full(ev, P[2])[0] if what == "oracle" else what
                np.testing.assert_allclose(got, want, rtol=1e-10, atol=tol)
    e.close()
