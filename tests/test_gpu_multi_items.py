"""The work list of a multi-event launch: tiles of every kind (one to three detectors, light and heavy binaries whose
tiles start in each waveform piece), tile lengths from shorter than a row to longer than any band, rejected sets
between good ones, batches at the list's block edges.  Each set against its own event's likelihood, bit-equal in
any order and batch, and from device memory.

Tolerance: the FP64 likelihood's 1e-8 absolute bound (phases of ~1e4 rad in FP64); other tiles only round the same
sums differently."""
import ctypes as C

import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import _lib, synth

pytestmark = pytest.mark.gpu

EVENTS = [dict(labels=[0], Tobs=4.0, m1=60.0, m2=45.0), dict(labels=[1, 0], Tobs=8.0, m1=12.0, m2=8.0),
          dict(labels=[0, 1, 2], Tobs=16.0, m1=3.0, m2=2.0), dict(labels=[2, 1, 0], Tobs=4.0, m1=30.0, m2=28.0)]


@pytest.fixture(scope="module")
def mixed_events(ora):
    evs = [synth.make_event(oracle_template(ora), fs=2048.0, fmin=16.0, chi1=0.2, chi2=-0.1, snr=18.0, seed=31 + k, **s)
           for k, s in enumerate(EVENTS)]
    hs = [q.Event.from_synthetic(ev) for ev in evs]
    yield evs, hs
    for h in hs:
        h.close()


def sets(evs, n, seed):
    rng = np.random.default_rng(seed)
    eo = rng.integers(0, len(evs), n).astype(np.int32)
    P = np.vstack([synth.jitter_params(rng, 1, evs[e].inj) if rng.random() < 0.5 else synth.draw_params(rng, 1, evs[e].inj)
                   for e in eo])
    return eo, np.ascontiguousarray(P)


@pytest.mark.parametrize("tiling", [(0, 0), (20, 64), (2048, 128), (4097, 64), (100000, 256)])
@pytest.mark.parametrize("n", [1, 5, 127, 128, 129, 300])
def test_sets_of_every_kind(mixed_events, tiling, n):
    evs, hs = mixed_events
    eo, P = sets(evs, n, n)
    want = np.empty(n)
    for e, h in enumerate(hs):
        if np.any(eo == e):
            want[eo == e] = h.lnl_full(P[eo == e], q.FP64)
    bad = n // 2 if n > 1 else -1
    if bad >= 0:
        P[bad, 2] = 1.5                              # outside the spin range
        want[bad] = -1e20
    b = q.Batch(hs)
    b.set_tiling(*tiling)
    got = b.lnl(eo, P, q.FP64, allow_invalid=True)
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-8)
    perm = np.random.default_rng(7).permutation(n)
    for prec in (q.FP64, q.MIXED):
        one = b.lnl(eo, P, prec, allow_invalid=True)
        assert np.array_equal(b.lnl(eo[perm], P[perm], prec, allow_invalid=True), one[perm])
        dP, dE, dL = q.DeviceBuffer(P.nbytes), q.DeviceBuffer(eo.nbytes), q.DeviceBuffer(8 * n)
        dP.upload(P)
        dE.upload(eo)
        vp = C.c_void_p
        assert _lib.lib().qcbc_lnl_multi_dev(b._h, vp(dE.ptr), vp(dP.ptr), n, vp(dL.ptr), prec, None) == 0
        assert _lib.lib().qcbc_synchronize() == 0
        assert np.array_equal(dL.download((n,)), one)
    b.close()
