"""The tilings of a batch: one per precision, set together, tuned apart, and left as they were by a tuning that
fails."""
import ctypes as C

import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch(ora):
    evs = [synth.make_event(oracle_template(ora), labels=lab, Tobs=T, fs=2048.0, fmin=16.0, m1=20.0, m2=15.0, chi1=0.1,
                            chi2=0.0, snr=18.0, seed=70 + k) for k, (lab, T) in enumerate([([0, 1], 8.0), ([0, 1, 2], 16.0)])]
    hs = [q.Event.from_synthetic(ev) for ev in evs]
    b = q.Batch(hs)
    eo = np.repeat(np.arange(2, dtype=np.int32), 40)
    P = np.vstack([synth.draw_params(np.random.default_rng(k), 40, ev.inj) for k, ev in enumerate(evs)])
    yield b, eo, P
    b.close()
    for h in hs:
        h.close()


def test_tuning_one_precision_leaves_the_other(batch):
    b, eo, P = batch
    assert b.tiling() == b.tiling(q.MIXED) == (2048, 256) and b.tiling(q.FP64) == (4096, 128)
    mixed = b.lnl(eo, P, q.MIXED)
    got = b.autotune(eo, P, q.FP64)
    assert got == b.tiling(q.FP64) == b.tiling()
    assert b.tiling(q.MIXED) == (2048, 256)
    assert np.array_equal(b.lnl(eo, P, q.MIXED), mixed)
    fp64, kept = b.lnl(eo, P, q.FP64), b.tiling(q.FP64)
    assert b.autotune(eo, P, q.MIXED) == b.tiling(q.MIXED)
    assert b.tiling(q.FP64) == kept and np.array_equal(b.lnl(eo, P, q.FP64), fp64)
    b.set_tiling(4096, 256)
    assert b.tiling(q.MIXED) == b.tiling(q.FP64) == (4096, 256)
    b.set_tiling(2048, 0)
    assert b.tiling(q.MIXED) == b.tiling(q.FP64) == (2048, 256)


def test_failed_tuning_changes_nothing(batch):
    L = _lib.lib()
    h = L.qcbc_batch_create_slots(1, 1 << 20)
    assert h
    n = (1 << 20) + 1                                   # times 1024 tiles of the first candidate: refused
    eo, P = np.zeros(n, dtype=np.int32), np.zeros((n, 11))
    pi = C.POINTER(C.c_int)
    t, th = C.c_int(), C.c_int()
    for prec, want in ((q.MIXED, (2048, 256)), (q.FP64, (4096, 128))):
        rc = L.qcbc_batch_autotune(h, eo.ctypes.data_as(pi), P.ctypes.data_as(C.POINTER(C.c_double)), n, prec)
        assert rc not in (0, _lib.QCBC_EDOM)
        assert L.qcbc_batch_get_tiling_of(h, prec, C.byref(t), C.byref(th)) == 0
        assert (t.value, th.value) == want
    L.qcbc_batch_destroy(h)
