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


def test_precisions_side_by_side_on_two_streams(batch):
    """Device-form calls of the two precisions at one tiling, queued on two streams: neither waits for the other,
    so they share no scratch."""
    b, eo, P = batch
    b.set_tiling(2048, 128)
    n = 60
    eo, P = np.tile(eo, n), np.tile(P, (n, 1))
    want = {p: b.lnl(eo, P, p) for p in (q.FP64, q.MIXED)}
    L, vp = _lib.lib(), C.c_void_p
    dP, dE = q.DeviceBuffer(P.nbytes), q.DeviceBuffer(eo.nbytes)
    dP.upload(P)
    dE.upload(eo)
    import torch
    streams = {p: torch.cuda.Stream() for p in want}
    outs = {p: [q.DeviceBuffer(8 * len(eo)) for _ in range(6)] for p in want}
    for k in range(6):
        for p in want:
            assert L.qcbc_lnl_multi_dev(vp(b._h), vp(dE.ptr), vp(dP.ptr), len(eo), vp(outs[p][k].ptr), p,
                                        vp(streams[p].cuda_stream)) == 0, _lib.last_error()
    torch.cuda.synchronize()
    for p in want:
        for k in range(6):
            assert np.array_equal(outs[p][k].download((len(eo),)), want[p]), (p, k)
    b.set_tiling(2048, 256)
