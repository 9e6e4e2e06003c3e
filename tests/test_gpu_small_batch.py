"""Batches small enough that the likelihood kernel makes the records itself, at the edges of that rule and of the
16 sets whose parameters travel as kernel arguments: FP64 against the CPU oracle and against the launch with a
setup of its own, the heterodyned likelihood against the same sets in a larger batch, and parameters read from
device memory or overwritten by the results.

Tolerance: the FP64 likelihood's 1e-8 absolute bound against the reference (phases of ~1e4 rad in FP64); the
other comparisons run the same code in the same order, or (other tiles) differ by the same rounding."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def make(ora, labels, Tobs=4.0):
    return synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=2048.0, fmin=16.0, m1=36.0, m2=29.0,
                            chi1=0.3, chi2=-0.1, snr=20.0, seed=5)


@pytest.mark.parametrize("labels", [[0], [2, 1], [0, 1, 2]])
@pytest.mark.parametrize("B", [1, 15, 16, 17, 48, 49, 148, 149])
def test_full_at_the_rule_edges(ora, labels, B):
    ev = make(ora, labels)
    P = synth.draw_params(np.random.default_rng(B), B, ev.inj)
    want, _ = ora.lnl_full_batch(ev, P)
    e = q.Event.from_synthetic(ev)
    got, rho = e.lnl_full(P, q.FP64, rho=True)
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-8)
    e.set_launch(3, 64)                              # blocks too small to make a record: two launches
    two, rho2 = e.lnl_full(P, q.FP64, rho=True)
    np.testing.assert_allclose(got, two, rtol=1e-10, atol=1e-8)
    np.testing.assert_allclose(rho, rho2, rtol=1e-10, atol=1e-10)
    e.close()


@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("B", [1, 16, 17])
def test_device_parameters(ora, B, in_place):
    ev = make(ora, [0, 1, 2])
    P = synth.draw_params(np.random.default_rng(B), B, ev.inj)
    e = q.Event.from_synthetic(ev)
    want = e.lnl_full(P, q.FP64)
    dP = q.DeviceBuffer(P.nbytes)
    dP.upload(P)
    dL = dP if in_place else q.DeviceBuffer(B * 8)
    assert _lib.lib().qcbc_lnl_full_dev(e.handle, dP.ptr, B, dL.ptr, None, q.FP64, None) == 0, _lib.last_error()
    assert _lib.lib().qcbc_synchronize() == 0
    assert np.array_equal(dL.download((B,)), want)
    e.close()


@pytest.mark.parametrize("precision", [q.FP64, q.MIXED])
@pytest.mark.parametrize("labels", [[1], [0, 1], [0, 1, 2]])
def test_heterodyned_same_bits_in_any_batch(ora, labels, precision):
    ev = make(ora, labels, Tobs=8.0)
    g = np.arange(160, 160 + 16 * 201, 16, dtype=np.int32)   # 201 points: more than a block's threads
    e = q.Event.from_synthetic(ev)
    e.het_setup(ev.inj, g, int(g[0]), int(g[-1]), 2)
    P = synth.jitter_params(np.random.default_rng(3), 129, ev.inj)
    P[7, 2] = 1.5
    want = e.lnl_het(P, precision, allow_invalid=True)
    for B in (1, 16, 17, 128):
        assert np.array_equal(e.lnl_het(P[:B], precision, allow_invalid=True), want[:B]), B
    assert want[7] == -1e20 and np.all(np.isfinite(want))
    e.close()
