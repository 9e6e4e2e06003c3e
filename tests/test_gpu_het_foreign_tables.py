"""Heterodyne tables given by the caller (qcbc_het_set) may hold frequencies beyond the event's bins.  Above the
model's cut-off the waveform is zero there; no per-bin table is read for such a point.

Tolerance: FP64 as the heterodyned likelihood elsewhere (1e-8); mixed 2e-3 in lnL, ten times the bound that holds for
whole-band grids (2e-4), as the point without signal makes its region's terms of order SNR^2 instead of the residual's."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("labels", [[1], [0, 1, 2]])
@pytest.mark.parametrize("far", [1.0e5, 1.0e9])
def test_frequency_beyond_the_bins(ora, labels, far):
    ev = synth.make_event(oracle_template(ora), labels=labels, Tobs=8.0, fs=2048.0, fmin=16.0, m1=36.0, m2=29.0,
                          chi1=0.3, chi2=-0.1, snr=20.0, seed=9)
    g = np.unique(np.round(np.geomspace(160, 3000, 41)).astype(np.int32))
    g = g[:len(g) // 2 * 2 - 1]
    t = dict(ora.heterodyne(ev, ev.inj, g, int(g[0]), int(g[-1]), 2))
    t["freq"] = t["freq"].copy()
    t["freq"][-1] = far
    P = synth.jitter_params(np.random.default_rng(2), 200, ev.inj)
    want, _ = ora.lnl_het_batch(ev, t, P)
    e = q.Event.from_synthetic(ev)
    e.het_set(t)
    b = q.Batch([e])
    zero = np.zeros(len(P), dtype=np.int32)
    for prec, tol in ((q.FP64, 1e-8), (q.MIXED, 2e-3)):
        for got in (e.lnl_het(P, prec), np.concatenate([e.lnl_het(P[:7], prec), e.lnl_het(P[7:], prec)]),
                    b.lnl_het(zero, P, prec)):
            np.testing.assert_allclose(got, want, rtol=0, atol=tol)
    b.close()
    e.close()
