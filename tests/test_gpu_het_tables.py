"""Heterodyne tables built on the device against the CPU oracle, where the launch shapes change: regions
of one bin up to and across the 1024-bin chunks, one to three points per region, a band wider than the
grid, one to three detectors, and a Tobs whose 1/(1/Tobs) is another double.

Tolerance: every entry is a sum of FP64 terms whose phase (up to 2 pi f Tobs ~ 1e4 rad here) carries a
few times 1e-16 relative rounding on either side, so terms agree to ~1e-12 of their size; 1e-11 of the
table's largest entry leaves a factor of ten for the sums (the bound the oracle itself is held to)."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu

REGIONS = {
    1: [1, 2, 255, 256, 257, 1023, 1024, 1025],
    2: [2, 3, 511, 1023, 1024, 1025, 2048],
    3: [3, 4, 1023, 1024, 1026, 2049],
}


@pytest.mark.parametrize("J,labels,Tobs,pad", [(1, [0], 4.0, 0), (2, [0, 1], 4.0, 37), (2, [2, 0, 1], 7.3, 0),
                                               (3, [0, 1, 2], 8.0, 5)])
def test_tables_match_oracle_at_chunk_edges(ora, J, labels, Tobs, pad):
    ev = synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=4000.0 if Tobs == 7.3 else 4096.0,
                          fmin=16.0, m1=9.0, m2=6.0, chi1=0.2, chi2=-0.3, snr=20.0, seed=811 + J, tc=Tobs - 1.0)
    grid = [int(20 * Tobs)]
    for U in REGIONS[J]:
        if grid[-1] + U >= ev.N // 2:
            break
        inner = sorted({grid[-1] + max(k, round(U * k / J)) for k in range(1, J)})
        grid += inner + [grid[-1] + U]
    g = np.array(grid, dtype=np.int32)
    assert (len(g) - 1) % J == 0 and np.all(np.diff(g) > 0)
    MN, MM = int(g[0]) - pad, min(int(g[-1]) + pad, ev.N // 2)
    e = q.Event.from_synthetic(ev)
    e.het_setup(ev.inj, g, MN, MM, J)
    t = e.het_export()
    o = ora.heterodyne(ev, ev.inj, g, MN, MM, J)
    assert abs(t["logLb"] - o["logLb"]) <= 1e-11 * (abs(o["logLb"]) + ev.snr ** 2)
    for k in ("freq", "amp", "phase", "IP", "SL", "lc", "ls", "aa", "rc", "rs"):
        np.testing.assert_allclose(t[k], o[k], rtol=0, atol=1e-11 * np.abs(o[k]).max(), err_msg=k)
    P = synth.jitter_params(np.random.default_rng(3), 3, ev.inj)
    Lo, _ = ora.lnl_het_batch(ev, o, P)
    np.testing.assert_allclose(e.lnl_het(P, q.FP64), Lo, rtol=0, atol=1e-8)
    e.close()
