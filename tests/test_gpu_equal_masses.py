"""Nearly equal masses with unequal spins.  There sqrt(1 - 4 eta) keeps only eta's rounding, which the final spin and
the fits' chi carry into the waveform on both sides of a comparison; whatever else takes the masses' difference has
to take it from the masses.  The likelihood's setup and the waveform outputs' round the masses alike, so lnL and the
inner products of the library's own template differ by FP64 rounding alone.

Tolerance: 1e-8 in lnL, as for the FP64 likelihood elsewhere (phases up to 1e5 rad, network SNR 30); a difference taken
from 1 - 4 eta shows as 1e-7 to 5e-7."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("below", [0.0, 1e-15, 1e-14, 1e-13, 1e-12])
@pytest.mark.parametrize("Tobs,m", [(16.0, 27.0), (32.0, 4.0)])
def test_likelihood_of_the_librarys_own_template(ora, Tobs, m, below):
    ev = synth.make_event(oracle_template(ora), labels=[0, 1], Tobs=Tobs, fs=2048.0, fmin=20.0, m1=1.01 * m, m2=m,
                          chi1=0.4, chi2=-0.4, snr=30.0, seed=23, tc=Tobs - 2.0)
    P = np.tile(ev.inj, (6, 1))
    P[:, 0] = P[:, 1] + 0.6 * np.log(0.25) - below
    P[:, 2], P[:, 3] = [-0.9, 0.9, 0.0, 0.8, -0.5, 0.3], [0.0, -0.9, 0.9, 0.1, 0.5, -0.3]
    e = q.Event.from_synthetic(ev)
    got = e.lnl_full(P, q.FP64)
    lo, hi = int(Tobs * 20.0), min(int(Tobs * 1024.0), ev.N // 2)
    i = np.arange(lo, hi)
    for p, L in zip(P, got):
        h = q.fulltemplates(ev.labels, ev.GMST, ev.freq, p, ev.N)
        want = 0.0
        for d, t, s in zip(ev.D, h, ev.SN):
            want += float(np.sum(4.0 * (d[i] * t[i] + d[ev.N - i] * t[ev.N - i]) / s[i]))
            want -= float(np.sum(2.0 * (t[i] ** 2 + t[ev.N - i] ** 2) / s[i]))
        assert abs(L - want) <= 1e-8
    e.close()
