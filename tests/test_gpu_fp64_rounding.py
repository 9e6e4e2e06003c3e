"""The FP64 likelihoods' rounding, against the oracle in long double: no larger than that of the plain 64-bit
evaluation of the same sets (the double oracle), bin by bin with the library's functions.

The folded phase has fewer operations per bin than the plain one, but what it rounds once per set is the same in
every bin and does not average out, so the long signals are where it shows (1e5 rad, 1e6 cycles).  Bound: as much
as the plain evaluation, and half as much again for the spread of an rms over 24 sets."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from oracle_ld import LD, Oracle
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wide(tmp_path_factory, ora):
    return Oracle(str(tmp_path_factory.mktemp("ld")))


def rms(x, want):
    return float(np.sqrt(np.mean((np.asarray(x).astype(LD) - want) ** 2)))


@pytest.mark.parametrize("labels,Tobs,fs,m1,m2", [([0, 1], 32.0, 2048.0, 5.0, 3.0), ([1], 64.0, 2048.0, 3.0, 2.0),
                                                  ([0, 1, 2], 128.0, 4096.0, 1.45, 1.3)])
def test_no_more_than_plain_64_bits(ora, wide, labels, Tobs, fs, m1, m2):
    ev = synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=fs, fmin=20.0, m1=m1, m2=m2, chi1=0.03,
                          chi2=-0.02, snr=30.0, seed=17, tc=Tobs - 2.0)
    rng = np.random.default_rng(5)
    mc = np.exp(ev.inj[0]) / synth.MSUN_SI * 4.925491e-6
    dmc = 0.15 / (3.0 / 128.0 * (np.pi * mc * 20.0) ** (-5.0 / 3.0))        # a few tenths of a radian over the band
    P = ev.inj + np.array([dmc, 10 * dmc, 0.005, 0.005, 0.3, 1e-4, 0.1, 0.02, 0.0, 0.3, 0.0]) * rng.normal(size=(24, 11))
    P[:, 0] = np.minimum(P[:, 0], P[:, 1] + 0.6 * np.log(0.25) - 1e-9)
    grid = np.unique(np.round(np.geomspace(20 * Tobs, 900 * Tobs, 47)).astype(np.int32))
    e = q.Event.from_synthetic(ev)
    want = wide.lnl_full(ev, P)
    plain = rms(ora.lnl_full_batch(ev, P)[0], want)
    small = e.lnl_full(P, q.FP64)
    large = e.lnl_full(np.vstack([P] * 8), q.FP64)[:24]
    print("full: plain %.2e, one launch %.2e, two %.2e" % (plain, rms(small, want), rms(large, want)))
    assert rms(small, want) <= 1.5 * plain and rms(large, want) <= 1.5 * plain
    want = wide.lnl_het(ev, ev.inj, grid, P)
    t = ora.heterodyne(ev, ev.inj, grid, int(grid[0]), int(grid[-1]), 2)
    plain = rms(ora.lnl_het_batch(ev, t, P)[0], want)
    e.het_setup(ev.inj, grid, int(grid[0]), int(grid[-1]), 2)
    small = e.lnl_het(P, q.FP64)
    large = e.lnl_het(np.vstack([P] * 6), q.FP64)[:24]
    print("heterodyned: plain %.2e, one launch %.2e, two %.2e" % (plain, rms(small, want), rms(large, want)))
    assert rms(small, want) <= 1.5 * plain and rms(large, want) <= 1.5 * plain
    e.close()
