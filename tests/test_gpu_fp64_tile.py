"""The FP64 full-likelihood tile against the CPU oracle where it can go wrong: rows that straddle the
waveform's piece boundaries, remainders of the two-row step, blocks of 32 to 256 threads, tiles around the
64-row table segments, one to three detectors, a Tobs that is no power of two, and sets outside the tables'
range (very heavy systems, extreme spins and a merger time far outside the segment take the per-bin
functions).

Tolerance: the phase reaches 2 pi f Tobs ~ 5e4 rad here, so each side's FP64 rounding is ~1e-11 rad per bin
and the inner products (network SNR 20, |lnL| below a few hundred) agree to ~1e-9; 1e-8 absolute is the
bound the FP64 likelihood is held to against the reference, taken relative above |lnL| = 100."""
import numpy as np
import pytest

import quickcbc_b200 as q
from conftest import oracle_template
from quickcbc_b200 import synth

pytestmark = pytest.mark.gpu


def _close(got, want):
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-8)


@pytest.fixture(scope="module", params=[(4.0, 2048.0, [1], 60.0, 40.0), (8.0, 4096.0, [0, 2], 20.0, 9.0),
                                        (7.3, 2000.0, [2, 1, 0], 30.0, 30.0), (32.0, 4096.0, [0, 1, 2], 5.0, 3.0)],
                ids=["4s-1det", "8s-2det", "7.3s-3det", "32s-3det"])
def case(request, ora):
    Tobs, fs, labels, m1, m2 = request.param
    ev = synth.make_event(oracle_template(ora), labels=labels, Tobs=Tobs, fs=fs, fmin=20.0, m1=m1, m2=m2, chi1=0.3,
                          chi2=-0.2, snr=20.0, seed=int(Tobs * 10))
    rng = np.random.default_rng(5)
    mc = np.exp(ev.inj[0]) / synth.MSUN_SI
    P = np.vstack([synth.jitter_params(rng, 3, ev.inj), synth.draw_params(rng, 4, ev.inj, mc=(0.6 * mc, 1.5 * mc))])
    want, _ = ora.lnl_full_batch(ev, P)
    return ev, P, want


@pytest.mark.parametrize("tiles,threads", [(0, 0), (1, 32), (1, 64), (2, 96), (1, 256), (7, 64), (33, 32)])
def test_launch_shapes(case, tiles, threads):
    ev, P, want = case
    e = q.Event.from_synthetic(ev)
    e.set_launch(tiles, threads)
    got, rho = e.lnl_full(P, q.FP64, rho=True)
    _close(got, want)
    assert np.all(np.isfinite(rho))
    e.close()


def test_one_tile_in_order_of_length(case, ora):
    ev, P, want = case
    e = q.Event.from_synthetic(ev)
    reps = 1300 // len(P) + 1                     # enough sets for one tile per set, longest first
    e.set_launch(1, 64)
    got = e.lnl_full(np.tile(P, (reps, 1)), q.FP64)
    _close(got, np.tile(want, reps))
    e.close()


def test_sets_outside_the_tables(ora):
    ev = synth.make_event(oracle_template(ora), labels=[0, 1], Tobs=4.0, fs=2048.0, fmin=16.0, m1=40.0, m2=30.0,
                          chi1=0.1, chi2=0.1, snr=15.0, seed=31)
    P = np.tile(ev.inj, (6, 1))
    for k, (m1, m2, c1, c2) in enumerate([(160.0, 140.0, 0.0, 0.0), (300.0, 250.0, -0.8, -0.8), (90.0, 5.0, 0.99, 0.9),
                                          (45.0, 44.0, 0.99, 0.99), (20.0, 1.0, -0.99, 0.5)]):
        P[k, 0], P[k, 1] = synth.masses_to_params(m1, m2)
        P[k, 2:4] = c1, c2
    P[5, 5] = 3.0e5                               # merger time far outside: 3e8 cycles of linear phase
    want, _ = ora.lnl_full_batch(ev, P)
    e = q.Event.from_synthetic(ev)
    got = e.lnl_full(P, q.FP64)
    # at 3e8 cycles one ulp of the phase is 4e-7 rad on either side
    np.testing.assert_allclose(got[:5], want[:5], rtol=1e-10, atol=1e-8)
    np.testing.assert_allclose(got[5], want[5], rtol=0, atol=1e-3 * (1.0 + abs(want[5])))
    e.close()
