"""The computed ringdown table against the literature: without the reference the product and the oracle take the same
table, so an error in it shows in no comparison of the two."""
import numpy as np

from quickcbc_b200 import qnm

# M omega of the l = m = 2, n = 0 Kerr mode, six digits (Leaver 1985 at a = 0; the tables of Berti, Cardoso and Will,
# Phys. Rev. D 73, 064030, elsewhere)
PUBLISHED = {0.0: (0.373672, 0.088962), 0.5: (0.464123, 0.085639), 0.7: (0.532600, 0.080793),
             0.9: (0.671614, 0.064869), 0.98: (0.825429, 0.038630), 0.99: (0.870893, 0.029390)}


def test_modes_against_published_values():
    w = qnm.kerr_mode(list(PUBLISHED))
    for got, (re, im) in zip(w, PUBLISHED.values()):
        assert abs(float(got.real) - re) <= 6e-7 and abs(float(-got.imag) - im) <= 6e-7


def test_table_rows():
    a, fr, fd = (np.array(x) for x in qnm.table())
    assert len(a) == 1003 and a[0] == -1.0 and a[-1] == 1.0 and np.all(np.diff(a) > 0)
    # the rows hold the modes, to six significant digits
    for s, w in zip(PUBLISHED, qnm.kerr_mode(list(PUBLISHED))):
        k = int(np.argmin(np.abs(a - s)))
        assert a[k] == s
        assert fr[k] == float("%.6g" % (float(w.real) / (2 * np.pi)))
        assert fd[k] == float("%.6g" % (float(-w.imag) / (2 * np.pi)))
    # frequencies rise with spin to 1 / 2 pi, the damping falls to zero
    assert np.all(np.diff(fr) > 0) and fr[-1] == float("%.6g" % (1 / (2 * np.pi)))
    assert fd[-1] == 0.0 and np.all(np.diff(fd[a >= 0.0]) < 0)
