"""The CPU oracle in long double: qcbc_oracle.c with its type and its quotients of whole numbers widened, so that a
64-bit result's own rounding can be measured."""
import ctypes as C
import os
import re
import subprocess

import numpy as np

from conftest import ROOT

LD = np.longdouble
_TABLES = ("amp", "phase", "IP", "SL", "lc", "ls", "aa", "rc", "rs")


def _wide(text):
    text = re.sub(r"\bdouble\b", "long double", text)
    text = re.sub(r"(\d+\.0*) / (\d+\.0*)(?!\d)", r"\1L / \2L", text).replace("1 / 6.0", "1.0L / 6.0L")
    text = re.sub(r"(#define O_PI(?:_4)?\s+[\d.]+)", r"\1L", text)
    text = re.sub(r"(#define O_TPI\s+)[\d.]+", r"\g<1>6.283185307179586476925286766559005768L", text)
    return text.replace("#include <math.h>", "#include <tgmath.h>")


class Oracle:
    def __init__(self, tmp):
        src = os.path.join(ROOT, "oracle")
        os.makedirs(os.path.join(tmp, "_build"), exist_ok=True)
        for name in ("qcbc_oracle.c", "qcbc_oracle.h", os.path.join("_build", "qnm_table.h")):
            with open(os.path.join(src, name)) as f, open(os.path.join(tmp, name), "w") as g:
                g.write(_wide(f.read()))
        lib = os.path.join(tmp, "liboracle_ld.so")
        subprocess.run(["gcc", "-std=gnu99", "-O2", "-fPIC", "-fopenmp", "-w", "-shared", "-o", lib,
                        os.path.join(tmp, "qcbc_oracle.c"), "-lm"], check=True)
        self.L = C.CDLL(lib)
        v, i, r = C.c_void_p, C.c_int, C.c_longdouble
        self.L.ora_lnl_full_batch.argtypes = [v, i, r, v, v, i, v, v, i, i, r, r, r, v, i]
        self.L.ora_lnl_full_batch.restype = r
        self.L.ora_heterodyne.argtypes = [v, i, r, v, v, i, v, v, i, r, v, i, i, i, i] + [v] * 10
        self.L.ora_lnl_het_batch.argtypes = [v, i, r, r, v, i, i] + [v] * 9 + [r, v, i, v, i]
        self.L.ora_lnl_het_batch.restype = r

    @staticmethod
    def _p(a):
        return a.ctypes.data_as(C.c_void_p)

    def _event(self, ev):
        self.lab = np.ascontiguousarray(ev.labels, dtype=np.int32)
        self.D, self.S, self.f = (np.ascontiguousarray(np.asarray(x).astype(LD)) for x in (ev.D, ev.SN, ev.freq))
        return self.lab, len(self.lab), LD(ev.GMST)

    def lnl_full(self, ev, P, fmax=1024.0):
        lab, n, gmst = self._event(ev)
        P, out = np.ascontiguousarray(P.astype(LD)), np.zeros(len(P), LD)
        self.L.ora_lnl_full_batch(self._p(lab), n, gmst, self._p(self.D), self._p(self.S), ev.SN.shape[1],
                                  self._p(self.f), self._p(P), len(P), ev.N, ev.Tobs, ev.fmin, fmax, self._p(out), 0)
        return out

    def lnl_het(self, ev, ref, grid, P):
        """Tables about ref on the grid (J = 2), and the sets' likelihood from them."""
        lab, n, gmst = self._event(ev)
        g = np.ascontiguousarray(grid, dtype=np.int32)
        M, NR = len(g), (len(g) - 1) // 2
        shapes = dict(amp=(n, M), phase=(n, M), IP=(NR, 3, 3), SL=(NR, n, 3), lc=(NR, n, 3), ls=(NR, n, 3), aa=(n, NR),
                      rc=(n, NR), rs=(n, NR))
        t = {k: np.zeros(s, LD) for k, s in shapes.items()}
        logLb = np.zeros(1, LD)
        ref, P, out = ref.astype(LD), np.ascontiguousarray(P.astype(LD)), np.zeros(len(P), LD)
        self.L.ora_heterodyne(self._p(lab), n, gmst, self._p(self.D), self._p(self.S), ev.SN.shape[1], self._p(self.f),
                              self._p(ref), ev.N, ev.Tobs, self._p(g), M, int(g[0]), int(g[-1]), 2,
                              *[self._p(t[k]) for k in _TABLES], self._p(logLb))
        f = g.astype(LD) / LD(ev.Tobs)
        self.L.ora_lnl_het_batch(self._p(lab), n, gmst, ev.Tobs, self._p(f), M, 2, *[self._p(t[k]) for k in _TABLES],
                                 logLb[0], self._p(P), len(P), self._p(out), 0)
        return out
