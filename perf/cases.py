"""Performance cases of the likelihood engine: what a sampler on top of it calls.

A case is one call (or the two calls that always go together) on an analysis that is already open:

  full      batched full likelihood of one event, FP64 or mixed, from host arrays (Event.lnl_full) or
            with parameters and results on the device (qcbc_lnl_full_dev)
  het       heterodyned likelihood, the production hot loop of a long run, host or device form
  multi     sets of many uneven events in one call (Batch.lnl / qcbc_lnl_multi_dev), the service's step
  tables    heterodyne tables for a given grid (Event.het_setup and het_export): once per analysis and
            whenever the reference point moves
  grid      the heterodyne grid search (Event.het_space): admission of an analysis
  redraw    noise marginalisation: a drawn PSD replaces the event's (set_psd_sample), then the likelihoods
            of the chains under it

Sizes are those of the synthetic configurations (4 s / 2 detectors / 2048 Hz, 16 s / 3 / 4096 Hz, 128 s
neutron-star binary, uneven batches of 4-64 s), of the reference's sampler (1 set per call, 12-16 chains)
and ragged ones between.  exact() restates every likelihood and table in 64-bit torch from the published
model (IMRPhenomD, arXiv:1508.07253; QNM frequencies by Leaver's method), with none of the engine's code.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import quickcbc_b200 as q
from quickcbc_b200 import ingest, synth
from quickcbc_b200._lib import check, lib

DEV = "cuda" if torch.cuda.is_available() else "cpu"
MSUN, PC = synth.MSUN_SI, synth.PC_SI


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference sampler's call on the smallest analysis: one chain, one set (latency)
        dict(name="full-fp64-1-4s", kind="full", prec="fp64", io="host", nifo=2, Tobs=4.0, fs=2048.0, fmin=16.0,
             mt=65.0, q=0.8, B=1),
        # 16 tempered chains stepped together on the same analysis
        dict(name="full-fp64-16-4s", kind="full", prec="fp64", io="host", nifo=2, Tobs=4.0, fs=2048.0, fmin=16.0,
             mt=65.0, q=0.8, B=16),
        # 64 chains x 32 proposals of a 16 s, three-detector analysis in the plain precision
        dict(name="full-fp64-2048-16s", kind="full", prec="fp64", io="dev", nifo=3, Tobs=16.0, fs=4096.0, fmin=20.0,
             mt=55.0, q=0.83, B=2048),
        # the same in mixed precision: the headline workload
        dict(name="full-mixed-2048-16s", kind="full", prec="mixed", io="dev", nifo=3, Tobs=16.0, fs=4096.0, fmin=20.0,
             mt=55.0, q=0.83, B=2048),
        # full likelihood of a long low-mass signal (burn-in, and checks of the heterodyned form); ragged count
        dict(name="full-fp64-201-128s", kind="full", prec="fp64", io="host", nifo=3, Tobs=128.0, fs=4096.0, fmin=20.0,
             mt=2.75, q=0.9, B=201),
        # the sampler's production call: one heterodyned set from a host thread
        dict(name="het-fp64-1-128s", kind="het", prec="fp64", io="host", nifo=3, Tobs=128.0, fs=4096.0, fmin=20.0,
             mt=2.75, q=0.9, B=1, M=47),
        # the batched heterodyned step, in both precisions
        dict(name="het-fp64-4096-128s", kind="het", prec="fp64", io="dev", nifo=3, Tobs=128.0, fs=4096.0, fmin=20.0,
             mt=2.75, q=0.9, B=4096, M=47),
        dict(name="het-mixed-1000-32s", kind="het", prec="mixed", io="host", nifo=2, Tobs=32.0, fs=2048.0, fmin=20.0,
             mt=8.0, q=0.6, B=1000, M=49),
        # the service's merged step over uneven live analyses (grouped by event), FP64
        dict(name="multi-fp64-24x64", kind="multi", prec="fp64", io="host", n_events=24, sets=64),
        # heterodyne tables of the long signal on the search's typical grid
        dict(name="tables-128s", kind="tables", nifo=3, Tobs=128.0, fs=4096.0, fmin=20.0, mt=2.75, q=0.9, M=47),
        # admission of a long analysis: the grid search
        dict(name="grid-128s", kind="grid", nifo=3, Tobs=128.0, fs=4096.0, fmin=16.0, mt=2.75, q=0.9),
        # noise marginalisation on the long analysis: PSD draw, rebuilt weights and tables, 12 chains
        dict(name="redraw-128s", kind="redraw", prec="fp64", nifo=3, Tobs=128.0, fs=4096.0, fmin=20.0, mt=2.75, q=0.9,
             B=12, M=47),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


# total masses whose signal from 20 Hz fits a segment (Newtonian chirp time, as for the listed ones)
_MASSES = {4.0: (50.0, 90.0), 8.0: (24.0, 60.0), 16.0: (14.0, 60.0), 32.0: (8.0, 14.0), 64.0: (4.5, 7.0), 128.0: (2.4, 3.6)}


def draw(rng):
    kind = rng.choice(["full", "full", "full", "het", "het", "multi", "tables", "grid", "redraw"])
    if kind == "multi":
        n = rng.randint(3, 32)
        return dict(kind=kind, prec=rng.choice(["fp64", "mixed"]), io=rng.choice(["host", "dev"]), n_events=n,
                    sets=rng.randint(1, 1536 // n))
    Tobs = rng.choice([4.0, 8.0, 16.0, 32.0, 64.0, 128.0] if kind != "grid" else [4.0, 8.0, 16.0, 32.0, 128.0])
    c = dict(kind=kind, nifo=rng.randint(1, 3), Tobs=Tobs, fs=rng.choice([2048.0, 4096.0]),
             fmin=rng.choice([16.0, 20.0]) if kind != "grid" else 16.0, mt=round(rng.uniform(*_MASSES[Tobs]), 3),
             q=round(rng.uniform(0.4, 1.0), 3))
    if kind in ("full", "het", "redraw"):
        c["prec"] = rng.choice(["fp64", "mixed"])
    if kind == "full":
        c["io"] = rng.choice(["host", "dev"])
        bins = c["nifo"] * Tobs * (1024.0 - c["fmin"])
        c["B"] = int(round(_log_uniform(rng, 1.0, min(2048.0, 2048.0 * 48192.0 / bins))))
    if kind == "het":
        c["io"] = rng.choice(["host", "dev"])
        c["B"] = int(round(_log_uniform(rng, 1.0, 4096.0)))
    if kind == "redraw":
        c["B"] = rng.randint(1, 16)
    if kind in ("het", "tables", "redraw"):
        c["M"] = 2 * rng.randint(18, 32) + 1
    return c


# ------------------------------------------------------------------ inputs, from the seed alone
def _band(c):
    N = int(round(c["Tobs"] * c["fs"]))
    return N, int(c["Tobs"] * c["fmin"]), min(int(c["Tobs"] * 1024.0), N // 2)


def _het_grid(c):
    """A geometric grid of M bins over the band the signal reaches (below the model's cut-off)."""
    N, lo, hi = _band(c)
    hi = min(hi - 1, int(0.15 / (c["mt"] * 4.925491e-6) * c["Tobs"]))
    M = int(c["M"])
    g = np.round(np.geomspace(lo, hi, M)).astype(np.int64)
    for k in range(1, M):                      # strictly increasing at the low end
        g[k] = max(g[k], g[k - 1] + 1)
    return g.astype(np.int32), int(lo), int(g[-1])


def _event_inputs(c, seed):
    """Network, noise, one injected signal scaled to SNR 20-30, PSD: tensors on the device."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    nifo, Tobs = int(c["nifo"]), float(c["Tobs"])
    labels = [int(x) for x in c["labels"]] if isinstance(c.get("labels"), (list, tuple)) else list(range(nifo))
    N, lo, hi = _band(c)
    nh = N // 2
    GMST = float(rng.uniform(0, 2 * np.pi))
    p = np.zeros(11)
    m2 = c["mt"] * c["q"] / (1 + c["q"])
    p[0], p[1] = synth.masses_to_params(c["mt"] - m2, m2)
    lim = 0.05 if c["mt"] < 4.0 else 0.4
    p[2:4] = rng.uniform(-lim, lim, size=2)
    p[5] = Tobs - 2.0
    p[6] = np.log(400e6 * PC)
    synth.random_extrinsic(rng, p)
    p[8], p[10] = 0.9 * p[8], 0.9 * p[10]      # room for the chains' jitter
    i = torch.arange(nh, device=DEV, dtype=torch.float64)
    f = i / Tobs
    f[0] = 1.0 / Tobs
    fs = torch.cat([f, torch.tensor([nh / Tobs], device=DEV, dtype=torch.float64)])
    x = fs / 215.0
    S = 1e-49 * (x ** -4.14 - 5.0 / x ** 2 + 111.0 * (1.0 - x ** 2 + 0.5 * x ** 4) / (1.0 + 0.5 * x ** 2))
    SN = S.expand(nifo, nh + 1).contiguous()
    ev = dict(labels=labels, GMST=GMST, Tobs=Tobs, N=N, lo=lo, hi=hi, SN=SN, f=f, fmin=float(c["fmin"]))

    def template(par):
        w = _Wave(torch.from_numpy(par[None, :]).to(DEV), ev)
        A, ph = w.projected(f[1:], taper=False)
        return A[0], ph[0]
    A, ph = template(p)
    s2 = float((4.0 * A[:, lo - 1:hi - 1] ** 2 / SN[:, lo:hi]).sum())
    snr = float(c.get("snr", 20.0 if c["mt"] > 10 else 30.0))
    p[6] += np.log(np.sqrt(s2) / snr)
    A, ph = template(p)
    D = torch.zeros(nifo, N, device=DEV, dtype=torch.float64)
    noise = torch.randn(2, nifo, nh - 1, device=DEV, dtype=torch.float64, generator=gen) * torch.sqrt(SN[:, 1:nh] / 4.0)
    D[:, 1:nh] = noise[0] + A * torch.cos(ph)
    D[:, nh + 1:] = (noise[1] + A * torch.sin(ph)).flip(1)
    return dict(ev, D=D, inj=p), rng


def _chains(c, inj, rng, B):
    """Chains about the peak, at the posterior's width: a few tenths of a radian over the band."""
    mc = math.exp(inj[0]) / MSUN * 4.925491e-6
    dmc = 0.15 / (3.0 / 128.0 * (math.pi * mc * 20.0) ** (-5.0 / 3.0))
    sig = np.array([dmc, 10 * dmc, 0.005, 0.005, 0.3, 1e-4, 0.1, 0.02, 0.02, 0.3, 0.05])
    P = inj[None, :] + sig * rng.normal(size=(B, 11))
    P[:, 8], P[:, 10] = np.clip(P[:, 8], -1, 1), np.clip(P[:, 10], -1, 1)
    P[:, 0] = np.minimum(P[:, 0], P[:, 1] + 0.6 * np.log(0.25) - 1e-9)
    return P


def _proposals(c, inj, rng, B):
    """Proposals of a full-likelihood run: wide (masses, spins, sky) for heavy systems, as the batched
    workload draws them; about the peak for neutron stars."""
    if c["mt"] < 14.0:
        return _chains(c, inj, rng, B)
    mc = math.exp(inj[0]) / MSUN
    return synth.draw_params(rng, B, inj, mc=(0.5 * mc, 1.4 * mc))


def _multi_inputs(c, seed):
    evs, P, eo = [], [], []
    for e, s in enumerate(synth.uneven_event_specs(int(c["n_events"]), seed=int(seed) * 64)):
        ce = dict(nifo=len(s["labels"]), labels=s["labels"], Tobs=s["Tobs"], fs=s["fs"], fmin=s["fmin"],
                  mt=s["m1"] + s["m2"], q=s["m2"] / s["m1"], snr=s["snr"])
        ev, rng = _event_inputs(ce, int(seed) * 64 + e)
        evs.append(ev)
        P.append(_proposals(ce, ev["inj"], rng, int(c["sets"])) if e % 2 else _chains(ce, ev["inj"], rng, int(c["sets"])))
        eo.append(np.full(int(c["sets"]), e, dtype=np.int32))
    return evs, np.concatenate(eo), np.ascontiguousarray(np.vstack(P))


def _open(ev):
    return q.Event(ev["labels"], ev["Tobs"], ev["GMST"], ev["N"], ev["D"].cpu().numpy(), ev["SN"].cpu().numpy(),
                   fmin=ev["fmin"])


def _inputs(c, seed):
    """(event inputs, parameter sets, PSD model arrays) of a one-event case."""
    ev, rng = _event_inputs(c, seed)
    P = model = None
    if c["kind"] == "full":
        P = _proposals(c, ev["inj"], rng, int(c["B"]))
    elif "B" in c:
        P = _chains(c, ev["inj"], rng, int(c["B"]))
    if c["kind"] == "redraw":
        model = synth.psd_model_arrays(rng, int(c["nifo"]), ev["Tobs"], ev["N"], nsample=2)
    return ev, P, model


def _prior(Tobs):
    """MCMC_all's prior box (QuickCBC.c:1871-1896, ConstCBC.h:48-57)."""
    lo = np.array([np.log(0.5 * MSUN), np.log(0.5 * MSUN), -0.85, -0.85, 0.0, max(Tobs - 3.5, 1.5), np.log(1e6 * PC),
                   0.0, -1.0, 0.0, -1.0])
    hi = np.array([np.log(160 * MSUN), np.log(300 * MSUN), 0.85, 0.85, 2 * np.pi, Tobs - 0.5, np.log(1e10 * PC),
                   2 * np.pi, 1.0, np.pi, 1.0])
    return lo, hi


@functools.lru_cache(None)
def _stream():
    """The program's stream: every device-form call of this process is ordered on it."""
    return torch.cuda.Stream()


def _device_state(st, P, nifo=None):
    st["d_params"] = torch.from_numpy(np.ascontiguousarray(P)).to(DEV)
    st["d_lnl"] = torch.zeros(len(P), device=DEV, dtype=torch.float64)
    if nifo:
        st["d_rho"] = torch.zeros(len(P), nifo, device=DEV, dtype=torch.float64)
    st["stream"] = ctypes.c_void_p(_stream().cuda_stream)


def prepare(case, seed):
    c = case
    st = dict(kind=c["kind"], io=c.get("io", "host"), prec=q.MIXED if c.get("prec") == "mixed" else q.FP64)
    if c["kind"] == "multi":
        evs, eo, P = _multi_inputs(c, seed)
        st["events"] = [_open(e) for e in evs]
        st["batch"] = q.Batch(st["events"])
        st["eo"], st["P"] = eo, P
        if st["io"] == "dev":
            _device_state(st, P)
            st["d_eo"] = torch.from_numpy(eo).to(DEV)
        return st
    ev, P, model = _inputs(c, seed)
    st["ev"] = _open(ev)
    st["P"] = P
    if c["kind"] in ("het", "redraw"):
        st["ev"].het_setup(ev["inj"], *_het_grid(c), 2)
    if c["kind"] == "tables":
        st["pref"], st["grid"] = ev["inj"], _het_grid(c)
    if c["kind"] == "grid":
        st["pref"], st["prior"] = ev["inj"], _prior(ev["Tobs"])
    if c["kind"] == "redraw":
        ns, nl, ffit, xs, lines = model
        st["model"] = ingest.PsdModel(ffit, xs, lines, nspline=ns, nlines=nl)
    if st["io"] == "dev":
        _device_state(st, P, nifo=int(c["nifo"]))
    return st


def run(state):
    s, kind = state, state["kind"]
    if kind == "full":
        if s["io"] == "host":
            return s["ev"].lnl_full(s["P"], s["prec"], rho=True)
        check(lib().qcbc_lnl_full_dev(s["ev"].handle, s["d_params"].data_ptr(), len(s["P"]), s["d_lnl"].data_ptr(),
                                      s["d_rho"].data_ptr(), s["prec"], s["stream"]))
        return s["d_lnl"], s["d_rho"]
    if kind == "het":
        if s["io"] == "host":
            return s["ev"].lnl_het(s["P"], s["prec"])
        check(lib().qcbc_lnl_het_dev(s["ev"].handle, s["d_params"].data_ptr(), len(s["P"]), s["d_lnl"].data_ptr(),
                                     s["prec"], s["stream"]))
        return s["d_lnl"]
    if kind == "multi":
        if s["io"] == "host":
            return s["batch"].lnl(s["eo"], s["P"], s["prec"])
        vp = ctypes.c_void_p
        check(lib().qcbc_lnl_multi_dev(vp(s["batch"]._h), vp(s["d_eo"].data_ptr()), vp(s["d_params"].data_ptr()),
                                       len(s["P"]), vp(s["d_lnl"].data_ptr()), s["prec"], s["stream"]))
        return s["d_lnl"]
    if kind == "tables":
        s["ev"].het_setup(s["pref"], *s["grid"], 2)
        return s["ev"].het_export()
    if kind == "grid":
        g, MN, MM = s["ev"].het_space(s["pref"], *s["prior"])
        out = np.full(256, -1, dtype=np.int32)     # the grid's length depends on the signal (about 50 bins)
        out[:len(g)] = g
        return out, len(g), MN, MM
    s["ev"].set_psd_sample(s["model"], 1)
    return s["ev"].lnl_het(s["P"], s["prec"]), s["ev"].lnl_full(s["P"], s["prec"])


# ------------------------------------------------------------------ what a pass cannot do without
def _full_work(nifo, bins, B, word):
    # per set and bin: 60 operations of the IMRPhenomD point, 14 per detector for the projection and
    # the two products; the weighted data (3 words per detector-bin) are read once
    return 3.0 * nifo * bins * word + B * (11 + 1 + nifo) * 8.0, B * bins * (60.0 + 14.0 * nifo)


def work(case):
    c = case
    word = 4.0 if c.get("prec") == "mixed" else 8.0
    if c["kind"] == "multi":
        by = fl = 0.0
        per = int(c["sets"])
        for _ in range(int(c["n_events"])):        # an event of the mix: two detectors, 16 s, 1004 Hz of band
            b, f = _full_work(2, 16.0 * 1004.0, per, word)
            by, fl = by + b, fl + f
        return dict(bytes=by, flops=fl)
    N, lo, hi = _band(c)
    nifo, bins = int(c["nifo"]), hi - lo
    if c["kind"] == "full":
        by, fl = _full_work(nifo, bins, int(c["B"]), word)
        return dict(bytes=by, flops=fl)
    if c["kind"] == "het":
        M, B = int(c["M"]), int(c["B"])
        # per set and grid point: the waveform, the projection, and half a region's 3 x 3 contractions of 3 vectors
        return dict(bytes=8.0 * (2 * nifo * M + M // 2 * (9 + 12 * nifo)) + B * 12 * 8.0,
                    flops=B * M * (60.0 + nifo * (14.0 + 36.0)))
    nh = N // 2
    tables = (8.0 * 3 * nifo * nh, nh * (60.0 + nifo * 50.0))     # D and S read once; template, weights, Legendre sums
    if c["kind"] == "tables":
        return dict(bytes=tables[0], flops=tables[1])
    if c["kind"] == "grid":
        # 23 waveforms for the Fisher matrix, one per direction and trial of the scaling (about 11 x 8), 11
        # for the grid's ratios; the PSD read once
        return dict(bytes=8.0 * nifo * nh, flops=bins * (23 + 88 + 11) * (60.0 + 14.0 * nifo))
    # redraw: PSD written and read, weights written, tables, then the chains' two likelihoods
    by, fl = _full_work(nifo, bins, int(c["B"]), word)
    return dict(bytes=by + tables[0] + 8.0 * nifo * nh * (1 + 3) + 4.0 * 3 * nifo * nh,
                flops=fl + tables[1] + nifo * nh * 40.0)


# ------------------------------------------------------------------ the same in 64 bits, by the published model
# Table V of arXiv:1508.07253: lambda = l00 + l10 eta + (l01 + l11 eta + l21 eta^2) xi + (...) xi^2 + (...) xi^3
_FITS = {
    "r1": [
        3931.8979897196696, -17395.758706812805, 3132.375545898835, 343965.86092361377, -1216256.5819981997,
        -70698.00600428853, 1383907.177859705, -3966276.1890979446, -60017.52423652596, 803515.1181825735,
        -2091710.365941658],
    "r2": [
        -40105.47653771657, 112253.0169706701, 23561.696065836168, -3476180.699403351, 11375936.70849482,
        754313.1127166454, -13084760.44625268, 36444584.853928134, 596226.612472288, -7427790.1143564405,
        18928977.514040343],
    "r3": [
        83208.35471266537, -191237.7264145924, -210916.2454782992, 8717975.08352568, -26914942.420669552,
        -1988980.6527362722, 30888029.960154563, -83908702.79256162, -1453503.1953446497, 17063528.990822166,
        -42748659.731120914],
    "g1": [
        0.006927402739328343, 0.03020474290328911, 0.006308024337706171, -0.12074130661131138, 0.26271598905781324,
        0.0034151773647198794, -0.10779338611188374, 0.27098966966891747, 0.0007374185938559283,
        -0.02749621038376281, 0.0733150789135702],
    "g2": [
        1.010344404799477, 0.0008993122007234548, 0.283949116804459, -4.049752962958005, 13.207828172665366,
        0.10396278486805426, -7.025059158961947, 24.784892370130475, 0.03093202475605892, -2.6924023896851663,
        9.609374464684983],
    "g3": [
        1.3081615607036106, -0.005537729694807678, -0.06782917938621007, -0.6689834970767117, 3.403147966134083,
        -0.05296577374411866, -0.9923793203111362, 4.820681208409587, -0.006134139870393713, -0.38429253308696365,
        1.7561754421985984],
    "v2": [
        0.8149838730507785, 2.5747553517454658, 1.1610198035496786, -2.3627771785551537, 6.771038707057573,
        0.7570782938606834, -2.7256896890432474, 7.1140380397149965, 0.1766934149293479, -0.7978690983168183,
        2.1162391502005153],
    "a1": [
        43.31514709695348, 638.6332679188081, -32.85768747216059, 2415.8938269370315, -5766.875169379177,
        -61.85459307173841, 2953.967762459948, -8986.29057591497, -21.571435779762044, 981.2158224673428,
        -3239.5664895930286],
    "a2": [
        -0.07020209449091723, -0.16269798450687084, -0.1872514685185499, 1.138313650449945, -2.8334196304430046,
        -0.17137955686840617, 1.7197549338119527, -4.539717148261272, -0.049983437357548705, 0.6062072055948309,
        -1.682769616644546],
    "a3": [
        9.5988072383479, -397.05438595557433, 16.202126189517813, -1574.8286986717037, 3600.3410843831093,
        27.092429659075467, -1786.482357315139, 5152.919378666511, 11.175710130033895, -577.7999423177481,
        1808.730762932043],
    "a4": [
        -0.02989487384493607, 1.4022106448583738, -0.07356049468633846, 0.8337006542278661, 0.2240008282397391,
        -0.055202870001177226, 0.5667186343606578, 0.7186931973380503, -0.015507437354325743, 0.15750322779277187,
        0.21076815715176228],
    "a5": [
        0.9974408278363099, -0.007884449714907203, -0.059046901195591035, 1.3958712396764088, -4.516631601676276,
        -0.05585343136869692, 1.7516580039343603, -5.990208965347804, -0.017945336522161195, 0.5965097794825992,
        -2.0608879367971804],
    "b1": [
        97.89747327985583, -42.659730877489224, 153.48421037904913, -1417.0620760768954, 2752.8614143665027,
        138.7406469558649, -1433.6585075135881, 2857.7418952430758, 41.025109467376126, -423.680737974639,
        850.3594335657173],
    "b2": [
        -3.282701958759534, -9.051384468245866, -12.415449742258042, 55.4716447709787, -106.05109938966335,
        -11.953044553690658, 76.80704618365418, -155.33172948098394, -3.4129261592393263, 25.572377569952536,
        -54.408036707740465],
    "b3": [
        -2.5156429818799565e-05, 1.9750256942201327e-05, -1.8370671469295915e-05, 2.1886317041311973e-05,
        8.250240316860033e-05, 7.157371250566708e-06, -5.5780000112270685e-05, 0.00019142082884072178,
        5.447166261464217e-06, -3.220610095021982e-05, 7.974016714984341e-05],
    "s1": [
        2096.551999295543, 1463.7493168261553, 1312.5493286098522, 18307.330017082117, -43534.1440746107,
        -833.2889543511114, 32047.31997183187, -108609.45037520859, 452.25136398112204, 8353.439546391714,
        -44531.3250037322],
    "s2": [
        -10114.056472621156, -44631.01109458185, -6541.308761668722, -266959.23419307504, 686328.3229317984,
        3405.6372187679685, -437507.7208209015, 1631817.1307344697, -7462.648563007646, -114585.25177153319,
        674402.4689098676],
    "s3": [
        22933.658273436497, 230960.00814979506, 14961.083974183695, 1194018.1342318142, -3104223.9693052764,
        -3038.166617199259, 1872032.2849093592, -7309145.012085539, 42738.22871475411, 467502.018616601,
        -3064853.498512499],
    "s4": [
        -14621.71522218357, -377812.8579387104, -9608.682631509726, -1710892.5257214056, 4332924.601416521,
        -22366.683262266528, -2501971.6386377467, 10274495.902259542, -85360.30079034246, -570025.3441737515,
        4396844.346849777],
}

# F+ / Fx of H1, L1, V1 with the reference's coefficients (Utilities.c:1004-1076) over the monomials below
_ANT_P = [
    [
        0.3104536562, 0.494778091, 1.424276331, -0.4559956644, -0.1552268274, 0.3104536562, -0.1552268276,
        -0.4928680677, 1.424276334, 0.3104536558, -0.9119913289, -0.9314082637, -0.712138166, 0.9119913288,
        -0.6209073089, 2.848552667, -0.9895561804, 0.2464340337, -0.9895561811, -0.7121381653, 0.4657041323],
    [
        -0.5608410611, -0.4945891833, -1.040573095, 0.363231261, 0.2804205304, -0.5608410611, 0.2804205305,
        -0.3865389475, -1.040573095, -0.5608410611, 0.7264625218, 1.427112041, 0.5202865467, -0.7264625224,
        1.121682123, -2.081146187, 0.9891783667, 0.1932694762, 0.9891783666, 0.5202865474, -0.7135560209],
    [
        0.3963351156, 0.465152434, -1.383399753, -0.3756662059, -0.1981675579, 0.3963351153, -0.1981675578,
        1.303555289, -1.383399752, 0.3963351158, -0.7513324118, 0.0798444642, 0.6916998761, 0.7513324118,
        -0.792670233, -2.766799504, -0.9303048681, -0.6517776444, -0.9303048681, 0.6916998765, -0.039922232],
]
_ANT_X = [
    [
        -1.424276332, -0.3104536551, -0.6209073087, -0.989556182, 0.3104536561, 0.9895561812, -1.424276332,
        -0.9119913298, 2.848552668, -0.911991329, 0.9314082638, -1.424276333, -0.1552268276, 0.3104536564,
        0.4947780906, -0.3104536556, 0.4928680679, 0.4559956636],
    [
        1.040573095, 0.5608410611, 1.121682122, 0.9891783668, -0.5608410611, -0.9891783668, 1.040573095,
        0.7264625222, -2.081146187, 0.7264625218, -1.427112042, 1.040573094, 0.2804205304, -0.560841061,
        -0.4945891833, 0.5608410611, 0.3865389466, -0.3632312614],
    [
        1.383399753, -0.396335116, -0.7926702326, -0.9303048681, 0.3963351158, 0.9303048686, 1.383399752,
        -0.7513324118, -2.766799505, -0.7513324118, -0.0798444646, 1.383399752, -0.1981675579, 0.3963351158,
        0.465152434, -0.3963351158, -1.303555288, 0.3756662059],
]
# exponents of cos psi, sin psi, cos delta, sin delta, cos(alpha - GMST), sin(alpha - GMST)
_MONO_P = [
    (2, 0, 0, 0, 1, 1), (0, 0, 1, 1, 1, 0), (2, 0, 0, 2, 2, 0), (0, 0, 1, 1, 0, 1), (0, 0, 0, 2, 1, 1),
    (1, 1, 0, 1, 0, 0), (0, 0, 0, 0, 1, 1), (2, 0, 0, 2, 0, 0), (2, 0, 0, 0, 2, 0), (2, 0, 0, 2, 1, 1),
    (1, 1, 1, 0, 1, 0), (2, 0, 0, 0, 0, 0), (0, 0, 0, 0, 2, 0), (2, 0, 1, 1, 0, 1), (1, 1, 0, 1, 2, 0),
    (1, 1, 0, 1, 1, 1), (2, 0, 1, 1, 1, 0), (0, 0, 0, 2, 0, 0), (1, 1, 1, 0, 0, 1), (0, 0, 0, 2, 2, 0),
    (0, 0, 0, 0, 0, 0)]
_MONO_X = [
    (1, 1, 0, 2, 2, 0), (1, 1, 0, 0, 1, 1), (2, 0, 0, 1, 2, 0), (2, 0, 1, 0, 0, 1), (0, 0, 0, 1, 2, 0),
    (1, 1, 1, 1, 1, 0), (0, 0, 0, 1, 1, 1), (2, 0, 1, 0, 1, 0), (2, 0, 0, 1, 1, 1), (1, 1, 1, 1, 0, 1),
    (1, 1, 0, 0, 0, 0), (1, 1, 0, 0, 2, 0), (0, 0, 0, 1, 0, 0), (2, 0, 0, 1, 0, 0), (0, 0, 1, 0, 0, 1),
    (1, 1, 0, 2, 1, 1), (1, 1, 0, 2, 0, 0), (0, 0, 1, 0, 1, 0)]
_DET = [[-2.161414928e6, 3.834695183e6, 4.600350224e6], [-74276.04192, 5.496283721e6, 3.224257016e6],
        [4546374.098, -842989.6972, 4378576.963]]


@functools.lru_cache(None)
def _qnm():
    """(spin, fring, fdamp, second derivatives) of the l = m = 2, n = 0 Kerr mode: Leaver's continued
    fractions (Proc. R. Soc. A 402, 285), at spins 0.002 apart, six significant digits as published."""
    spins = np.arange(-150, 496) * 2 / 1000.0
    s, m = -2.0, 2.0
    a = spins / 2.0

    def angular(c, A):
        def be(p):
            return p * (p - 1) + 2 * p * (3 - 2 * c) - (2 * c * 3 - 6) - (c * c + 2 + A)
        r = 0.0 * c
        for p in range(30, 0, -1):
            r = (-2 * p * (p + 4)) * (2 * c * p) / (be(p) - r)
        return be(0) - r

    def separation(c, A):
        for _ in range(8):
            f, h = angular(c, A), 1e-6
            A = A - f * 2 * h / (angular(c, A + h) - angular(c, A - h))
        return A

    def radial(w, A, n_max=600):
        b = np.sqrt(1 - 4 * a * a + 0j)
        x = (w / 2 - a * m) / b
        c0 = 1 - s - 1j * w - 2j * x
        c1 = -4 + 2j * w * (2 + b) + 4j * x
        c2 = s + 3 - 3j * w - 2j * x
        c3 = w * w * (4 + 2 * b - a * a) - 2 * a * m * w - s - 1 + (2 + b) * 1j * w - A + (4 * w + 2j) * x
        c4 = s + 1 - 2 * w * w - (2 * s + 3) * 1j * w - (4 * w + 2j) * x
        root = np.sqrt(-2j * w * b)
        D = -(1 - np.where(root.real > 0, root, -root) / np.sqrt(n_max))
        for n in range(n_max, -1, -1):
            al, be = n * n + (c0 + 1) * n + c0, -2 * n * n + (c1 + 2) * n + c3
            if n == 0:
                return be - al * D
            D = (n * n + (c2 - 3) * n + c4 - c2 + 2) / (be - al * D)

    j = spins
    wr = 1.5251 - 1.1568 * (1 - j) ** 0.1292
    w = 2 * wr * (1 - 0.5j / (0.7 + 1.4187 * (1 - j) ** -0.4990))
    A = np.full(len(a), 4.0 + 0j)
    for k in range(1, 9):
        A = separation(a * w * k / 8, A)
    for _ in range(8):
        h = 1e-6
        f = radial(w, A)
        d = (radial(w + h, separation(a * (w + h), A)) - radial(w - h, separation(a * (w - h), A))) / (2 * h)
        w = w - f / d
        A = separation(a * w, A)
    out = [spins]
    for y in (w.real / 2 / (2 * np.pi), -w.imag / 2 / (2 * np.pi)):
        out.append(np.array([float("%.6g" % v) for v in y]))
    out += [_natural_spline(spins, y) for y in out[1:]]
    return [torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for v in out]


def _natural_spline(x, y):
    """Second derivatives of the natural cubic spline."""
    n, h = len(x), np.diff(x)
    T = np.zeros((n, n))
    r = np.zeros(n)
    T[0, 0] = T[-1, -1] = 1.0
    k = np.arange(1, n - 1)
    T[k, k - 1], T[k, k], T[k, k + 1] = h[:-1], 2 * (h[:-1] + h[1:]), h[1:]
    r[1:-1] = 6 * (np.diff(y[1:]) / h[1:] - np.diff(y[:-1]) / h[:-1])
    return np.linalg.solve(T, r)


def _spline(x, y, m2, v):
    lo = torch.clamp(torch.searchsorted(x, v.contiguous(), right=True) - 1, 0, len(x) - 2)
    h, dx = x[lo + 1] - x[lo], v - x[lo]
    b = (y[lo + 1] - y[lo]) / h - h * (2 * m2[lo] + m2[lo + 1]) / 6.0
    return y[lo] + dx * (b + dx * (0.5 * m2[lo] + dx * (m2[lo + 1] - m2[lo]) / (6.0 * h)))


class _Wave:
    """IMRPhenomD and its projection on the network for parameter sets P [B, 11] ([B, 1] per coefficient)."""
    GAMMA = 0.577215664901532860606512090082402431

    def __init__(self, P, ev):
        col = [P[:, k:k + 1] for k in range(11)]
        pi, mtsun = math.pi, 4.925491025543575903411922162094833998e-6
        self.ev = ev
        mc, mt = torch.exp(col[0]), torch.exp(col[1])
        eta = (mc / mt) ** (5.0 / 3.0)
        dm = torch.where(eta > 0.25, torch.zeros_like(eta), torch.sqrt(torch.clamp(1.0 - 4.0 * eta, min=0.0)))
        m1, m2 = mt * (1 + dm) / 2 / MSUN, mt * (1 - dm) / 2 / MSUN
        x1, x2 = col[2], col[3]
        swap = ~(m1 > m2)
        m1, m2 = torch.where(swap, m2, m1), torch.where(swap, m1, m2)
        x1, x2 = torch.where(swap, x2, x1), torch.where(swap, x1, x2)
        phi0, self.ts, dist = 0.5 * col[4], ev["Tobs"] - col[5], torch.exp(col[6])
        M = m1 + m2
        eta = m1 * m2 / (M * M)
        self.eta, self.Msec = eta, M * mtsun
        self.scale = M * 1.476625061404649406193430731479084713e3 * M * mtsun / dist
        e2, e3, e4 = eta ** 2, eta ** 3, eta ** 4
        S = torch.sqrt(torch.clamp(1.0 - 4.0 * eta, min=0.0))
        a1, a2 = 0.5 * (1 + S), 0.5 * (1 - S)
        chi = (x1 + x2) / 2.0 * (1.0 - eta * 76.0 / 113.0) + S * ((x1 - x2) / 2.0)
        s = a1 ** 2 * x1 + a2 ** 2 * x2
        spin = (3.4641016151377544 * eta - 4.399247300629289 * e2 + 9.397292189321194 * e3 - 13.180949901606242 * e4 +
                (1 - 0.0850917821418767 * eta - 5.837029316602263 * e2) * s +
                (0.1014665242971878 * eta - 2.0967746996832157 * e2) * s ** 2 +
                (-1.3546806617824356 * eta + 4.108962025369336 * e2) * s ** 3 +
                (-0.8676969352555539 * eta + 2.064046835273906 * e2) * s ** 4)
        sr = s / (a1 ** 2 + a2 ** 2)
        erad = ((0.055974469826360077 * eta + 0.5809510763115132 * e2 - 0.9606726679372312 * e3 + 3.352411249771192 * e4) *
                (1 + (-0.0030302335878845507 - 2.0066110851351073 * eta + 7.7050567802399215 * e2) * sr)) / \
            (1 + (-0.6714403054720589 - 1.4756929437702908 * eta + 7.304676214885011 * e2) * sr)
        x, yr, yd, mr, md = _qnm()
        self.fRD = _spline(x, yr, mr, spin) / (1 - erad)
        self.fDM = _spline(x, yd, md, spin) / (1 - erad)
        xi = chi - 1.0

        def fit(name):
            c = _FITS[name]
            return (c[0] + c[1] * eta + (c[2] + c[3] * eta + c[4] * e2) * xi +
                    (c[5] + c[6] * eta + c[7] * e2) * xi ** 2 + (c[8] + c[9] * eta + c[10] * e2) * xi ** 3)
        self.g = [fit("g1"), fit("g2"), fit("g3")]
        g1, g2, g3 = self.g
        root = torch.sqrt(torch.clamp(1 - g2 * g2, min=0.0))
        self.fmax = torch.abs(self.fRD + torch.where(g2 <= 1, self.fDM * (root - 1) * g3 / g2, -self.fDM * g3 / g2))
        self.a0 = math.sqrt(2.0 / 3.0) * torch.sqrt(eta) / pi ** (1 / 6.0)
        x1s, x2s, Pi2 = x1 * x1, x2 * x2, pi * pi
        self.ai = [
            (-969 + 1804 * eta) * pi ** (2 / 3.0) / 672.0,
            (x1 * (81 * (1 + S) - 44 * eta) + x2 * (81 - 81 * S - 44 * eta)) * pi / 48.0,
            (-27312085.0 - 10287648 * x2s - 10287648 * x1s * (1 + S) + 10287648 * x2s * S +
             24 * (-1975055 + 857304 * x1s - 994896 * x1 * x2 + 857304 * x2s) * eta + 35371056 * e2) *
            pi ** (4 / 3.0) / 8.128512e6,
            pi ** (5 / 3.0) * (x2 * (-285197 * (-1 + S) + 4 * (-91902 + 1579 * S) * eta - 35632 * e2) +
                               x1 * (285197 * (1 + S) - 4 * (91902 + 1579 * S) * eta - 35632 * e2) +
                               42840 * (-1.0 + 4 * eta) * pi) / 32256.0,
            -(Pi2 * (-336 * (-3248849057.0 + 2943675504 * x1s - 3339284256 * x1 * x2 + 2943675504 * x2s) * e2 -
                     324322727232 * e3 -
                     7 * (-177520268561 + 107414046432 * x2s + 107414046432 * x1s * (1 + S) - 107414046432 * x2s * S +
                          11087290368 * (x1 + x2 + x1 * S - x2 * S) * pi) +
                     12 * eta * (-545384828789 - 176491177632 * x1 * x2 + 202603761360 * x2s +
                                 77616 * x1s * (2610335 + 995766 * S) - 77287373856 * x2s * S +
                                 5841690624 * (x1 + x2) * pi + 21384760320 * Pi2))) / 6.0085960704e10,
            fit("r1"), fit("r2"), fit("r3")]
        # intermediate amplitude: the quartic through value and slope at f1 and f3 and the value at f2
        f1, f3 = torch.full_like(eta, 0.014), self.fmax
        f2 = f1 + (f3 - f1) / 2.0
        v1, v2, v3 = self.amp_ins(f1), fit("v2"), self.amp_mrd(f3)
        ai = self.ai
        d1 = (2 / 3.0 * ai[0] * f1 ** (-1 / 3.0) + ai[1] + 4 / 3.0 * ai[2] * f1 ** (1 / 3.0) + 5 / 3.0 * ai[3] * f1 ** (2 / 3.0) +
              2 * ai[4] * f1 + 7 / 3.0 * ai[5] * f1 ** (4 / 3.0) + 8 / 3.0 * ai[6] * f1 ** (5 / 3.0) + 3 * ai[7] * f1 ** 2)
        fg = self.fDM * g3
        d2 = v3 * (-g2 / fg - 2.0 * (f3 - self.fRD) / ((f3 - self.fRD) ** 2 + fg ** 2))
        q12, q23 = (v2 - v1) / (f2 - f1), (v3 - v2) / (f3 - f2)
        r0, r1, r2 = (q12 - d1) / (f2 - f1), (q23 - q12) / (f3 - f1), (d2 - q23) / (f3 - f2)
        t0, t1 = (r1 - r0) / (f3 - f1), (r2 - r1) / (f3 - f1)
        self.nodes, self.newton = (f1, f2, f3), (v1, d1, r0, t0, (t1 - t0) / (f3 - f1))
        # TaylorF2 (arXiv:1508.07253 eq. 27) with its aligned-spin terms
        d, m1M, m2M = (m1 - m2) / M, m1 / M, m2 / M
        SL, dS = m1M ** 2 * x1 + m2M ** 2 * x2, d * (m2M * x2 - m1M * x1)
        pf = 3.0 / (128.0 * eta)
        sigma = eta * (721.0 / 48.0 - 247.0 / 48.0) * x1 * x2 + ((719.0 - 233.0) / 96.0) * (m1M ** 2 * x1s + m2M ** 2 * x2s)
        ss3 = (326.75 / 1.12 + 557.5 / 1.8 * eta) * eta * x1 * x2
        for mm, xs in ((m1M, x1s), (m2M, x2s)):
            ss3 = ss3 + ((4703.5 / 8.4 + 2935.0 / 6.0 * mm - 120.0 * mm * mm) +
                         (-4108.25 / 6.72 - 108.5 / 1.2 * mm + 125.5 / 3.6 * mm * mm)) * mm * mm * xs
        gam = (554345.0 / 1134.0 + 110.0 * eta / 9.0) * SL + (13915.0 / 84.0 - 10.0 * eta / 3.0) * dS
        one = torch.ones_like(eta)
        v = [one, 0 * one, 5.0 * (743.0 / 84.0 + 11.0 * eta) / 9.0, -16.0 * pi + 188.0 * SL / 3.0 + 25.0 * dS,
             5.0 * (3058.673 / 7.056 + 5429.0 / 7.0 * eta + 617.0 * e2) / 72.0 - 10.0 * sigma,
             5.0 / 9.0 * (7729.0 / 84.0 - 13.0 * eta) * pi - gam,
             11583.231236531 / 4.694215680 - 640.0 / 3.0 * Pi2 - 6848.0 / 21.0 * self.GAMMA +
             eta * (-15737.765635 / 3.048192 + 2255.0 / 12.0 * Pi2) + e2 * 76055.0 / 1728.0 - e3 * 127825.0 / 1296.0 -
             6848.0 / 21.0 * math.log(4.0) + pi * (3760.0 * SL + 1490.0 * dS) / 3.0 + ss3 - ss3,
             pi * (77096675.0 / 254016.0 + 378515.0 / 1512.0 * eta - 74045.0 / 756.0 * e2) +
             (-8980424995.0 / 762048.0 + 6586595.0 * eta / 756.0 - 305.0 * e2 / 36.0) * SL -
             (170978035.0 / 48384.0 - 2876425.0 * eta / 672.0 - 4735.0 * e2 / 144.0) * dS]
        vl5, vl6 = 5.0 / 3.0 * (7729.0 / 84.0 - 13.0 * eta) * pi - 3.0 * gam, -6848.0 / 21.0 * one
        sg = [fit("s1"), fit("s2"), fit("s3"), fit("s4")]
        self.al, self.be = [fit("a%d" % k) for k in range(1, 6)], [fit("b%d" % k) for k in range(1, 4)]
        pv, pl5, pl6 = [u * pf for u in v], vl5 * pf, vl6 * pf
        t = pi ** (1 / 3.0)
        self.pq = [pv[5] - pi / 4, pv[7] * t * t, pv[6] * t, pl6 * t, pl5, pv[4] / t, pv[3] / (t * t), pv[2] / pi,
                   pv[0] / t ** 5, sg[0], sg[1] * 0.75, sg[2] * 0.6, sg[3] / 2]
        fj = torch.full_like(eta, 0.018)
        u = (pi * 0.018) ** (1 / 3.0)
        lu = math.log(u)
        D = (2.0 * pv[7] * u ** 7 + (pv[6] + pl6 * (1.0 + lu)) * u ** 6 + pl5 * u ** 5 - pv[4] * u ** 4 - 2.0 * pv[3] * u ** 3 -
             3.0 * pv[2] * u ** 2 - 5.0 * pv[0]) / (u ** 8 * 3.0 / pi)
        # slopes as the reference joins them (its inspiral and intermediate derivatives carry 1/eta)
        D = D + (sg[0] + sg[1] * u / t + sg[2] * u ** 2 / (t * t) + sg[3] / pi * u ** 3) / eta
        b, al = self.be, self.al
        dint = lambda f: (b[0] + b[2] / f ** 4 + b[1] / f) / eta                    # noqa: E731
        dmrd = lambda f: (al[0] + al[1] / f ** 2 + al[2] / f ** 0.25 + al[3] /      # noqa: E731
                          (self.fDM * (1 + ((f - al[4] * self.fRD) / self.fDM) ** 2))) / eta
        self.C2I = D - dint(fj)
        self.C1I = self.phi_ins(fj) - self.phi_int(fj) / eta - self.C2I * fj
        fm = 0.5 * self.fRD
        self.fm = fm
        at = self.phi_int(fm) / eta + self.C1I + self.C2I * fm
        self.C2M = self.C2I + dint(fm) - dmrd(fm)
        self.C1M = at - self.phi_mrd(fm) / eta - self.C2M * fm
        self.t0, self.ref = dmrd(self.fmax), self.Msec * 100.0
        self.pre = 2.0 * phi0 + self.phase(self.ref)
        self._projection(col, mc / MSUN, mt / MSUN)

    def _projection(self, col, mc, mt):
        ev, pi = self.ev, math.pi
        t = 4.92569043916e-6
        mc, M = mc * t, mt * t
        eta = torch.clamp((mc / M) ** (5.0 / 3.0), max=0.25)
        dm = torch.sqrt(1.0 - 4.0 * eta)
        c1, c2 = col[2], col[3]
        chi = (M * (1 + dm) / 2 * c1 + M * (1 - dm) / 2 * c2) / M
        th = (eta * col[5] / (5.0 * M)) ** -0.125
        x = (1.0 + (11.0 / 32.0 * eta + 743.0 / 2688.0) * th ** 2 +
             (-3.0 * pi / 10.0 + (113.0 * chi - 38.0 * eta * (c1 + c2)) / 160.0) * th ** 3 +
             (1855099.0 / 14450688.0 + 56975.0 / 258048.0 * eta + 371.0 / 2048.0 * eta ** 2 +
              (-3386880.0 * chi ** 2 + 1512.0 * c1 * c2) / 14450688.0) * th ** 4 -
             (7729.0 / 21504.0 - 13.0 / 256.0 * eta) * pi * th ** 5 +
             (-720817631400877.0 / 288412611379200.0 + 53.0 / 200.0 * pi ** 2 + 107.0 / 280.0 * 0.5772156649 +
              (25302017977.0 / 4161798144.0 - 451.0 / 2048.0 * pi ** 2) * eta - 30913.0 / 1835008.0 * eta ** 2 +
              235925.0 / 1769472.0 * eta ** 3 + 107.0 / 280.0 * torch.log(2.0 * th)) * th ** 6)
        self.fbegin = th ** 3 / (8.0 * M * pi) * x
        cp, sp, sd = torch.cos(col[9]), torch.sin(col[9]), col[8]
        cd = torch.sqrt(torch.clamp(1 - sd * sd, min=0.0))
        ca, sa = torch.cos(col[7] - ev["GMST"]), torch.sin(col[7] - ev["GMST"])
        v = (cp, sp, cd, sd, ca, sa)

        def poly(row, monos):
            out = 0.0
            for k, e in zip(row, monos):
                term = k
                for w, n in zip(v, e):
                    for _ in range(n):
                        term = term * w
                out = out + term
            return out
        Ap, Ac = (1.0 + col[10] ** 2) / 2.0, -col[10]
        self.F, self.lam, self.td = [], [], []
        for k in ev["labels"]:
            fp, fx = poly(_ANT_P[k], _MONO_P), poly(_ANT_X[k], _MONO_X)
            self.F.append(torch.sqrt(Ap ** 2 * fp ** 2 + Ac ** 2 * fx ** 2))
            lam = torch.atan2(Ac * fx, Ap * fp)
            self.lam.append(torch.where(lam < 0, lam + 2 * pi, lam))
            # cos and sin of GMST - alpha
            self.td.append(-(_DET[k][0] * cd * ca - _DET[k][1] * cd * sa + _DET[k][2] * sd) / 299792458.0)

    def amp_ins(self, f):
        a, t = self.ai, f ** (1 / 3.0)
        return (1.0 + t * t * a[0] + f * a[1] + f * t * a[2] + f * t * t * a[3] + f * f * a[4] + f * f * t * a[5] +
                f * f * t * t * a[6] + f ** 3 * a[7])

    def amp_mrd(self, f):
        fg, df = self.fDM * self.g[2], f - self.fRD
        return torch.exp(-df * self.g[1] / fg) * (fg * self.g[0]) / (df * df + fg * fg)

    def phi_ins(self, f):
        k, t = self.pq, f ** (1 / 3.0)
        lv = torch.log(t * math.pi ** (1 / 3.0))
        return (k[0] + k[1] * t * t + k[2] * t + k[3] * lv * t + k[4] * lv + k[5] / t + k[6] / (t * t) + k[7] / f +
                k[8] / (f * t * t) + (k[9] * f + k[10] * f * t + k[11] * f * t * t + k[12] * f * f) / self.eta)

    def phi_int(self, f):
        b = self.be
        return b[0] * f - b[2] / (3.0 * f ** 3) + b[1] * torch.log(f)

    def phi_mrd(self, f):
        a = self.al
        return -a[1] / f + 4.0 / 3.0 * a[2] * f ** 0.75 + a[0] * f + a[3] * torch.atan((f - a[4] * self.fRD) / self.fDM)

    def phase(self, f):
        return torch.where(f < 0.018, self.phi_ins(f), torch.where(
            f >= self.fm, self.phi_mrd(f) / self.eta + self.C1M + self.C2M * f,
            self.phi_int(f) / self.eta + self.C1I + self.C2I * f))

    def projected(self, freq, taper):
        """(amplitude, phase) [B, nifo, n] at freq [n]; zero at and below the start frequency, or tapered."""
        f = self.Msec * freq[None, :]
        v, n = self.newton, self.nodes
        x = f - n[0]
        mid = v[0] + x * (v[1] + x * (v[2] + (f - n[1]) * (v[3] + (f - n[2]) * v[4])))
        a = torch.where(f < 0.014, self.amp_ins(f), torch.where(f >= self.fmax, self.amp_mrd(f), mid))
        a = self.scale * self.a0 * f ** (-7.0 / 6.0) * a
        inside = freq[None, :] <= 0.2 / self.Msec
        ph = torch.where(inside, self.phase(f) - (self.t0 * (f - self.ref) + self.pre), torch.zeros_like(f))
        a = torch.where(inside, a, torch.zeros_like(a))
        if taper:
            fb = self.fbegin
            a = a * torch.where(freq[None, :] < fb, torch.exp(10.0 * (freq[None, :] - fb) / fb), torch.ones_like(a))
        else:
            a = torch.where(freq[None, :] > self.fbegin, a, torch.zeros_like(a))
        a = a * (0.31539156525252 / math.sqrt(self.ev["Tobs"]))
        X = [2 * math.pi * freq[None, :] * (self.ts - td) + lam - ph for td, lam in zip(self.td, self.lam)]
        return torch.stack([F * a for F in self.F], 1), torch.stack(X, 1)


def _sets(P):
    return torch.from_numpy(np.ascontiguousarray(P)).to(DEV)


def _exact_full(ev, P, SN):
    lo, hi, N = ev["lo"], ev["hi"], ev["N"]
    k = torch.arange(max(lo, 1), hi, device=DEV)
    f, dr, di, S = ev["f"][k], ev["D"][:, k], ev["D"][:, N - k], SN[:, k]
    lnl, rho = [], []
    step = max(1, int(6e6 // (len(k) * len(ev["labels"]))))
    for b in range(0, len(P), step):
        A, x = _Wave(_sets(P[b:b + step]), ev).projected(f, taper=False)
        hd = 4.0 * (A * (dr * torch.cos(x) + di * torch.sin(x)) / S).sum(-1)
        hh = 4.0 * (A * A / S).sum(-1)
        lnl.append((hd - 0.5 * hh).sum(-1))
        rho.append(hd / torch.sqrt(hh))
    return torch.cat(lnl), torch.cat(rho)


def _gram(J, U):
    """Discrete Legendre polynomials on U + 1 points (QuickCBC.c:5055-5094)."""
    k = torch.arange(U + 1, device=DEV, dtype=torch.float64)
    c0, c1, c2 = torch.zeros_like(k), U - 2 * k, torch.full_like(k, float(U))
    d0, d1, d2 = c2.clone(), 2 * c1, c2.clone()
    out = [torch.ones_like(k), c1 / U]
    for i in range(1, J):
        d0, d2 = d0 + 2.0, d2 - 2.0
        c0, c1, c2 = c0 + d0, c1 + d1, c2 + d2
        out.append((c1 * out[i] - c0 * out[i - 1]) / c2)
    return torch.stack(out)


def _exact_tables(ev, grid, SN):
    """The heterodyne tables about the injection (QuickCBC.c:5112-5299)."""
    fgrid, MN, MM = grid
    J, N, nh, nifo = 2, ev["N"], ev["N"] // 2, len(ev["labels"])
    NR = (len(fgrid) - 1) // J
    w = _Wave(_sets(ev["inj"][None, :]), ev)
    j = torch.arange(1, nh, device=DEV)
    f = ev["f"]
    A, ph = (v[0] for v in w.projected(f, taper=True))
    H, _ = w.projected(f, taper=False)
    H = H[0]
    cp, sp = torch.cos(ph), torch.sin(ph)
    rr, ri = torch.zeros_like(A), torch.zeros_like(A)
    rr[:, 1:] = ev["D"][:, j] - (H * cp)[:, 1:]
    ri[:, 1:] = ev["D"][:, N - j] - (H * sp)[:, 1:]
    S = SN[:, :nh]
    RC, RS, AA = 2 * (rr * cp + ri * sp) * A / S, 2 * (-rr * sp + ri * cp) * A / S, A * A / S
    for v in (RC, RS, AA):
        v[:, 0] = 0.0
    b = slice(MN, MM)
    hh = 4.0 * (H[:, b] ** 2 / S[:, b]).sum(-1)
    hr = 4.0 * ((rr * H * cp + ri * H * sp)[:, b] / S[:, b]).sum(-1)
    g = torch.from_numpy(fgrid.astype(np.int64)).to(DEV)
    t = dict(fgrid=None, freq=g.double() / ev["Tobs"], amp=A[:, g], phase=ph[:, g], logLb=float((hr + 0.5 * hh).sum()),
             M=None, J=None, NR=None, MN=None, MM=None, Nifo=None)
    edge = g[0:NR * J:J]
    t["aa"], t["rc"], t["rs"] = AA[:, edge], RC[:, edge], RS[:, edge]
    IP, SL, lc, ls = [], [], [], []
    for r in range(NR):
        k0, k1 = int(fgrid[r * J]), int(fgrid[(r + 1) * J])
        pol = _gram(J, k1 - k0)
        at = torch.from_numpy((fgrid[r * J:r * J + J + 1] - k0).astype(np.int64)).to(DEV)
        IP.append(torch.linalg.inv(pol[:, at]).T)
        s = slice(k0, k1 + 1)
        for dst, v in ((SL, AA), (lc, RC), (ls, RS)):
            dst.append(v[:, s] @ pol.T)
    for name, v in (("IP", IP), ("SL", SL), ("lc", lc), ("ls", ls)):
        t[name] = torch.stack(v)
    return t


def _exact_het(ev, t, P):
    """log_likelihood_het (QuickCBC.c:5303-5444) from the tables t."""
    J, NR = 2, t["SL"].shape[0]
    A, ph = _Wave(_sets(P), ev).projected(t["freq"], taper=True)
    ar, d = t["amp"], t["phase"] - ph
    hc, hs = 2 * (ar - A * torch.cos(d)) / ar, 2 * A * torch.sin(d) / ar
    L = torch.full((len(P),), t["logLb"], device=DEV, dtype=torch.float64)
    at = (torch.arange(NR, device=DEV)[:, None] * J + torch.arange(J + 1, device=DEV)[None, :])
    sums = []
    for vec, proj, edge in ((hc * hc + hs * hs, t["SL"], t["aa"]), (hc, t["lc"], t["rc"]), (hs, t["ls"], t["rs"])):
        u = torch.einsum("rac,bdrc->bdra", t["IP"], vec[:, :, at])
        s = torch.einsum("bdra,rda->b", u, proj)
        # regions share their end points: those of all but the last two are taken off again
        last = vec[:, :, (torch.arange(NR - 2, device=DEV) + 1) * J]
        sums.append(s - (last * edge[None, :, 1:NR - 1]).sum((1, 2)))
    return L - (sums[1] + sums[2] + 0.5 * sums[0])


def _exact_psd(model, k, nifo, Tobs, nh):
    """makespec (Utilities.c:1908-1955): exp of a natural spline of log S, times Lorentzian lines."""
    ns, nl, ffit, xs, lines = model
    f = torch.arange(nh, device=DEV, dtype=torch.float64) / Tobs
    rows = []
    for i in range(nifo):
        x, y = ffit[i, :ns[i]], xs[i, k, :ns[i]]
        m2 = _natural_spline(x, y)
        sm = torch.exp(_spline(*(torch.from_numpy(np.ascontiguousarray(v)).to(DEV) for v in (x, y, m2)), f))
        add = torch.zeros_like(f)
        for lf, lh, lQ, lw, ld in lines[i, k, :nl[i]]:
            ax = torch.abs(f - lf)
            z = torch.where(ax > ld, torch.exp(-(ax - ld) / ld), torch.ones_like(f))
            term = z * lh / (f * f / lf ** 2 + (lQ * (1 - f * f / lf ** 2)) ** 2)
            add = add + torch.where(ax < lw, term, torch.zeros_like(f))
        S = sm * (1 + add)
        S[0], S[-1] = math.exp(y[0]), math.exp(y[-1])
        rows.append(S)
    return torch.stack(rows)


def exact(case, seed):
    c = case
    if c["kind"] == "multi":
        evs, eo, P = _multi_inputs(c, seed)
        return torch.cat([_exact_full(ev, P[eo == e], ev["SN"])[0] for e, ev in enumerate(evs)])
    if c["kind"] == "grid":
        return None                            # whole numbers: they stay equal
    ev, P, model = _inputs(c, seed)
    if c["kind"] == "full":
        return _exact_full(ev, P, ev["SN"])
    if c["kind"] == "redraw":
        S = _exact_psd(model, 1, int(c["nifo"]), ev["Tobs"], ev["N"] // 2)
        return _exact_het(ev, _exact_tables(ev, _het_grid(c), S), P), _exact_full(ev, P, S)[0]
    t = _exact_tables(ev, _het_grid(c), ev["SN"])
    return t if c["kind"] == "tables" else _exact_het(ev, t, P)
