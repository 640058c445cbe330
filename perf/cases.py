"""Timed cases of the land-surface step: what users of this package run, through
its public entry points, over the range of sizes they run it at.

A case is a dict of plain values; its ``kind`` names the entry point:

* ``hour``     one hourly step per call (``Columns.run`` with one hour of forcing),
               the form a host program that owns the hour loop uses; with
               ``diag`` the diagnostics are written too, as the drop-in
               ``timestep_body`` needs them.  Each pass is the next hour of a
               day of forcing, the state carried along.
* ``span``     several hours in one call (``Columns.run``), the accumulators on;
               ``release`` switches on the IBIS 3.0 formulation of the release
               parameter file (sunlit/shaded canopies, vmax and slope mixing,
               capacity split), ``f64`` runs the float64 kernels, ``midyear``
               carries the running annual sums of a state part-way through a
               year.  Each pass starts from the same state, as a sensitivity or
               calibration loop does.
* ``host``     the same from pinned host forcing to host state (``Columns.run_host``).
* ``dayloop``  days of the day loop (``DayLoop.run_month``: daily cadence, forcing
               generated from daily weather, hourly steps with hourly methane,
               the period's wetland methane).
* ``cadence``  the daily cadence alone (``DayLoop.end`` and the next ``DayLoop.begin``).
* ``ensemble`` a calibration ensemble, sites x parameter vectors with records of
               uneven length, in one persistent launch (``Ensemble.run``);
               ``daily`` generates the hours from day records.

``exact`` restates the daily cadence in float64.  The hourly step has no value
here: its physics is some two thousand lines, which this file does not restate
(``tests/`` hold it to the float64 oracle).
"""
import math

import numpy as np
import torch

from ibis_b200 import layout as L
from ibis_b200 import synth
from ibis_b200.columns import Columns
from ibis_b200.daily import DayLoop
from ibis_b200.ensemble import Ensemble, make_ensemble
from ibis_b200.forcing import daily_planes
from ibis_b200.params import (FLAG_CH4, FLAG_COEFM_MIX, FLAG_GPP_CAPACITY, FLAG_SUNSHADE_L, FLAG_SUNSHADE_U,
                              FLAG_VMAX_MIX, DayParams, StepParams)

DEV = "cuda"
GRID = 95333          # land cells of the half-degree grid
SITES = 356           # tower sites of the calibration network
RELEASE = FLAG_SUNSHADE_U | FLAG_SUNSHADE_L | FLAG_VMAX_MIX | FLAG_COEFM_MIX | FLAG_GPP_CAPACITY


def listed():
    return [
        # one hour of a handful of sites with diagnostics: a coupled single-site or drop-in run, latency only
        dict(name="hour_sites", kind="hour", cells=16, diag=True, doy=172, hour0=9),
        # one hour of a region with diagnostics: the drop-in called hour by hour
        dict(name="hour_region", kind="hour", cells=5003, diag=True, doy=100, hour0=6),
        # one hour of a continent, no diagnostics: the plain per-step launch
        dict(name="hour_continent", kind="hour", cells=33001, diag=False, doy=172, hour0=10),
        # a day of the tower network in one launch
        dict(name="day_sites", kind="span", cells=SITES, hours=24, doy=172, hour0=0, release=False, f64=False),
        # six-hourly coupling of a region: a batch that fills part of the chip's blocks
        dict(name="span_region", kind="span", cells=12007, hours=6, doy=280, hour0=10, release=False, f64=False),
        # the same for the whole grid: the headline batch
        dict(name="span_grid", kind="span", cells=GRID, hours=6, doy=172, hour0=10, release=False, f64=False,
             midyear=True),
        # the release formulation on a continent
        dict(name="span_release", kind="span", cells=33001, hours=6, doy=172, hour0=10, release=True, f64=False),
        # float64 parity runs of a thousand columns
        dict(name="span_f64", kind="span", cells=1009, hours=3, doy=172, hour0=9, release=False, f64=True),
        # host forcing in, host state out, half the grid: batches too large to keep their forcing on the GPU
        dict(name="host_half", kind="host", cells=50001, hours=6, doy=172, hour0=10, midyear=True),
        # the day loop of a site network: daily cadence, generated forcing, monthly methane
        dict(name="dayloop_sites", kind="dayloop", cells=200, days=1, doy=152),
        # the daily cadence of the whole grid
        dict(name="cadence_grid", kind="cadence", cells=GRID, doy=152),
        # a calibration batch: sites x 64 parameter vectors, 4 to 12 hours each
        dict(name="ensemble_hours", kind="ensemble", sites=89, vectors=64, least=4, most=12, daily=False),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], odd more often than not."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, n | 1) if rng.random() < 0.8 else n


def draw(rng):
    when = dict(doy=rng.randrange(1, 366), hour0=rng.randrange(9, 13))
    kind = rng.choice(["hour", "hour", "span", "span", "span", "release", "f64", "host", "dayloop", "cadence",
                       "ensemble", "ensemble"])
    if kind == "hour":
        return dict(kind="hour", cells=_size(rng, 16, 33001), diag=rng.random() < 0.5, **when)
    if kind == "span":
        if rng.random() < 0.25:
            return dict(kind="span", cells=_size(rng, 1, SITES), hours=24, release=False, f64=False, **when)
        cells = _size(rng, 64, GRID)
        return dict(kind="span", cells=cells, hours=rng.randrange(2, 7), release=False, f64=False,
                    midyear=cells > 20000, **when)
    if kind == "release":
        return dict(kind="span", cells=_size(rng, 64, 33001), hours=rng.randrange(2, 7), release=True, f64=False,
                    **when)
    if kind == "f64":
        return dict(kind="span", cells=_size(rng, 16, 2000), hours=rng.randrange(1, 4), release=False, f64=True,
                    **when)
    if kind == "host":
        cells = _size(rng, 1000, GRID)
        return dict(kind="host", cells=cells, hours=rng.randrange(2, 7), midyear=cells > 20000, **when)
    if kind == "dayloop":
        return dict(kind="dayloop", cells=_size(rng, 16, 300), days=1, doy=when["doy"])
    if kind == "cadence":
        return dict(kind="cadence", cells=_size(rng, 1000, GRID), doy=when["doy"])
    if rng.random() < 0.3:
        return dict(kind="ensemble", sites=rng.randrange(3, 10), vectors=32, least=24, most=24, daily=True)
    return dict(kind="ensemble", sites=rng.randrange(3, 90), vectors=rng.choice([16, 31, 64]), least=2,
                most=rng.randrange(4, 13), daily=False)


# ---------------------------------------------------------------------------- inputs

def _workload(cells, hours, seed, doy, hour0, release=False):
    """Columns drawn as the repository's synthetic day workload draws them, with
    ``hours`` of forcing from hour ``hour0`` of day ``doy``."""
    rng = np.random.Generator(np.random.PCG64(seed))
    lat = rng.uniform(-60.0, 80.0, size=cells)
    stat = synth.make_columns(rng, cells, 0.5)
    forc = synth.make_forcing(rng, lat, hours, start_doy=doy, start_hour=hour0)
    prog = synth.make_initial(rng, stat, {k: v[0] for k, v in forc.items()})
    params = StepParams(co2conc=390.0e-6)
    if release:
        params.flags |= RELEASE
    return prog, stat, forc, params, lat, rng


def _dayloop(case, seed):
    prog, stat, _, params, lat, rng = _workload(case["cells"], 1, seed, case["doy"], 0)
    dayst = synth.make_dayst(rng, stat, lat)
    cols = Columns.from_host(prog, stat, dtype=torch.float32, device=DEV, acc=True)
    params.flags |= FLAG_CH4
    loop = DayLoop(cols, params, DayParams(), dayst, lat=lat, seed=seed, jday=case["doy"], day=0)
    return cols, loop, rng, lat, stat


def _day_sums(rng, n):
    """The step's daily sums and last stress values as a day leaves them."""
    u = rng.uniform
    return dict(adrain=u(0.0, 12.0, n) * (u(0, 1, n) < 0.4), adsnow=u(0.0, 4.0, n) * (u(0, 1, n) < 0.1),
                adaet=u(0.2, 5.0, n), a10ancub=u(0.0, 0.08, n), a10ancls=u(0.0, 0.05, n), a10ancl3=u(0.0, 0.05, n),
                a10ancl4=u(0.0, 0.08, n), stresstu_last=u(0.05, 1.0, n), stresstl_last=u(0.05, 1.0, n))


def _year_sums(rng, stat):
    """The running annual sums of a state part-way through a year, as a checkpoint carries them."""
    n = stat["fu"].shape[0]
    u = rng.uniform
    npp = stat["frac"] * u(0.02, 0.2, (n, L.NPFT))
    return dict(aynpp=npp, aynpptot=npp.sum(1), aygpptot=u(1.8, 2.2, n) * npp.sum(1), aytrunof=u(5.0, 200.0, n),
                aytdrain=u(5.0, 300.0, n), afsena=u(1.0e8, 6.0e8, n))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind)
    if kind == "ensemble":
        rng = np.random.Generator(np.random.PCG64(seed))
        hours = rng.integers(case["least"], case["most"] + 1, size=case["sites"])
        spec = make_ensemble(case["sites"], case["vectors"], seed=seed, site_hours=hours, daily=case["daily"])
        s["ens"] = Ensemble(spec, device=DEV)
        return s
    if kind in ("dayloop", "cadence"):
        cols, loop, rng, lat, stat = _dayloop(case, seed)
        s.update(cols=cols, loop=loop, jday=case["doy"])
        if kind == "dayloop":
            daily = synth.make_daily_weather(rng, lat, case["days"])
            s["daily"] = torch.from_numpy(daily_planes(daily, cols.ld)).to(DEV)
            cols.set_acc(_year_sums(rng, stat))
            s["start"] = [t.clone() for t in (cols.prog, cols.stat, cols.acc, loop.dayst, loop.wet)]
        else:
            n = case["cells"]
            cols.set_prog(dict(tsoi=rng.uniform(255.0, 305.0, (n, L.NSOILAY)),
                               wsoi=rng.uniform(0.05, 1.0, (n, L.NSOILAY)),
                               wisoi=rng.uniform(0.0, 0.6, (n, L.NSOILAY)) * (rng.uniform(0, 1, (n, 1)) < 0.3)))
            cols.set_acc(_day_sums(rng, n))
            td = np.zeros(cols.ld, dtype=np.float32)
            td[:n] = rng.uniform(258.0, 303.0, n)
            s["td"] = torch.from_numpy(td).to(DEV)
        return s
    hours = 24 if kind == "hour" else case["hours"]
    dtype = torch.float64 if case.get("f64") else torch.float32
    prog, stat, forc, params, _, rng = _workload(case["cells"], hours, seed, case["doy"], case["hour0"],
                                               case.get("release", False))
    cols = Columns.from_host(prog, stat, dtype=dtype, device=DEV, diag=case.get("diag", False), acc=True)
    if case.get("midyear"):
        cols.set_acc(_year_sums(rng, stat))
    s.update(cols=cols, params=params, hour=0, prog0=cols.prog.clone(), acc0=cols.acc.clone())
    if kind == "host":
        s["forc"] = torch.from_numpy(synth.forcing_planes(forc, cols.ld)).pin_memory()
        s["out"] = torch.empty(cols.prog.shape, dtype=torch.float32).pin_memory()
    else:
        s["forc"] = cols.forcing(forc)
    return s


# ---------------------------------------------------------------------------- passes

def _columns_out(cols):
    n = cols.ncell
    out = dict(prog=cols.prog[:, :n], acc=cols.acc[:, :n])
    if cols.diag is not None:
        out["diag"] = cols.diag[:, :n]
    return out


def run(s):
    kind = s["kind"]
    if kind == "ensemble":
        e = s["ens"]
        e.reset()
        e.run()
        return dict(prog=e.prog[:, :e.nrun], acc=e.acc[:, :e.nrun])
    cols = s["cols"]
    n = cols.ncell
    if kind == "hour":
        h = s["hour"]
        s["hour"] = (h + 1) % 24
        cols.run(s["forc"][h:h + 1], s["params"])
        return _columns_out(cols)
    if kind == "span":
        cols.prog.copy_(s["prog0"])
        cols.acc.copy_(s["acc0"])
        cols.run(s["forc"], s["params"])
        return _columns_out(cols)
    if kind == "host":
        cols.prog.copy_(s["prog0"])
        cols.acc.copy_(s["acc0"])
        cols.run_host(s["forc"], s["params"], host_prog=s["out"])
        return dict(prog=s["out"][:, :n], acc=cols.acc[:, :n])
    loop = s["loop"]
    if kind == "dayloop":
        for t, t0 in zip((cols.prog, cols.stat, cols.acc, loop.dayst, loop.wet), s["start"]):
            t.copy_(t0)
        loop.jday, loop.day = s["jday"], 0
        loop.run_month(s["daily"], from_mean=True)
        return dict(prog=cols.prog[:, :n], stat=cols.stat[:, :n], acc=cols.acc[:, :n], dayst=loop.dayst[:, :n],
                    wet=loop.wet[:, :n])
    loop.end(s["td"])
    loop.begin(s["td"])
    return dict(stat=cols.stat[:, :n], acc=cols.acc[:, :n], dayst=loop.dayst[:, :n])


# ---------------------------------------------------------------------------- work

# Planes the step reads of the static inputs (of 135: the optional and switch
# planes apart) and the accumulator planes a launch sums (values and Kahan terms).
STAT_READ, ACC_PLANES = 113, 2 * 25
# Arithmetic of one column-hour, from the formulae (three canopy passes, two
# bands of radiation over two stories, snow, soil water and heat).
STEP_FLOPS = 8000.0


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        runs = case["sites"] * case["vectors"]
        hours = 0.5 * (case["least"] + case["most"])
        state = 4.0 * (2 * L.N_PROG + 2 * ACC_PLANES + L.N_RUN) * runs
        rec = 48.0 * case["sites"] * (hours / 24.0 if case["daily"] else hours)
        return dict(bytes=state + rec + 4.0 * STAT_READ * case["sites"], flops=STEP_FLOPS * runs * hours)
    n = case["cells"]
    if kind == "cadence":
        # end: 19 state, 5 static, 9 sums and 39 daily-state planes in, 33 out; begin: 33 in, 38 out
        return dict(bytes=4.0 * n * (72 + 33 + 33 + 38), flops=1500.0 * n)
    if kind == "dayloop":
        hours = 24 * case["days"]
        return dict(bytes=4.0 * n * (2 * L.N_PROG + STAT_READ + 2 * ACC_PLANES + case["days"] * (L.N_DAILY + 176)),
                    flops=STEP_FLOPS * n * hours)
    hours = 1 if kind == "hour" else case["hours"]
    word = 8.0 if case.get("f64") else 4.0
    planes = 2 * L.N_PROG + STAT_READ + 2 * ACC_PLANES + L.N_FORC * hours + (L.N_DIAG if case.get("diag") else 0)
    return dict(bytes=word * planes * n, flops=STEP_FLOPS * n * hours)


# ---------------------------------------------------------------------------- exact

def exact(case, seed):
    """The daily cadence in float64 from the same float32 inputs; no value for the hourly step."""
    if case["kind"] != "cadence":
        return None
    s = prepare(case, seed)
    cols, loop, n = s["cols"], s["loop"], case["cells"]
    host = lambda t: t[:, :n].double().cpu().numpy()
    G, S, A, D = host(cols.prog), host(cols.stat), host(cols.acc), host(loop.dayst)
    td = s["td"][:n].double().cpu().numpy()
    p, P = loop.day_params, loop.params
    _cadence_end(G, S, A, D, td, p, P)
    _cadence_begin(S, A, D, td, p, P)
    return dict(stat=S, acc=A, dayst=D)


def _at(group, name, k=0):
    return L.OFF[group][name][0] + k


def _f32(x):
    return float(np.float32(x))


def _cadence_end(G, S, A, D, td, p, P):
    """A day's end: 10-day means, annual sums, decomposition factors, soil C/N, respiration."""
    d = lambda name: D[_at("DAYST", name)].copy()
    acc = lambda name: A[_at("ACC", name)] - A[L.N_ACC + _at("ACC", name)]

    def put(name, v):
        D[_at("DAYST", name)] = v

    zw = math.exp(-0.1)
    put("a10td", zw * d("a10td") + (1.0 - zw) * td)
    for k in ("a10ancub", "a10ancls", "a10ancl3", "a10ancl4"):
        put(k, zw * d(k) + (1.0 - zw) * acc(k) / 86400.0)
    put("ayprcp", d("ayprcp") + acc("adrain") + acc("adsnow"))
    put("ayaet", d("ayaet") + acc("adaet"))

    h = np.asarray(P.hsoi, dtype=np.float64)[:4]
    lay = lambda name, k: G[_at("PROG", name, k)]
    mean4 = lambda name: sum(lay(name, k) * h[k] for k in range(4)) / h.sum()

    def factor(t, w, i):
        safe = np.maximum(t, _f32(237.13))
        inv = _f32(1.0 / (np.float32(288.16) - np.float32(227.13)))
        ft = np.minimum(np.exp(_f32(p.lt_e0) * (inv - 1.0 / (safe - _f32(227.13)))), 10.0)
        wf = (1.0 - i) * w * 100.0 - (p.wfps_opt - 60.0)
        wet = _f32(0.000371) * wf * wf - _f32(0.0748) * wf + _f32(4.13)
        return np.clip(ft * np.where(wf >= 60.0, wet, np.exp((wf - 60.0) ** 2 / -800.0)) * p.k_scale, _f32(0.001), 10.0)

    dl = factor(lay("tsoi", 0), lay("wsoi", 0), lay("wisoi", 0))
    ds = factor(mean4("tsoi"), mean4("wsoi"), mean4("wisoi"))
    put("decompl", dl)
    put("decomps", ds)

    # soil carbon and nitrogen, one day; the stored factors round to float32 first
    dl, ds = dl.astype(np.float32).astype(np.float64), ds.astype(np.float32).astype(np.float64)
    c, tot = p.cnr, 1.0 / P.ndaypy
    sand = sum(0.01 * S[_at("STAT", "sand", k)] * h[k] for k in range(4)) / h.sum()
    fall = dict(l=d("falll"), r=d("fallr"), w=d("fallw"))
    pool = {k: d("clit" + k) for k in ("lm", "ls", "ll", "rm", "rs", "rl", "wm", "ws", "wl")}
    slop, slon, pas, cmic = d("csoislop"), d("csoislon"), d("csoipas"), d("totcmic")
    begin = sum(pool.values()) + slop + slon + pas + cmic
    most = p.fbsom * begin
    protected, open_ = np.minimum(cmic, most), np.maximum(0.0, cmic - most)
    for o, cn, last in (("l", p.cnleaf, 5), ("r", p.cnroot, 5), ("w", p.cnwood, 7)):
        fl = p.bgc_fmax * cn * cn / (p.rconst + cn * cn)
        fs = (1.0 / cn - fl / c[4] - (1.0 - fl) / c[6]) / (1.0 / c[last] - 1.0 / c[6])
        for kind, f in (("m", 1.0 - fl - fs), ("s", fs), ("l", fl)):
            pool[o + kind] = pool[o + kind] + f * fall[o] * tot
    rate_of = lambda k: dl if k in ("lm", "ls", "ll", "wm", "ws", "wl") else ds
    out = {k: np.minimum(rate_of(k) * getattr(p, "k" + k) * v, v) for k, v in pool.items()}
    onb, opb, osb = (np.minimum(ds * k * v, v) for k, v in ((p.knb, slon), (p.kpb, slop), (p.ksb, pas)))
    ons, ops = np.minimum(ds * p.kns * slon, slon), np.minimum(ds * p.kps * slop, slop)
    obp = np.minimum(p.kbp * protected, protected) * p.effac
    obn = np.minimum(p.kbn * open_, open_) * p.effac
    gain = sum(out[k] * getattr(p, "y" + k) for k in ("rs", "ws", "ls", "lm", "rm", "wm"))
    gain = gain + onb * p.ynb + opb * p.ypb + osb * p.ysb
    lig = p.lig_frac * sum(out[k] * getattr(p, "y" + k) for k in ("ll", "rl", "wl"))
    died = 0.5 * (p.ybn * obn + p.ybp * obp)
    leach = 0.30e-3 / 18.0 * (0.01 + 0.04 * sand)
    put("ynleach", d("ynleach") + leach * (pas / c[1] + slop / c[2] + slon / c[3]))
    put("yrleach", d("yrleach") + leach * (pas + slop + slon))
    net = 0.0
    for y, cn, o in ((p.yrs, c[5], out["rs"]), (p.yls, c[5], out["ls"]), (p.yws, c[7], out["ws"]),
                     (p.ywm, c[7], out["wm"]), (p.ylm, c[6], out["lm"]), (p.yrm, c[6], out["rm"]),
                     (p.ynb, c[3], onb), (p.ypb, c[2], opb), (p.ysb, c[1], osb)):
        net = net + (1.0 / cn - y / c[0]) * o
    net = net + ops * (1.0 / c[2] - 1.0 / c[1]) + ons * (1.0 / c[3] - 1.0 / c[1])
    net = net + 0.5 * (obn + obp) * (2.0 / c[0] - 1.0 / c[3] - 1.0 / c[2])
    net = net + p.lig_frac * (out["ll"] + out["rl"] + out["wl"]) * (2.0 / c[4] - 1.0 / c[2] - 1.0 / c[3])
    tnmin = np.maximum(0.0, net) / (86400.0 * 0.014)
    cmic = np.maximum(0.0, cmic + gain - obp - obn)
    new_slon = np.maximum(0.0, slon + lig + died - onb - ons - leach * slon)
    new_slop = np.maximum(0.0, slop + lig + died - opb - ops - leach * slop)
    new_pas = np.maximum(0.0, pas + p.yns * ons + p.yps * ops - osb - leach * pas)
    for k in pool:
        pool[k] = np.maximum(0.0, pool[k] - out[k])
        put("clit" + k, pool[k])
    soil, litter = new_pas + new_slop + cmic + new_slon, sum(pool.values())
    put("csoipas", new_pas)
    put("csoislon", new_slon)
    put("csoislop", new_slop)
    put("totcmic", cmic)
    put("totlit", litter)
    put("totalit", sum(v for k, v in pool.items() if k[0] != "r"))
    put("totrlit", sum(v for k, v in pool.items() if k[0] == "r"))
    put("totcsoi", soil)
    put("totfall", fall["l"] + fall["r"] + fall["w"])
    put("tnmin", tnmin)
    put("storedn", d("storedn") + tnmin)
    rh = (begin + (fall["l"] + fall["r"] + fall["w"]) * tot - (litter + soil) - leach * (pas + slop + slon)) \
        / (86400.0 * 0.012)
    S[_at("STAT", "tco2mic")] = rh
    conv = _f32(12.0e-3 * 86400.0)
    put("ayco2mic", d("ayco2mic") + rh * conv)
    put("ayco2root", d("ayco2root") + d("tco2root") * conv)


def _cadence_begin(S, A, D, td, p, P):
    """A day's beginning: phenology from the 10-day means and the last stress, the daily sums zeroed."""
    d = lambda name: D[_at("DAYST", name)].copy()
    tm, dd, eps = 273.16, 1.0 / p.ddays, P.epsilon
    su, sl = A[_at("ACC", "stresstu_last")], A[_at("ACC", "stresstl_last")]
    a10 = d("a10td")
    thr_u = np.maximum(np.maximum(tm, d("tc") + p.tthresh_u_offset + tm), p.tthresh_u_abs + tm)
    gu, gl = p.gthresh_u_c + tm, p.gthresh_l_c + tm
    agddu = np.where(a10 < gu, 0.0, d("agddu") + td - gu)
    agddl = np.where(a10 < gl, 0.0, d("agddl") + td - gl)
    grow = lambda sum_, thresh, ramp: np.minimum(1.0, np.maximum(0.0, sum_ - thresh) / ramp)
    tempu = np.where(a10 < thr_u, np.maximum(0.0, d("tempu") - dd), grow(agddu, p.gdd_thresh_u, p.gdd_ramp_u))
    templ = np.where(a10 < p.tthresh_l_c + tm, np.maximum(0.0, d("templ") - dd),
                     grow(agddl, p.gdd_thresh_l, p.gdd_ramp_l))

    def drop(name, anc, s):
        dry = (d(anc) < p.drop_thresh) | (s < p.drop_stress_thresh)
        return np.where(dry, np.maximum(p.drop_floor, d(name) - dd), np.minimum(1.0, d(name) + dd))

    dropu, dropls = drop("dropu", "a10ancub", su), drop("dropls", "a10ancls", sl)
    dropl4, dropl3 = drop("dropl4", "a10ancl4", sl), drop("dropl3", "a10ancl3", sl)
    one = np.ones_like(td)
    up = [one, dropu, one, one, tempu, one, tempu, tempu]
    low = [one, np.minimum(templ, dropls), np.minimum(templ, dropl4), np.minimum(templ, dropl3)]
    plai = [D[_at("DAYST", "plai", j)] * f for j, f in enumerate(up + low)]
    upper, lower = sum(plai[:8]), sum(plai[8:])
    for j in range(12):
        S[_at("STAT", "frac", j)] = plai[j] / np.maximum(upper if j < 8 else lower, eps)
    lai0 = np.minimum(lower / np.maximum(S[_at("STAT", "fl")], eps), 12.0)
    S[_at("STAT", "lai", 0)] = lai0
    S[_at("STAT", "lai", 1)] = np.minimum(upper / np.maximum(S[_at("STAT", "fu")], eps), 12.0)
    S[_at("STAT", "zbot", 0)] = 0.05
    S[_at("STAT", "ztop", 0)] = np.minimum(np.maximum(0.25, 0.25 * lai0), S[_at("STAT", "zbot", 1)] - 0.5)
    for name, v in dict(tempu=tempu, templ=templ, agddu=agddu, agddl=agddl, dropu=dropu, dropls=dropls,
                        dropl3=dropl3, dropl4=dropl4).items():
        D[_at("DAYST", name)] = v
    for k in ("adrain", "adsnow", "adaet", "a10ancub", "a10ancls", "a10ancl3", "a10ancl4"):
        A[_at("ACC", k)] = 0.0
        A[L.N_ACC + _at("ACC", k)] = 0.0
