"""The FP32 kernels' soil-water solve (``soil_water32``, ibis_b200/csrc/ibis_f32.cuh)
restated in NumPy: soilh2o (python-port/ibis/physics/soil_physics.py:196-373) for the
hour's increments, as the kernel forms it -- the drainage boundary as a sixth interface to
a layer of the same soil and water, all powers from one (w**(2n+2) is the square of
w**(n+1)), and an interface's exponent from the difference of the layers'.

In float64 it is the oracle's solve.  In float32 (the elimination too) its bounds are
those of the increment form before it (test_soil_water_increments.py): the same system,
each term in as many roundings or fewer, solved for increments of at most a few percent
of the content, so that the elimination's rounding is far below the content's.
"""
import numpy as np
import pytest

from ibis_b200 import synth
from oracle.column import soil_water

NL = 6


def _thomas(lo, di, up, r):
    """The kernel's elimination, in the operands' type."""
    n = di.shape[1]
    gam, x = np.zeros_like(r), np.zeros_like(r)
    alp = 1 / di[:, 0]
    gam[:, 0], x[:, 0] = up[:, 0] * alp, r[:, 0] * alp
    for k in range(1, n - 1):
        alp = 1 / (di[:, k] - lo[:, k] * gam[:, k - 1])
        gam[:, k] = up[:, k] * alp
        x[:, k] = (r[:, k] - lo[:, k] * x[:, k - 1]) * alp
    x[:, -1] = (r[:, -1] - lo[:, -1] * x[:, -2]) / (di[:, -1] - lo[:, -1] * gam[:, -2])
    for k in range(n - 2, -1, -1):
        x[:, k] = x[:, k] - gam[:, k] * x[:, k + 1]
    return x


def pairs(wsoi, wisoi, poros, porosflo, S, hsoi, fwtop, fwpud, wpud, P, T=np.float64, consistent=False):
    """The kernel's operations in type T; the geometry is formed in double and rounded to T."""
    c = lambda x: np.asarray(x, T)
    w, wi, por, pflo = c(wsoi), c(wisoi), c(poros), c(porosflo)
    h = np.asarray(hsoi, np.float64)
    n = w.shape[0]
    ghost = lambda x: np.concatenate([x, x[:, -1:]], axis=1)
    hyd, bex = c(S["hydraul"]), c(S["bex"])
    hs = hyd * c(S["suction"]) * bex
    w_, wi_, hyd_, hs_, bex_ = (ghost(x) for x in (w, wi, hyd, hs, bex))
    e, f, g = (np.zeros((n, NL + 1), T) for _ in range(3))
    for k in range(1, NL + 1):
        inside = k < NL
        hm = 0.5 * (h[k - 1] + h[k]) if inside else 1.0
        wp, wm = (T(0.5 * h[k] / hm), T(1.0 - 0.5 * h[k] / hm)) if inside else (T(0), T(1))
        a = wm * hyd_[:, k - 1] + wp * hyd_[:, k]
        b = wm * hs_[:, k - 1] + wp * hs_[:, k]
        nn = np.floor(bex_[:, k - 1] + wp * (bex_[:, k] - bex_[:, k - 1]) + T(0.5))
        ws = wp * w_[:, k - 1] + wm * w_[:, k] if consistent else wm * w_[:, k - 1] + wp * w_[:, k]
        wa = np.minimum(ws, T(1))
        pw1 = wa ** (nn.astype(np.int32) + 1)
        wam1 = pw1 * pw1
        bwn1 = b * pw1
        bwn = bwn1 * wa
        bwn1 = np.where(bwn < T(1e-9), T(0), bwn1)
        nd = (nn + T(2)) * bwn1 * ((w_[:, k] - w_[:, k - 1]) * (T(1.0 / hm) if inside else T(0)))
        m1, aw = nn * T(2) + T(2), a * wam1
        zi = np.maximum(T(1) - np.maximum(wi_[:, k - 1], wi_[:, k]), T(0)) ** 2
        if inside:
            e[:, k] = zi * (wa * (m1 * aw - nd))
            f[:, k] = zi * (nd - (m1 + T(1)) * aw)
            g[:, k] = zi * np.maximum(bwn, T(1e-9))
        else:
            e[:, k] = -(zi * aw * wa) * T(P.bperm)
    lo, di, up, r = (np.zeros((n, NL), T) for _ in range(4))
    for k in range(NL):
        hb = 0.5 * h[0] if k == 0 else 0.5 * h[k - 1] + 0.5 * h[k]
        hp = 0.5 * (h[k] + h[k + 1]) if k < NL - 1 else 1.0
        above, below = h[max(k - 1, 0)], h[min(k + 1, NL - 1)]
        dt = T(P.dtime) / np.maximum(pflo[:, k] * T(h[k]), T(1e-30))
        gb, gn = g[:, k] * T(1.0 / hb), g[:, k + 1] * T(1.0 / hp)
        d1 = dt * (f[:, k] * T(0.5 * h[k] / hb) - gb)
        d3 = dt * (T(0) - f[:, k + 1] * T(0.5 * h[k] / hp) - gn)
        d2m = dt * (f[:, k] * T(0.5 * above / hb) - f[:, k + 1] * T(0.5 * below / hp) + gn + gb)
        rk = e[:, k + 1] - e[:, k]
        if k == 0:
            rk = rk + (c(fwtop) + c(fwpud)) / T(P.rhow)
        wu = w[:, k - 1] if k else np.zeros(n, T)
        wd = w[:, k + 1] if k < NL - 1 else np.zeros(n, T)
        r[:, k] = dt * rk - d2m * w[:, k] - d1 * wu - d3 * wd
        lo[:, k], di[:, k], up[:, k] = d1, T(1) + d2m, d3
    dl = _thomas(lo, di, up, r)
    wflo = np.zeros((n, NL + 1), T)
    wflo[:, NL] = -T(P.rhow) * e[:, NL]
    over_kg, out = np.zeros(n, T), w.copy()
    for k in range(NL - 1, -1, -1):
        zz = T(P.rhow) * T(h[k]) * por[:, k] * np.maximum(T(1) - wi[:, k], T(P.epsilon))
        dw = dl[:, k] + over_kg * (T(1) / zz)
        over = (w[:, k] - T(1)) + dw
        over_kg = np.maximum(over, T(0)) * zz
        dw = np.where(over > 0, T(1) - w[:, k], dw)
        wflo[:, k] = wflo[:, k + 1] + dw * zz * T(1.0 / P.dtime)
        out[:, k] = np.where(over > 0, T(1), w[:, k] + dw)
    pud = np.maximum(c(wpud) + (over_kg - c(fwpud) * T(P.dtime)), T(0))
    wflo[:, 0] = wflo[:, 0] + over_kg * T(1.0 / P.dtime) - c(fwpud)
    return out, pud, wflo


def _case(regime, n=2000):
    wl = synth.make_workload(n, 1, seed=7)
    rng = np.random.default_rng(3)
    lo, hi = {"mixed": (0.05, 1.0), "wet": (0.9, 1.0), "dry": (0.05, 0.4)}[regime]
    w = rng.uniform(lo, hi, size=(n, NL)).astype(np.float32).astype(np.float64)
    wi = np.where(rng.uniform(size=(n, NL)) < 0.2, rng.uniform(0, 0.5, size=(n, NL)), 0.0)
    por = wl.stat["poros"][:, :NL]
    pflo = np.maximum(por * np.maximum(1 - wi, wl.params.epsilon), wl.params.epsilon)
    S = {k: wl.stat[k][:, :NL] for k in ("hydraul", "suction", "bex")}
    return (w, wi, por, pflo, S, np.asarray(wl.params.hsoi[:NL], np.float64), rng.uniform(0, 2e-5, n),
            rng.uniform(0, 1e-5, n), rng.uniform(0, 5, n), wl.params)


@pytest.mark.parametrize("regime", ["dry", "wet", "mixed"])
def test_in_float64_it_is_the_oracles_solve(regime):
    args = _case(regime)
    for got, want, bound in zip(pairs(*args), soil_water(*args), (1e-13, 1e-12, None)):
        assert np.abs(got - want).max() <= (1e-10 * np.abs(want).max() if bound is None else bound)


@pytest.mark.parametrize("regime", ["dry", "wet", "mixed"])
def test_in_float32_it_keeps_the_increment_forms_bounds(regime):
    args = _case(regime)
    w0, _, f0 = soil_water(*args)
    w, _, f = pairs(*args, T=np.float32)
    assert w.dtype == f.dtype == np.float32
    assert np.abs(w.astype(np.float64) - w0).max() <= 6e-7
    assert np.abs(f.astype(np.float64) - f0).max() <= 1e-5 * np.abs(f0).max()
