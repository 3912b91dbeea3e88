"""Timed cases of the Box Least Squares engine: what its users run, from one
short light curve through the drop-in API to uneven batches of many sectors.

Sizes are those of this repository's benchmark and tests: single-sector curves
(27.4 d, 2-minute cadence, 15 000 points, 5000 periods 0.5-13.7 d, six
durations), the uneven batch (1-13 sectors, 2- or 30-minute cadence, per-curve
frequency-uniform grids, eight durations 0.02-0.30 d), the screening shape
(1312 points, 128 bins) and the 2000-point curve of the parity tests.  Times
are cadence grids with mid-sector gaps and dropped cadences, on a barycentric
time axis (the light-travel term moves the cadence by 1e-4), as survey
pipelines deliver them; flux is white noise, some curves with a box transit.

A case is a dict of plain values:
  entry     how the search is called: "power" (BoxLeastSquaresGPU.power on host
            arrays), "power_batch" (host arrays), "targets"
            (run_vbls_exact_parity on host arrays), "plan" (a kept plan on
            device tensors), "screen" (BLSEngine.screen on device tensors),
            "session" (PipelinedSession: pinned host inputs to pinned outputs)
  method    "parity" or "fast";  objective, max_bins, n_bins as SearchConfig
  curves, sectors, cadence_min, points, periods, pmin, pmax, durations;
            sectors = 0: each curve has its own sectors, cadence, points (1000
            to what its cadences allow) and periods, drawn from `shapes`
  errors    "uniform" (one error per curve), "point" (one per point), "none"
  flux      "f32" or "f64"
"""
from __future__ import annotations

import math
from typing import Any, Dict, List, Optional

import numpy as np
import torch

from astro_transit_gpu_b200 import BoxLeastSquaresGPU, power_batch, run_vbls_exact_parity
from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, PipelinedSession, SearchConfig

SECTOR_DAYS = 27.4
GAP_DAYS = 1.0
FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")
SECTOR_DURATIONS = (0.04, 0.06, 0.08, 0.12, 0.16, 0.20)


def listed() -> List[Dict[str, Any]]:
    return [
        # the smallest call: a 2000-point curve, default method, host arrays in and out
        dict(name="one_short_fast", entry="power", method="fast", objective="fast", n_bins=200,
             max_bins=0, curves=1, sectors=1, cadence_min=18.0, points=2000, periods=1000,
             pmin=3.0, pmax=4.0, durations=3, errors="uniform", flux="f64"),
        # one sector curve with per-point errors through the drop-in API, reference defaults
        dict(name="one_sector_parity", entry="power", method="parity", objective="snr", n_bins=0,
             max_bins=2000, curves=1, sectors=1, cadence_min=2.0, points=15000, periods=5000,
             pmin=0.5, pmax=13.7, durations=6, errors="point", flux="f32"),
        # the benchmark's batch: one error per curve, likelihood objective, no bin cap
        dict(name="sector_batch_parity", entry="plan", method="parity", objective="likelihood",
             n_bins=0, max_bins=0, curves=128, sectors=1, cadence_min=2.0, points=15000,
             periods=5000, pmin=0.5, pmax=13.7, durations=6, errors="uniform", flux="f32"),
        # the same curves with the default (fast) method
        dict(name="sector_batch_fast", entry="plan", method="fast", objective="fast", n_bins=200,
             max_bins=0, curves=192, sectors=1, cadence_min=2.0, points=15000, periods=5000,
             pmin=0.5, pmax=13.7, durations=6, errors="uniform", flux="f32"),
        # pipeline photometry carries one error per point: weighted curves, odd sizes
        dict(name="weighted_batch_parity", entry="plan", method="parity", objective="snr",
             n_bins=0, max_bins=0, curves=64, sectors=1, cadence_min=2.0, points=17011,
             periods=4001, pmin=0.5, pmax=13.7, durations=5, errors="point", flux="f64"),
        dict(name="weighted_batch_fast", entry="plan", method="fast", objective="fast",
             n_bins=300, max_bins=0, curves=64, sectors=2, cadence_min=2.0, points=30001,
             periods=4999, pmin=0.5, pmax=20.0, durations=8, errors="point", flux="f32"),
        # the uneven batch: 1-13 sectors, 2- and 30-minute cadence, one grid per curve
        dict(name="uneven_parity", entry="plan", method="parity", objective="likelihood",
             n_bins=0, max_bins=0, curves=96, sectors=0, cadence_min=0.0, points=0, periods=0,
             shapes=2, pmin=0.5, pmax=0.0, durations=8, errors="uniform", flux="f32"),
        dict(name="uneven_fast", entry="plan", method="fast", objective="fast", n_bins=200,
             max_bins=0, curves=96, sectors=0, cadence_min=0.0, points=0, periods=0,
             shapes=2, pmin=0.5, pmax=0.0, durations=8, errors="uniform", flux="f32"),
        # full-frame-image targets of one sector on their shared time axis, host arrays
        dict(name="ffi_targets", entry="targets", method="parity", objective="snr", n_bins=0,
             max_bins=2000, curves=256, sectors=1, cadence_min=30.0, points=1200, periods=2000,
             pmin=0.5, pmax=13.0, durations=5, errors="point", flux="f32"),
        # winner-take-all screening: many periods, only the best record per target
        dict(name="screen", entry="screen", method="fast", objective="fast", n_bins=128,
             max_bins=0, curves=96, sectors=1, cadence_min=27.0, points=1312, periods=20000,
             pmin=0.5, pmax=13.0, durations=8, errors="uniform", flux="f32"),
        # a year of 2-minute data: long curves, long periods, fine bins
        dict(name="year_parity", entry="plan", method="parity", objective="likelihood", n_bins=0,
             max_bins=0, curves=2, sectors=13, cadence_min=2.0, points=200000, periods=10000,
             pmin=0.5, pmax=150.0, durations=8, errors="uniform", flux="f32"),
        # end to end: curves from pinned host memory, every output back to the host
        dict(name="session_parity", entry="session", method="parity", objective="likelihood",
             n_bins=0, max_bins=0, curves=96, sectors=1, cadence_min=2.0, points=15000,
             periods=5000, pmin=0.5, pmax=13.7, durations=6, errors="uniform", flux="f32"),
    ]


def _loguniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> Dict[str, Any]:
    kind = rng.choice(("one", "one", "sector", "sector", "sector", "uneven", "ffi", "screen",
                       "year", "session", "batch"))
    method = rng.choice(("parity", "fast"))
    c: Dict[str, Any] = dict(method=method, errors=rng.choice(("uniform", "point", "none")),
                             flux=rng.choice(("f32", "f64")), pmin=rng.uniform(0.4, 0.8))
    if kind == "uneven":
        c.update(entry="plan", curves=rng.randint(24, 72), sectors=0, cadence_min=0.0, points=0,
                 periods=0, shapes=rng.randint(3, 1 << 30), pmax=0.0,
                 durations=rng.randint(4, 8))
    elif kind == "ffi":
        method = c["method"] = "parity"
        c.update(entry="targets", errors=rng.choice(("none", "point")),
                 curves=int(_loguniform(rng, 16, 256)), sectors=1, cadence_min=30.0,
                 points=rng.randint(900, 1250), periods=int(_loguniform(rng, 300, 2000)),
                 pmax=rng.uniform(8.0, 13.0), durations=rng.randint(3, 8))
    elif kind == "screen":
        c.update(entry="screen", curves=rng.randint(16, 96), sectors=1, cadence_min=27.0,
                 points=rng.randint(1000, 1350), periods=int(_loguniform(rng, 2000, 20000)),
                 pmax=rng.uniform(8.0, 13.0), durations=rng.randint(3, 8))
        method = c["method"] = "fast"
    elif kind == "year":
        c.update(entry="plan", curves=rng.randint(1, 2), sectors=rng.randint(6, 13),
                 cadence_min=2.0, points=int(_loguniform(rng, 60000, 110000)),
                 periods=int(_loguniform(rng, 2000, 10000)), pmax=rng.uniform(30.0, 80.0),
                 durations=rng.randint(4, 8))
    elif kind == "one":
        c.update(entry="power", curves=1, sectors=1, cadence_min=rng.choice((2.0, 10.0)),
                 points=int(_loguniform(rng, 1000, 3500)),
                 periods=int(_loguniform(rng, 500, 10000)), pmax=rng.uniform(4.0, 13.7),
                 durations=rng.randint(3, 8))
        if c["cadence_min"] == 2.0:
            c["points"] = int(_loguniform(rng, 4000, 18000))
    else:
        entry = {"sector": "plan", "session": "session", "batch": "power_batch"}[kind]
        c.update(entry=entry, curves=int(_loguniform(rng, 8, 96)), sectors=rng.randint(1, 3),
                 cadence_min=rng.choice((2.0, 2.0, 10.0)), points=0,
                 periods=int(_loguniform(rng, 1000, 5000)), pmax=rng.uniform(6.0, 13.7),
                 durations=rng.randint(3, 8))
        full = c["sectors"] * (SECTOR_DAYS - GAP_DAYS) * 1440.0 / c["cadence_min"]
        c["points"] = int(full * rng.uniform(0.6, 0.98))
    if method == "fast":
        c.update(objective="fast", n_bins=int(_loguniform(rng, 100, 500)), max_bins=0)
    else:
        c.update(objective=rng.choice(("snr", "likelihood")), n_bins=0,
                 max_bins=rng.choice((0, 0, 2000)))
        if c["entry"] == "targets":
            c["max_bins"] = 2000
    return c


# ------------------------------------------------------------------ inputs ---

def _spec(case):
    """(sectors, cadence in days, points, periods) of every curve."""
    rng = np.random.default_rng(case.get("shapes", 0))
    out = []
    for _ in range(case["curves"]):
        n_sec, cad = case["sectors"], case["cadence_min"] / 1440.0
        if n_sec == 0:
            n_sec = int(rng.integers(1, 14))
            cad = (2.0 if rng.uniform() < 0.5 else 30.0) / 1440.0
        avail = int(n_sec * (SECTOR_DAYS - GAP_DAYS) / cad)
        n = case["points"]
        if n == 0:
            n = int(np.exp(rng.uniform(np.log(1e3), np.log(2e5))))
        n = min(n, avail)
        base = n_sec * SECTOR_DAYS
        n_per = case["periods"]
        if n_per == 0:
            n_per = int(np.clip((2.0 - 2.0 / base) * 84.0 * base, 1000, 60000))
        out.append((n_sec, cad, n, n_per))
    return out


def _durations(case) -> np.ndarray:
    if case["sectors"] == 1 and case["durations"] == 6:
        return np.array(SECTOR_DURATIONS)
    if case["sectors"] in (0, 13):
        return np.geomspace(0.02, 0.3, case["durations"])
    return np.linspace(0.04, 0.25, case["durations"])


def _periods(case, n_sec, n_per) -> np.ndarray:
    pmax = case["pmax"] or 0.5 * n_sec * SECTOR_DAYS
    if case["sectors"] == 1:
        return np.geomspace(case["pmin"], pmax, n_per)
    return 1.0 / np.linspace(1.0 / case["pmin"], 1.0 / pmax, n_per)


def _inputs(case, seed) -> Dict[str, Any]:
    """Host arrays: per-curve lists t, y, dy (None without errors), periods
    (one grid, or one per curve when the curves differ) and durations."""
    rng = np.random.default_rng([int(seed), 2])
    shared = case["entry"] == "targets"
    spec = _spec(case)
    fdt = np.float64 if case["flux"] == "f64" else np.float32
    ts, ys, es, ps = [], [], [], []
    for c, (n_sec, cad, n, n_per) in enumerate(spec):
        if c == 0 or not shared:
            off = rng.uniform(1300.0, 2700.0)
            g = np.arange(0.0, SECTOR_DAYS, cad)
            g = g[(g < 0.5 * (SECTOR_DAYS - GAP_DAYS)) | (g >= 0.5 * (SECTOR_DAYS + GAP_DAYS))]
            g = np.concatenate([off + s * SECTOR_DAYS + g for s in range(n_sec)])
            keep = rng.random(g.size).argpartition(n - 1)[:n] if n < g.size else np.arange(g.size)
            t = np.sort(g[keep])
            # barycentric light-travel time
            t = t + 0.0055 * np.sin(2 * np.pi * t / 365.25 + rng.uniform(0.0, 2 * np.pi))
        sig = math.exp(rng.uniform(math.log(2e-4), math.log(5e-3)))
        dy = None
        if case["errors"] == "point":
            dy = (sig * rng.uniform(0.8, 1.25, t.size)).astype(np.float32)
        elif case["errors"] == "uniform":
            dy = np.full(t.size, sig, np.float32)
        y = 1.0 + rng.standard_normal(t.size, dtype=np.float32) * (sig if dy is None else dy)
        if rng.uniform() < 0.3:
            period = rng.uniform(0.5, min(13.0, 0.5 * n_sec * SECTOR_DAYS))
            ph = (t - t[0] - rng.uniform(0.0, period) + 0.5 * period) % period - 0.5 * period
            y[np.abs(ph) < 0.5 * rng.uniform(0.03, 0.25)] *= 1.0 - rng.uniform(3e-4, 1e-2)
        ts.append(t)
        ys.append(y.astype(fdt))
        es.append(dy)
        ps.append(_periods(case, n_sec, n_per))
    one_grid = case["sectors"] != 0
    return {"t": ts, "y": ys, "dy": None if case["errors"] == "none" else es,
            "periods": ps[0] if one_grid else ps, "durations": _durations(case)}


def _weights(dy) -> np.ndarray:
    dy = np.asarray(dy, np.float64)
    return (1.0 / (dy * dy)).astype(np.float32)


def _config(case) -> SearchConfig:
    if case["method"] == "fast":
        return SearchConfig("fast", n_bins=case["n_bins"])
    return SearchConfig("parity", objective=case["objective"], max_bins=case["max_bins"] or None)


def prepare(case, seed) -> Dict[str, Any]:
    """What a program holds before the call: host arrays for the host entry
    points, a batch or plan on the device, or a session with loaded inputs."""
    inp = _inputs(case, seed)
    entry = case["entry"]
    state: Dict[str, Any] = {"case": case}
    if entry in ("power", "power_batch"):
        return {**state, "inputs": inp}
    if entry == "targets":
        state["time"] = inp["t"][0]
        state["flux"] = np.stack(inp["y"])
        state["weights"] = None if inp["dy"] is None else np.stack([_weights(e) for e in inp["dy"]])
        state["periods"], state["durations"] = inp["periods"], inp["durations"]
        return state
    engine = BLSEngine.get()
    fdt = np.float64 if case["flux"] == "f64" else np.float32
    if entry == "session":
        pt = np.concatenate([[0], np.cumsum([len(t) for t in inp["t"]])])
        s = PipelinedSession(engine, pt, inp["periods"], inp["durations"], _config(case),
                             parts=4, y_dtype=fdt, weighted=inp["dy"] is not None)
        s.load(np.concatenate(inp["t"]), np.concatenate(inp["y"]),
               None if inp["dy"] is None else np.concatenate([_weights(e) for e in inp["dy"]]))
        return {**state, "session": s}
    batch = CurveBatch.from_arrays(inp["t"], inp["y"], inp["dy"], periods=inp["periods"],
                                   durations=inp["durations"], flux_dtype=fdt)
    state["engine"], state["batch"] = engine, batch
    if entry == "plan":
        state["plan"] = engine.plan(batch, _config(case))
    return state


def _result(r) -> Dict[str, Any]:
    return {"power": r.power, "depth": r.depth, "depth_err": r.depth_err, "t0": r.transit_time,
            "duration": r.duration, "window": r.window,
            "best": np.array([r.best_period, r.best_t0, r.best_duration, r.best_depth,
                              r.best_power])}


def run(state):
    case = state["case"]
    entry = case["entry"]
    kw = {}
    if case["method"] == "fast":
        kw["n_bins"] = case["n_bins"]
    else:
        kw["objective"] = case["objective"]
        kw["max_bins"] = case["max_bins"] or None
    if entry == "power":
        i = state["inputs"]
        bls = BoxLeastSquaresGPU(i["t"][0], i["y"][0], None if i["dy"] is None else i["dy"][0])
        return _result(bls.power(i["periods"], i["durations"], method=case["method"], **kw))
    if entry == "power_batch":
        i = state["inputs"]
        res = [_result(r) for r in power_batch(i["t"], i["y"], i["dy"], periods=i["periods"],
                                               durations=i["durations"], method=case["method"],
                                               **kw)]
        return {k: np.stack([r[k] for r in res]) for k in res[0]}
    if entry == "targets":
        out = run_vbls_exact_parity(state["time"], state["flux"], state["periods"],
                                    state["durations"], state["weights"],
                                    max_bins=case["max_bins"], objective=case["objective"])
        return {k: out[k] for k in ("power_array", "depth_array", "t0_array", "dur_array", "snr",
                                    "best_period")}
    if entry == "session":
        return state["session"].run()
    if entry == "screen":
        return state["engine"].screen(state["batch"], _config(case))
    state["plan"].execute()
    return state["plan"].outputs


def work(case) -> Dict[str, float]:
    """Bytes: every input point (t 8 B, flux, weight) and period read once,
    every output written once.  Operations: one fold of a point costs about
    six (a multiplication, floor, a fused multiply-add, a multiplication, two
    sums); counted for every (point, period) pair."""
    spec = _spec(case)
    per_point = 8 + (8 if case["flux"] == "f64" else 4) + (0 if case["errors"] == "none" else 4)
    points = float(sum(s[2] for s in spec))
    periods = float(sum(s[3] for s in spec))
    out = 0.0 if case["entry"] == "screen" else 28.0 * periods
    return {"bytes": points * per_point + 8.0 * periods + out,
            "flops": 6.0 * float(sum(s[2] * s[3] for s in spec))}


# ------------------------------------------------- the path in 64 bits -------

def _exact_curve(case, t, y, dy, periods, durations, dev) -> Dict[str, np.ndarray]:
    """One curve by the plain definition in float64: fold every point, sum
    weights and weighted flux per bin, evaluate every box."""
    td = torch.from_numpy(np.asarray(t)).to(dev)
    d = td - td[0]
    yd = torch.from_numpy(np.asarray(y, np.float64)).to(dev)
    w = (torch.ones_like(yd) if dy is None else
         torch.from_numpy(_weights(dy).astype(np.float64)).to(dev))
    yd = yd - (w * yd).sum() / w.sum()
    fast = case["method"] == "fast"
    os_ = 10
    bin_dur = float(durations.min()) / os_
    ibd = 1.0 / bin_dur
    nd = len(durations)
    res = {k: np.zeros(len(periods)) for k in ("power", "depth", "depth_err", "t0", "duration")}
    inf = float("inf")
    for p, P in enumerate(np.asarray(periods, np.float64)):
        P = float(P)
        m = d * (1.0 / P)
        k = torch.floor(m)
        if fast:
            nb = case["n_bins"]
            slot = ((m - k) * nb).to(torch.int64) + 1
            size = nb + 2
        else:
            nb = int(math.ceil(P * ibd)) + os_
            if case["max_bins"] and nb >= case["max_bins"]:
                nb = case["max_bins"] - 1
            slot = torch.clamp(((d - P * k) * ibd).to(torch.int64) + 1, 1, nb)
            size = nb + 1
        hw = torch.bincount(slot, w, size)
        hy = torch.bincount(slot, w * yd, size)
        if not fast:  # the first bins repeat at the end of the cycle
            for j in range(1, os_ + 1):
                hw[nb - os_ + j - 1] = hw[j]
                hy[nb - os_ + j - 1] = hy[j]
        cw, cy = torch.cumsum(hw[:nb + 1], 0), torch.cumsum(hy[:nb + 1], 0)
        wt, yt = (cw[nb], cy[nb]) if fast else (w.sum(), (w * yd).sum())
        best = None
        for q in range(nd):
            dur = float(durations[q])
            if fast:
                L = max(1, int(dur / P * nb + 0.5))
                if L >= nb:
                    continue
                s = torch.arange(nb, device=dev)
                e = s + L
                wrap = e > nb
                e = torch.where(wrap, e - nb, e)
                wi = cw[e] - cw[s] + torch.where(wrap, wt, torch.zeros_like(wt))
                si = cy[e] - cy[s] + torch.where(wrap, yt, torch.zeros_like(yt))
            else:
                L = max(1, int(math.floor(dur * ibd + 0.5)))
                if L > nb:
                    continue
                wi, si = cw[L:] - cw[:nb + 1 - L], cy[L:] - cy[:nb + 1 - L]
            wo = wt - wi
            ok = (wi > 1e-9 * wt) & (wo > 1e-9 * wt)
            dep = (yt - si) / wo - si / wi
            score = dep * dep * wi * wo
            if not fast:
                ok &= dep >= 0
            score = torch.where(ok, score, torch.full_like(score, -inf))
            v, i = torch.max(score, 0)
            best_q = torch.stack([v, i.to(v.dtype), wi[i], wo[i], dep[i],
                                  torch.full_like(v, float(q)), torch.full_like(v, float(L))])
            best = best_q if best is None else torch.where(best_q[0] > best[0], best_q, best)
        v, s, wi, wo, dep, q, L = best.tolist()
        if v == -inf:
            continue
        err = math.sqrt(1.0 / wi + 1.0 / wo)
        res["power"][p] = (math.sqrt(max(dep * dep * wi * wo, 0.0)) if fast else
                           0.5 * dep * dep * wi * wo / (wi + wo)
                           if case["objective"] == "likelihood" else dep / err)
        res["depth"][p], res["depth_err"][p] = dep, err
        if fast:
            res["duration"][p] = durations[int(q)]
            res["t0"][p] = s / nb * P + t[0]
        else:
            res["duration"][p] = L * bin_dur
            res["t0"][p] = math.fmod(s * bin_dur + 0.5 * L * bin_dur + t[0], P)
    return res


def exact(case, seed) -> Optional[Any]:
    """The path in 64 bits with torch, for the cases of one or a few curves
    (a period at a time: longer ones would take minutes)."""
    spec = _spec(case)
    if case["entry"] != "power" or sum(s[3] for s in spec) > 5000:
        return None
    inp = _inputs(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    r = _exact_curve(case, inp["t"][0], inp["y"][0],
                     None if inp["dy"] is None else inp["dy"][0], inp["periods"],
                     inp["durations"], dev)
    b = int(np.argmax(r["power"]))
    return {"power": r["power"], "depth": r["depth"], "depth_err": r["depth_err"], "t0": r["t0"],
            "duration": r["duration"], "window": None,
            "best": np.array([inp["periods"][b], r["t0"][b], r["duration"][b], r["depth"][b],
                              r["power"][b]])}
