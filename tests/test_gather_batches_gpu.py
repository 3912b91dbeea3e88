"""GPU tests of the prefix-gather search on batches of unlike curves.

The search tables of a batch lie one after another in shared arrays, so a curve
that is not gathered must leave its neighbours' tables alone, and its own periods
must go to the scatter kernel.  Every comparison is exact: the search sums are
integers, whichever kernel takes a period.
"""
import numpy as np
import pytest

import recipes as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")
DURS = np.array([0.04, 0.06, 0.08, 0.12, 0.16, 0.20])
CHECKED = np.array([0.9, 1.999, 3.71, 5.0, 9.13, 12.4, 13.7, 27.0])
N_PER = 1600


@pytest.fixture(scope="module")
def engine():
    from astro_transit_gpu_b200.engine import BLSEngine
    return BLSEngine.get()


def config(kind, n_bins=200):
    from astro_transit_gpu_b200.engine import SearchConfig
    if kind == "fixed":
        return SearchConfig("fast", n_bins=n_bins)
    return SearchConfig("parity", objective="likelihood")


def grid(kind):
    """The checked periods and fillers whose look-ups are few against their points."""
    lo, hi = (6.0, 13.0) if kind == "fixed" else (0.9, 2.2)
    return np.concatenate([CHECKED, np.geomspace(lo, hi, N_PER - len(CHECKED))])


def dense_curve(seed, n=14001):
    rng = np.random.default_rng(seed)
    g = R.cadence_grid()
    t = g[:n] + 0.0055 * np.sin(2 * np.pi * g[:n] / 365.25 + seed)
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    return t, R.inject_box(t, y, 3.71, t[0] + 1.2, 0.10, 1.5e-3).astype(np.float32)


def oracle_outputs(kind, t, y, w):
    if kind == "fixed":
        return O.eng_fixed(t, y, w, CHECKED, DURS, n_bins=200)
    return O.eng_binned(t, y, w, CHECKED, DURS, objective="likelihood")


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("kind", ["binned", "fixed"])
def test_empty_curves_between_dense_ones(engine, kind, weighted):
    """A curve without points gives zeros and leaves its neighbours' results alone."""
    from astro_transit_gpu_b200.engine import CurveBatch, split_outputs
    a, b = dense_curve(1), dense_curve(2, 14337)
    none = (np.zeros(0), np.zeros(0, np.float32))
    curves = [none] + [a, b] * 12 + [none, none] + [b, a] * 12 + [none]
    weight = lambda c: np.full(len(c[0]), 1.0e6, np.float32)  # noqa: E731
    batch = CurveBatch.from_arrays([c[0] for c in curves], [c[1] for c in curves],
                                   periods=grid(kind), durations=DURS,
                                   weights=[weight(c) for c in curves] if weighted else None)
    outs = split_outputs(batch, engine.search(batch, config(kind)))
    want = {id(c): oracle_outputs(kind, *c, weight(c) if weighted else None) for c in (a, b)}
    for c, o in zip(curves, outs):
        for f in FIELDS:
            if c is none:
                assert np.all(o[f] == (-1 if f == "window" else 0)), f
            else:
                assert np.array_equal(o[f][:len(CHECKED)], want[id(c)][f]), f


def test_plans_of_other_bin_counts_leave_a_plan_usable(engine):
    """The gather kernel's shared memory grows with the bin count; plans of fewer
    and of more bins, made later, must not change what an earlier plan may use."""
    from astro_transit_gpu_b200.engine import CurveBatch, split_outputs
    t, y = dense_curve(3)
    batch = CurveBatch.from_arrays([t] * 8, [y] * 8, periods=grid("fixed"), durations=DURS)
    plans = [engine.plan(batch, config("fixed", n)) for n in (500, 100, 300)]
    want = [O.eng_fixed(t, y, None, CHECKED, DURS, n_bins=n) for n in (500, 100, 300)]
    try:
        for i in (0, 2, 1, 0):
            plans[i].execute()
            plans[i].check()
            for o in split_outputs(batch, plans[i].outputs):
                for f in FIELDS:
                    assert np.array_equal(o[f][:len(CHECKED)], want[i][f]), (i, f)
    finally:
        for p in plans:
            p.close()


def test_more_gathered_periods_than_32_bits_count(engine):
    """2^16 targets screened over 2^16 periods: 2^32 gathered periods.  The periods
    exceed the time span and the bins are two, so each takes 128 look-ups."""
    import torch
    from astro_transit_gpu_b200.engine import CurveBatch
    nc, n, n_per = 1 << 16, 4096, 1 << 16
    dev = engine.device
    t = np.arange(n) * 0.01
    periods = np.geomspace(1.1, 3.0, n_per) * t[-1]
    dur = np.array([0.2 * t[-1]])
    gen = torch.Generator(dev).manual_seed(5)
    y = torch.randn(nc * n, generator=gen, device=dev, dtype=torch.float32)
    batch = CurveBatch(
        t=torch.from_numpy(t).to(dev), y=y, w=None, periods=torch.from_numpy(periods).to(dev),
        durations=torch.from_numpy(dur).to(dev), point_offset=np.arange(nc + 1, dtype=np.int64) * n,
        period_begin=np.zeros(nc, np.int64), period_count=np.full(nc, n_per, np.int64),
        dur_begin=np.zeros(nc, np.int64), dur_count=np.ones(nc, np.int32),
        out_begin=np.zeros(nc, np.int64), time_offset=np.zeros(nc, np.int64))
    key = torch.zeros(nc, dtype=torch.int64, device=dev)
    best = torch.empty(nc, dtype=torch.int32, device=dev)
    plan = engine.plan(batch, config("fixed", 2), {"best_key": key, "best_period": best})
    try:
        plan.execute()
        plan.check()
    finally:
        plan.close()
    got = best.cpu().numpy()
    assert got.min() >= 0
    for c in (0, 1, nc // 2, nc - 1):
        o = O.eng_fixed(t, y[c * n:(c + 1) * n].cpu().numpy(), None, periods, dur, n_bins=2)
        assert got[c] == np.argmax(o["power"]), c
