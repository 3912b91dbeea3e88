"""GPU tests of the prefix-gather search (csrc/bls_gather.cuh).

Dense, time-ordered curves of a batch with enough periods are searched by table
look-ups instead of scattered histograms.  The result is the same, bit for bit:
every output is compared with the oracle's mirror of the engine arithmetic, and
with the engine's no-allocation entry shape (the scatter path) where the oracle
would be slow.  The shapes are those where a look-up can go wrong: boundaries that fall on
points (times and bins on one grid), several points in a cell, points in the
trash slot, the V42 padding at the end of the period, windows as long as the
period or as the buffer, one cycle, periods beyond the time span, flat flux
(every window ties) and weighted curves.
"""
import numpy as np
import pytest

import recipes as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")
COPIES = 48    # curves of a batch and
N_PER = 1600   # periods of each, most of them fillers: enough work for the tables to pay


@pytest.fixture(scope="module")
def engine():
    from astro_transit_gpu_b200.engine import BLSEngine
    return BLSEngine.get()


def search(engine, t, y, w, periods, durs, cfg):
    """`COPIES` equal curves whose grids are `periods` and fillers; the checked
    periods' outputs of every copy must agree."""
    from astro_transit_gpu_b200.engine import CurveBatch, split_outputs
    fill = np.geomspace(0.9, 2.2, N_PER - len(periods))
    grid = np.concatenate([periods, fill])
    b = CurveBatch.from_arrays([t] * COPIES, [np.asarray(y, np.float32)] * COPIES, periods=grid,
                               durations=durs, weights=None if w is None else [w] * COPIES)
    outs = split_outputs(b, engine.search(b, cfg))
    for o in outs[1:]:
        for f in FIELDS:
            assert np.array_equal(o[f], outs[0][f]), f
    return {f: outs[0][f][:len(periods)] for f in FIELDS}


def check(engine, t, y, w, periods, durs, cfg):
    periods = np.asarray(periods, np.float64)
    durs = np.asarray(durs, np.float64)
    got = search(engine, t, y, w, periods, durs, cfg)
    y32 = np.asarray(y, np.float32)
    if cfg.method == "fast":
        ora = O.eng_fixed(t, y32, w, periods, durs, n_bins=cfg.n_bins)
    else:
        ora = O.eng_binned(t, y32, w, periods, durs, objective=cfg.objective or "snr",
                           max_bins=cfg.max_bins or 0, oversample=cfg.oversample)
    for f in FIELDS:
        bad = np.flatnonzero(got[f] != ora[f])
        assert bad.size == 0, (f, bad[:5], got[f][bad[:5]], ora[f][bad[:5]])


def config(kind, **kw):
    from astro_transit_gpu_b200.engine import SearchConfig
    if kind == "fixed":
        return SearchConfig("fast", n_bins=kw.get("n_bins", 200))
    return SearchConfig("parity", objective=kw.get("objective", "likelihood"),
                        max_bins=kw.get("max_bins"), oversample=kw.get("oversample", 10))


def curve(kind, n=14001, seed=3):
    """(t, y, dy): a 2-minute curve of one sector, by kind."""
    rng = np.random.default_rng(seed)
    g = R.cadence_grid()
    if kind == "grid":          # t - t[0] and the bins are multiples of one step
        t = np.arange(n) * 0.002
    elif kind == "contiguous":  # every cadence, barycentric
        t = g[:n] + 0.0055 * np.sin(2 * np.pi * g[:n] / 365.25)
    else:
        t = g[np.sort(rng.choice(g.size, n, replace=False))]
        t = t + 0.0055 * np.sin(2 * np.pi * t / 365.25 + 0.3)
    if kind == "doubled":       # a few points share a time or nearly do
        t[1000:1008] = t[1000]
        t[5000] = t[4999] + 1e-9
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y = R.inject_box(t, y, 3.71, t[0] + 1.2, 0.10, 1.5e-3)
    if kind == "flat":
        y[:] = 1.0
    if kind == "plateaus":
        y = R.inject_box(t, np.ones(n), 2.5, t[0] + 0.7, 0.2, 1e-2)
    if kind == "flare":
        y[700:704] += 5.0
    return t, y, np.full(n, 1e-3)


PERIODS = [0.9, 1.0, 1.28, 1.999, 2.0, 2.5, 3.71, 5.0, 6.001, 9.13, 12.4, 13.7, 27.0, 26.39, 40.0,
           0.13, 0.25, 0.5, 0.5004]
DURS = [0.04, 0.06, 0.08, 0.12, 0.16, 0.20]


@pytest.mark.parametrize("weights", ["uniform", "point", None])
@pytest.mark.parametrize("kind", ["sampled", "contiguous", "grid", "doubled", "flat", "plateaus",
                                  "flare"])
def test_astropy_bins_equal_the_oracle(engine, kind, weights):
    t, y, dy = curve(kind)
    rng = np.random.default_rng(7)
    if weights == "point":
        dy = dy * rng.uniform(0.7, 1.4, dy.size)
    w = None if weights is None else (1.0 / dy ** 2).astype(np.float32)
    check(engine, t, y, w, PERIODS, DURS, config("binned"))


@pytest.mark.parametrize("durs,kw", [
    ([0.04], {}),
    ([0.04, 0.05], {"objective": "snr"}),
    ([0.04, 0.77], {}),                        # windows of 192 bins: the longest kept
    ([0.04, 0.78], {}),                        # longer: scattered
    ([0.02 * 2 ** (i / 2) for i in range(7)], {"oversample": 5}),
    ([0.064, 0.2], {"oversample": 16}),
    ([0.04, 0.3, 5.0], {}),                    # longer than short periods
    (DURS, {"max_bins": 300}),                 # capped: the last bin collects the rest
    (DURS, {"max_bins": 2000}),
])
def test_window_lengths_and_caps(engine, durs, kw):
    t, y, dy = curve("sampled", n=15003, seed=5)
    w = (1.0 / dy ** 2).astype(np.float32)
    check(engine, t, y, w, PERIODS, durs, config("binned", **kw))


@pytest.mark.parametrize("n_bins", [2, 31, 127, 200, 300, 511, 512])
@pytest.mark.parametrize("kind,weights", [("sampled", "uniform"), ("grid", "uniform"),
                                          ("doubled", "point"), ("flat", None)])
def test_fixed_bins_equal_the_oracle(engine, kind, weights, n_bins):
    n = 16000
    t, y, dy = curve(kind, n=n, seed=9)
    rng = np.random.default_rng(8)
    if weights == "point":
        dy = dy * rng.uniform(0.7, 1.4, n)
    w = None if weights is None else (1.0 / dy ** 2).astype(np.float32)
    check(engine, t, y, w, PERIODS, DURS, config("fixed", n_bins=n_bins))


def test_bin_counts_that_fill_the_prefix_buffer(engine):
    """Every bin count around whole look-up steps (128 boundaries) and around the
    buffer's 384 entries, neighbours side by side in one batch."""
    t, y, dy = curve("sampled", n=15003, seed=11)
    w = (1.0 / dy ** 2).astype(np.float32)
    bins = np.concatenate([np.arange(110, 146), np.arange(240, 272), np.arange(368, 400),
                           np.arange(500, 524), np.arange(620, 664)])
    check(engine, t, y, w, (bins - 10.5) * 0.004, DURS, config("binned"))


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8191, 16384])
def test_sizes_around_the_shortest_table(engine, n):
    t, y, dy = curve("contiguous", n=n, seed=n)
    w = (1.0 / dy ** 2).astype(np.float32)
    check(engine, t, y, w, PERIODS, DURS, config("binned"))
    check(engine, t, y, w, PERIODS, DURS, config("fixed"))
