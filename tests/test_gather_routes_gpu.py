"""GPU tests of the prefix-gather search that make sure it ran.

Each batch is dense enough, and has periods enough, for the tables to pay; the
number of periods the gather kernel took (`SearchPlan.gathered`) is asserted.  Its
outputs are compared bit for bit with those of the same plan without tables (every
period of every curve scattered) and, on the checked periods, with the oracle's
mirror of the engine arithmetic.  Both kernels add exact integers, so nothing may
differ.  The curves are those where a look-up can go wrong: points on bin
boundaries, several points in a cell, points in the trash slot, bins on either side of
whole look-up blocks, periods beyond the span, equal windows, unequal weights.
"""
import numpy as np
import pytest

import recipes as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")
COPIES = 48
N_PER = 1600
CHECKED = np.array([0.9, 1.0, 1.28, 1.999, 2.0, 2.5, 3.71, 5.0, 6.001, 9.13, 12.4, 13.7, 27.0,
                    26.39, 40.0, 0.13, 0.25, 0.5, 0.5004])
DURS = np.array([0.04, 0.06, 0.08, 0.12, 0.16, 0.20])
KINDS = ["sampled", "contiguous", "grid", "doubled", "flat", "plateaus", "flare", "spike"]


@pytest.fixture(scope="module")
def engine():
    from astro_transit_gpu_b200.engine import BLSEngine
    return BLSEngine.get()


def config(geom, **kw):
    from astro_transit_gpu_b200.engine import SearchConfig
    if geom == "fixed":
        return SearchConfig("fast", n_bins=kw.get("n_bins", 200))
    return SearchConfig("parity", objective=kw.get("objective", "likelihood"),
                        max_bins=kw.get("max_bins"), oversample=kw.get("oversample", 10))


def curve(kind, n, cadence, seed):
    rng = np.random.default_rng(seed)
    if kind in ("grid", "spike"):  # times and bins are multiples of one step
        t = np.arange(n) * cadence
    else:
        g = np.arange(n + n // 10) * cadence + 1400.0
        t = g[:n] if kind == "contiguous" else g[np.sort(rng.choice(g.size, n, replace=False))]
        t = t + 0.0055 * np.sin(2 * np.pi * t / 365.25 + 0.3)
    if kind == "doubled":  # a few points share a time or nearly do
        t[1000:1006] = t[1000]
        t[3000] = t[2999] + 1e-9
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y = R.inject_box(t, y, 3.71, t[0] + 1.2, 0.10, 1.5e-3)
    if kind == "flat":
        y[:] = 1.0
    if kind == "plateaus":
        y = R.inject_box(t, np.ones(n), 2.5, t[0] + 0.7, 0.2, 1e-2)
    if kind == "spike":  # equal but for one point: windows tie by the hundred
        y[:] = 1.0
        y[n // 3] += 1e-3
    if kind == "flare":
        y[700:704] += 5.0
    return t, y.astype(np.float32)


def weights(kind, n, seed=7):
    if kind is None:
        return None
    if kind == "uniform":
        return np.full(n, 1.0e6, np.float32)
    return (1.0e6 / np.random.default_rng(seed).uniform(0.7, 1.4, n) ** 2).astype(np.float32)


def fillers(geom, n, span):
    """Periods whose look-ups are few against their points."""
    return np.geomspace(0.9, 2.2, n) if geom == "binned" else np.geomspace(0.51, 1.5, n) * span


def run(engine, curves, ws, grid, durs, cfg, table_bytes=-1):
    import torch
    from astro_transit_gpu_b200.engine import CurveBatch, split_outputs
    b = CurveBatch.from_arrays([c[0] for c in curves], [c[1] for c in curves], periods=grid,
                               durations=durs, weights=ws)
    plan = engine.plan(b, cfg, stream=torch.cuda.current_stream(), table_bytes=table_bytes)
    try:
        plan.execute()
        plan.check()
        return split_outputs(b, plan.outputs), plan.gathered()
    finally:
        plan.close()


def oracle_outputs(c, w, periods, durs, cfg):
    if cfg.method == "fast":
        return O.eng_fixed(*c, w, periods, durs, n_bins=cfg.n_bins)
    return O.eng_binned(*c, w, periods, durs, objective=cfg.objective,
                        max_bins=cfg.max_bins or 0, oversample=cfg.oversample)


def compare(engine, curves, ws, checked, grid, durs, cfg, oracle_curves=1):
    """Gathered outputs equal the scattered ones everywhere and the oracle's on the
    first curves' checked periods; returns the counts of gathered periods."""
    got, count = run(engine, curves, ws, grid, durs, cfg)
    ref, none = run(engine, curves, ws, grid, durs, cfg, table_bytes=0)
    assert none == {"counting": 0, "weighted": 0, "given_back": 0}
    for c, (o, r) in enumerate(zip(got, ref)):
        for f in FIELDS:
            bad = np.flatnonzero(o[f] != r[f])
            assert bad.size == 0, (c, f, bad[:5], o[f][bad[:5]], r[f][bad[:5]])
    for c in range(oracle_curves):
        ora = oracle_outputs(curves[c], None if ws is None else ws[c], checked, durs, cfg)
        for f in FIELDS:
            assert np.array_equal(got[c][f][:len(checked)], ora[f]), (c, f)
    return count


def check(engine, kind, wkind, geom, durs=DURS, checked=CHECKED, n=15003, **kw):
    """A batch of three curves in turn; every period it can gather is gathered."""
    cadence = {"binned": 0.0008, "fixed": 0.002}[geom]
    three = [curve(kind, n + 64 * i, cadence, 11 + i) for i in range(3)]
    w3 = [weights(wkind, len(c[0])) for c in three]
    curves, ws = three * (COPIES // 3), w3 * (COPIES // 3)
    fill = fillers(geom, N_PER - len(checked), max(c[0].max() - c[0].min() for c in three))
    count = compare(engine, curves, ws if wkind else None, checked,
                    np.concatenate([checked, fill]), durs, config(geom, **kw))
    mine, other = (("weighted", "counting") if wkind == "point" else ("counting", "weighted"))
    assert count[other] == 0
    if kind == "flat" or (geom == "binned" and kind == "doubled"):
        assert count[mine] == 0  # every window equal; points that share a cell
    elif geom == "binned":  # a curve's periods are gathered all (but those of few bins) or none
        assert count[mine] >= COPIES * (N_PER - 4)
    else:                 # the long periods at least
        assert count[mine] >= COPIES * len(fill)
    if kind in ("sampled", "contiguous"):
        assert count["given_back"] == 0
    if kind == "spike" and geom == "binned" and wkind != "point":
        assert count["given_back"] > 0


@pytest.mark.parametrize("wkind", ["uniform", "point", None])
@pytest.mark.parametrize("kind", KINDS)
def test_astropy_bins(engine, kind, wkind):
    check(engine, kind, wkind, "binned")


@pytest.mark.parametrize("n_bins", [2, 127, 128, 200, 300, 511])
@pytest.mark.parametrize("wkind", ["uniform", "point", None])
@pytest.mark.parametrize("kind", KINDS)
def test_fixed_bins(engine, kind, wkind, n_bins):
    # (a period of many bins pays on more points)
    check(engine, kind, wkind, "fixed", n=45003 if n_bins > 300 else 15003, n_bins=n_bins)


@pytest.mark.parametrize("wkind", ["uniform", "point"])
@pytest.mark.parametrize("durs,kw", [
    ([0.04], {}),
    ([0.04, 0.05], {"objective": "snr"}),
    ([0.04, 0.768], {}),                       # windows of 192 bins: the longest kept
    ([0.02 * 2 ** (i / 2) for i in range(7)], {"oversample": 5}),
    ([0.064, 0.2], {"oversample": 16}),
    ([0.04, 0.2], {"max_bins": 300}),          # capped: the last bin collects the rest
])
def test_window_lengths_and_caps(engine, wkind, durs, kw):
    check(engine, "sampled", wkind, "binned", np.array(durs), **kw)


@pytest.mark.parametrize("wkind", ["uniform", "point"])
def test_astropy_bin_counts_that_fill_the_prefix_buffer(engine, wkind):
    bins = np.concatenate([np.arange(110, 146), np.arange(240, 272), np.arange(368, 400),
                           np.arange(500, 524), np.arange(620, 664)])
    check(engine, "sampled", wkind, "binned", checked=(bins - 10.5) * 0.004)


@pytest.mark.parametrize("wkind", ["uniform", "point"])
@pytest.mark.parametrize("n", [4096, 4097, 8191, 16384])
def test_fixed_bins_of_short_and_whole_tables(engine, wkind, n):
    check(engine, "contiguous", wkind, "fixed", n=n, n_bins=100)


@pytest.mark.parametrize("geom", ["binned", "fixed"])
def test_unlike_curves_in_one_batch(engine, geom):
    """Short, sparse, unsorted, flat, empty and dense curves, of equal and of unequal
    weights: every curve's table sits between those of others."""
    cadence = 0.0008 if geom == "binned" else 0.002
    rng = np.random.default_rng(3)
    dense = curve("sampled", 15003, cadence, 1)
    more = curve("doubled", 17001, cadence, 2)
    short = curve("sampled", 1000, cadence, 3)
    sparse = curve("sampled", 4200, 0.02, 4)
    flat = curve("flat", 15003, cadence, 5)
    mixed = tuple(x[rng.permutation(15003)] for x in curve("contiguous", 15003, cadence, 6))
    empty = (np.zeros(0), np.zeros(0, np.float32))
    kinds = [(dense, "uniform"), (short, "point"), (dense, "point"), (mixed, "uniform"),
             (sparse, "point"), (more, "uniform"), (flat, "uniform"), (more, "point"), (empty, "uniform")]
    curves = [c for c, _ in kinds] * 8
    ws = [weights(k, len(c[0])) for c, k in kinds] * 8
    grid = np.concatenate([CHECKED, fillers(geom, N_PER - len(CHECKED), cadence * 15003)])
    count = compare(engine, curves, ws, CHECKED, grid, DURS, config(geom), len(kinds) - 1)
    assert count["counting"] >= 8 * len(grid) / 2
    assert count["weighted"] >= 8 * len(grid) / 2


@pytest.mark.parametrize("decades", [2, 6, 12])
@pytest.mark.parametrize("geom", ["binned", "fixed"])
def test_weights_of_many_magnitudes(engine, geom, decades):
    """The lightest points weigh less than the filter's error, or round to nothing."""
    cadence = 0.0008 if geom == "binned" else 0.002
    three = [curve("sampled", 15003 + 64 * i, cadence, 21 + i) for i in range(3)]
    rng = np.random.default_rng(4)
    w3 = [(1.0e6 * 10.0 ** -rng.uniform(0, decades, len(c[0]))).astype(np.float32) for c in three]
    fill = fillers(geom, N_PER - len(CHECKED), max(c[0].max() - c[0].min() for c in three))
    count = compare(engine, three * 16, w3 * 16, CHECKED, np.concatenate([CHECKED, fill]), DURS,
                    config(geom))
    assert count["weighted"] >= 48 * len(fill)


@pytest.mark.parametrize("wkind", ["uniform", "point"])
def test_spacings_just_below_a_cell(engine, wkind):
    """Spacings of 0.99991 cells: a few points share one, which the table finds out late."""
    n = 15003
    t = np.arange(n) * (0.0008 * 0.99991)
    y = (1.0 + np.random.default_rng(1).normal(0.0, 1e-3, n)).astype(np.float32)
    grid = np.concatenate([CHECKED, fillers("binned", N_PER - len(CHECKED), t[-1])])
    w = weights(wkind, n)
    count = compare(engine, [(t, y)] * COPIES, [w] * COPIES, CHECKED, grid, DURS, config("binned"))
    assert count["counting"] == 0 and count["weighted"] == 0
