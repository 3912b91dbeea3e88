"""Exact cadences put points on the bin boundaries of the first cycle, which are the
same for every period; on which side of them a point lies is decided once per curve."""
import numpy as np
import pytest

import test_gather_routes_gpu as G

pytestmark = pytest.mark.gpu
engine = G.engine


@pytest.mark.parametrize("wkind", ["uniform", "point"])
@pytest.mark.parametrize("cadence", [0.0008, 0.001, 0.0004, 0.00075])
def test_points_on_the_first_cycle_s_boundaries(engine, wkind, cadence):
    """Periods that end on a bin boundary, within a few table units (2^-24 of a cell, a
    cell being the bin width over up to eight) of one, and anywhere; one cycle to many."""
    n, b = 15003, 0.004
    unit = b / 5 * 2.0 ** -24
    steps = np.array([0.0, 0.4, 1.0, 2.0, 3.0, 5.0, 7.9, 8.1, 12.0, 40.0, 1e5])
    near = np.concatenate([m * b + s * steps * unit
                           for m in (131, 250, 400.5, 997, 3200) for s in (-1, 1)])
    span = n * cadence
    checked = np.concatenate([near, [0.6123, 0.9 * span, 1.1 * span, 4.0 * span]])
    y = 1.0 + np.random.default_rng(8).normal(0.0, 1e-3, n)
    for t0 in (0.0, 2457000.3):
        t = t0 + np.arange(n) * cadence
        c = (t, G.R.inject_box(t, y, 1.7, t0 + 0.4, 0.1, 2e-3).astype(np.float32))
        grid = np.concatenate([checked, np.geomspace(0.9, 2.2, G.N_PER - len(checked))])
        w = G.weights(wkind, n)
        count = G.compare(engine, [c] * G.COPIES, [w] * G.COPIES, checked, grid, G.DURS,
                          G.config("binned"))
        assert sum(count.values()) in (0, G.COPIES * len(grid))
        if b / 8 <= cadence <= 0.0008:  # (a table has at most eight cells per bin)
            assert count["counting" if wkind == "uniform" else "weighted"] == G.COPIES * len(grid)
