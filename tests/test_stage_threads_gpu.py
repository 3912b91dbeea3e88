"""GPU test of the stage kernel's CTA sizes: 512 or 1024 threads for the curves of a
small batch, by the longest, and 256 where the batch holds more points than one such
curve per SM.  The staged sums are integers, so every size gives the same outputs."""
import numpy as np
import pytest

import recipes as R
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [1, 31, 513, 4097, 17999, 18000])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_every_cta_size_gives_the_oracles_outputs(n, weighted, dtype):
    from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, SearchConfig, split_outputs
    eng = BLSEngine.get()
    rng = np.random.default_rng(n)
    t = np.sort(rng.uniform(0.0, 27.0, n)) + 1325.0
    y = R.inject_box(t, 1.0 + rng.normal(0.0, 1e-3, n), 3.71, t[0] + 1.2, 0.10, 1.5e-3).astype(dtype)
    w = (1.0e6 / rng.uniform(0.7, 1.4, n) ** 2).astype(np.float32) if weighted else None
    per = np.array([0.7, 1.9, 3.71, 8.8])
    for copies in (1, 160):
        b = CurveBatch.from_arrays([t] * copies, [y] * copies, periods=per,
                                   durations=R.SECTOR_DURATIONS, flux_dtype=dtype,
                                   weights=None if w is None else [w] * copies)
        for cfg, ora in ((SearchConfig("parity", objective="likelihood"),
                          O.eng_binned(t, y, w, per, R.SECTOR_DURATIONS, objective="likelihood")),
                         (SearchConfig("fast", n_bins=150),
                          O.eng_fixed(t, y, w, per, R.SECTOR_DURATIONS, n_bins=150))):
            for o in split_outputs(b, eng.search(b, cfg)):
                for f in FIELDS:
                    assert np.array_equal(o[f], ora[f]), (copies, cfg.method, f)
