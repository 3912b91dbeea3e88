"""The largest fixed-bin search atb_search_curve_static accepts: a period's bins and two
more entries fill the shared memory that each of two CTAs per SM can have.  A
caller that sized its bins to that limit must not be refused by a later build."""
import numpy as np
import pytest

import recipes as R
from astro_transit_gpu_b200.engine import SearchConfig
from oracle import oracle as O
from test_zz_no_alloc import FIELDS, call_static

pytestmark = pytest.mark.gpu

LARGEST_FIXED = 6813


def test_largest_fixed_bin_count_is_accepted():
    t, y, dy = R.sector_curve(n=3000, seed=8)
    y = y.astype(np.float32)
    w = (1.0 / dy ** 2).astype(np.float32)
    per = R.sector_periods(40)
    rc, err, out = call_static(t, y, w, per, R.SECTOR_DURATIONS,
                               SearchConfig("fast", n_bins=LARGEST_FIXED))
    assert rc == 0, err
    ora = O.eng_fixed(t, y, w, per, R.SECTOR_DURATIONS, n_bins=LARGEST_FIXED)
    for f in FIELDS:
        assert np.array_equal(out[f], ora[f]), f


def test_more_bins_than_that_are_refused():
    t, y, _ = R.sector_curve(n=300, seed=9)
    rc, err, _ = call_static(t, y.astype(np.float32), None, R.sector_periods(4),
                             R.SECTOR_DURATIONS, SearchConfig("fast", n_bins=LARGEST_FIXED + 100))
    assert rc == 1 and err
