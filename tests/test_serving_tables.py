"""Look-up tables never narrow what a server admits, and stay within its budget."""
from collections import namedtuple

import numpy as np
import pytest

from astro_transit_gpu_b200.serving import request_bytes, spare_bytes

R = namedtuple("R", "nbytes")
FIELDS = ("power", "depth", "depth_err", "t0", "duration", "window")


@pytest.mark.parametrize("n", [1000, 4096, 15000, 2**18 - 1, 2**18])
def test_a_dense_request_needs_no_room_for_tables(n):
    # inputs and staged points 32 B, grids and outputs 36 B a period, 8 B a duration
    assert request_bytes(n, 5000, 6) == 32 * n + 36 * 5000 + 48 + 4096


def test_tables_take_half_of_what_nobody_needs():
    assert spare_bytes(1000, 400, []) == 300
    assert spare_bytes(1000, 400, [R(100), R(100)]) == 200
    assert spare_bytes(1000, 900, [R(200)]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("spare", [0, 64 << 20])
def test_budgets_with_and_without_room_for_tables(spare):
    """One dense request of 30 000 periods: admitted by a budget of its own bytes
    (scattered), and searched with tables, which count as held, where the budget has
    room for them.  Same results."""
    from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, SearchConfig
    from astro_transit_gpu_b200.serving import BLSServer
    rng = np.random.default_rng(5)
    n, durs = 15000, np.array([0.04, 0.08, 0.16])
    t = np.arange(n) * (2.0 / 1440.0) + 1500.0
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    per = np.linspace(1.0, 5.0, 30000)
    need = request_bytes(n, len(per), len(durs))
    with BLSServer(memory_budget=need + spare, n_streams=1) as srv:
        got = srv.submit(t, y, periods=per, durations=durs, method="parity").result(timeout=300)
    st = srv.stats()
    assert st["max_held_bytes"] <= need + spare
    assert (st["max_held_bytes"] > need) == (spare > 0)
    engine = BLSEngine.get()
    batch = CurveBatch.from_arrays([t], [y], periods=per, durations=durs, flux_dtype=np.float64)
    ref = engine.search(batch, SearchConfig("parity", objective="snr"))
    for k in FIELDS:
        assert np.array_equal(got[k], ref[k].cpu().numpy()), k
