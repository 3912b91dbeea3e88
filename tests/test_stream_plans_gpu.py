"""Calls that make a plan for themselves make it in their stream's order: a plan of
device-wide allocations maps and unmaps its scratch on every call."""
import numpy as np
import pytest

import recipes as R

pytestmark = pytest.mark.gpu


def _curves(n_curves=6, n=6000):
    rng = np.random.default_rng(31)
    t = [np.arange(n) * R.CADENCE_2MIN + 1500.0 + c for c in range(n_curves)]
    return t, [(1.0 + rng.normal(0.0, 1e-3, n)).astype(np.float32) for _ in t]


@pytest.fixture()
def streams_of_plans(monkeypatch):
    from astro_transit_gpu_b200.engine import BLSEngine
    seen, plan = [], BLSEngine.plan

    def record(self, *args, **kw):
        p = plan(self, *args, **kw)
        seen.append(p.stream)
        return p

    monkeypatch.setattr(BLSEngine, "plan", record)
    return seen


def test_power_batch(streams_of_plans):
    import torch
    from astro_transit_gpu_b200 import power_batch
    t, y = _curves()
    per, dur = np.linspace(0.6, 4.0, 400), np.array([0.05, 0.1])
    want = power_batch(t, y, periods=per, durations=dur)
    with torch.cuda.stream(torch.cuda.Stream()):
        got = power_batch(t, y, periods=per, durations=dur)
    assert len(streams_of_plans) == 2 and None not in streams_of_plans
    for a, b in zip(want, got):
        assert np.array_equal(a.power, b.power) and np.array_equal(a.window, b.window)
        assert a.top_candidates == b.top_candidates


def test_screen(streams_of_plans):
    import torch
    from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, SearchConfig
    t, y = _curves()
    batch = CurveBatch.from_arrays(t, y, periods=np.linspace(0.6, 4.0, 400),
                                   durations=np.array([0.05, 0.1]))
    engine, cfg = BLSEngine.get(), SearchConfig("fast", n_bins=200)
    full = engine.search(batch, cfg)["power"].cpu().numpy().reshape(len(t), -1)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    got = engine.screen(batch, cfg, stream=s)
    assert None not in streams_of_plans
    assert np.array_equal(got["best_index"].cpu().numpy(), full.argmax(1))
    assert np.array_equal(got["power"].cpu().numpy(), full.max(1))


def test_screen_waits_for_the_callers_stream():
    """The batch may still be on its way when screen is called with another stream."""
    import torch
    from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, SearchConfig
    t, y = _curves()
    batch = CurveBatch.from_arrays(t, y, periods=np.linspace(0.6, 4.0, 400),
                                   durations=np.array([0.05, 0.1]))
    engine, cfg = BLSEngine.get(), SearchConfig("fast", n_bins=200)
    want = engine.screen(batch, cfg)
    flux = batch.y.clone()
    batch.y.copy_(torch.flip(flux, (0,)))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # about 50 ms of the caller's stream
    batch.y.copy_(flux)
    got = engine.screen(batch, cfg, stream=s)
    for k, v in want.items():
        assert torch.equal(got[k], v), k
