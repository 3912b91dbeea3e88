"""The result line of bench.py survives what only adds to it (CPU)."""
import numpy as np

import bench


def test_missing_plain_kernels_do_not_lose_the_line(monkeypatch):
    def missing(*args):
        raise FileNotFoundError("bls_f32_t1.cubin missing")

    monkeypatch.setattr(bench, "plain_gpu_baseline", missing)
    line = {"value": 2.0, "vs_baseline": None}
    line.update(bench.plain_gpu_report(2.0, {}, 1.0, None))
    assert line["value"] == 2.0 and line["vs_baseline"] is None
    assert "bls_f32_t1.cubin" in line["plain_gpu_baseline"]["unavailable"]


def test_plain_kernels_give_the_ratio(monkeypatch):
    monkeypatch.setattr(bench, "plain_gpu_baseline", lambda *a: {"value": 4.0})
    got = bench.plain_gpu_report(2.0, {}, 1.0, None)
    assert got["vs_baseline"] == 0.5 and got["plain_gpu_baseline"] == {"value": 4.0}


def test_gathered_periods_are_not_measured_in_reductions():
    """A scattered launch is measured in shared-memory reductions, one of
    gathered periods is not: it issues none."""
    r = bench.search_roofline("uniform", "parity", 1024, 0.0, None, 2.0, 30.0, 60.0, 1.0)
    assert r["frac"] == 0.5 and r["bound"] == "smem" and r["traffic"] > 0
    r = bench.search_roofline("uniform", "parity", 1024, 1.0, 3.0e9, 2.0, 30.0, 60.0, 1.0)
    assert r["frac"] is None and r["kernel"] == "gather_kernel<BINNED>"
    assert abs(r["achieved"] - 1500.0) < 1e-9
    r = bench.search_roofline("mixed", "fast", 512, 0.25, None, 2.0, 30.0, 60.0, 1.0)
    assert r["achieved"] is None and "search_kernel" in r["kernel"]


def test_table_lookups():
    # 10 d of data, 0.004 d bins: 2.5 d has 5 cycles of 626 boundaries, 12 d one of 3001
    t = np.linspace(0.0, 10.0, 1000)
    got = bench.table_lookups(t, np.array([2.5, 12.0]), np.array([0.04, 0.08]))
    assert got == 5 * 5 * 128 + 24 * 128


def test_durations_shared_or_per_curve():
    assert bench.curve_durations([0.04, 0.08], 5) == [0.04, 0.08]
    assert bench.curve_durations([np.array([0.04]), np.array([0.08])], 1)[0] == 0.08
