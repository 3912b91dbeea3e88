"""The result line of bench.py survives what only adds to it (CPU)."""
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
