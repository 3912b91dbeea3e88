"""The kernels of a plan with look-up tables start before their predecessors have ended
(and wait for them): results in graphs, back to back and on several streams."""
import numpy as np
import pytest

import recipes as R
import test_gather_routes_gpu as G

pytestmark = pytest.mark.gpu
engine = G.engine


def plan_of(engine, geom, wkind, seed, stream, table_bytes=-1):
    from astro_transit_gpu_b200.engine import CurveBatch
    cadence = 0.0008 if geom == "binned" else 0.002
    c = [G.curve("sampled", 15003 + 64 * i, cadence, seed + i) for i in range(3)]
    c.append(G.curve("sampled", 1000, cadence, seed))  # scattered
    b = CurveBatch.from_arrays([x[0] for x in c] * 12, [x[1] for x in c] * 12,
                               periods=G.fillers(geom, G.N_PER, 15003 * cadence),
                               durations=G.DURS,
                               weights=[G.weights(wkind, len(x[0])) for x in c] * 12)
    return engine.plan(b, G.config(geom), stream=stream, table_bytes=table_bytes)


def outputs(plan):
    return {f: plan.outputs[f].cpu().numpy() for f in G.FIELDS}


@pytest.mark.parametrize("wkind", ["uniform", "point"])
@pytest.mark.parametrize("geom", ["binned", "fixed"])
def test_chained_kernels(engine, geom, wkind):
    import torch
    streams = [torch.cuda.Stream() for _ in range(3)]
    want, plans = [], []
    for i, s in enumerate(streams):
        with torch.cuda.stream(s):
            p = plan_of(engine, geom, wkind, 40 + i, s, table_bytes=0)
            p.execute()
            p.check()
            want.append(outputs(p))
            p.close()
            plans.append(plan_of(engine, geom, wkind, 40 + i, s))
            plans[-1].execute()
    torch.cuda.synchronize()
    graphs = []
    for p, s in zip(plans, streams):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            p.execute(s)
        graphs.append(g)
    for how in ("direct", "graph"):
        for p in plans:
            for f in G.FIELDS:
                p.outputs[f].zero_()
        torch.cuda.synchronize()
        for _ in range(3):  # back to back, three streams at once
            for p, s, g in zip(plans, streams, graphs):
                with torch.cuda.stream(s):
                    g.replay() if how == "graph" else p.execute(s)
        torch.cuda.synchronize()
        for p, w in zip(plans, want):
            p.check()
            assert sum(p.gathered().values()) >= 36 * 1500
            for f in G.FIELDS:
                assert np.array_equal(outputs(p)[f], w[f]), (how, f)
    del graphs
    for p in plans:
        p.close()


def test_plans_that_run_beside_others_take_tables_earlier():
    """Six curves are too few for tables when the GPU waits for them, not when it is shared."""
    import torch
    from astro_transit_gpu_b200.engine import BLSEngine, CurveBatch, SearchConfig
    rng = np.random.default_rng(7)
    n, nc = 34536, 6
    t = [1000.0 + np.arange(n) * R.CADENCE_2MIN * 1.0001 for _ in range(nc)]
    y = [(1.0 + rng.normal(0.0, 1e-3, n)).astype(np.float32) for _ in range(nc)]
    batch = CurveBatch.from_arrays(t, y, periods=np.geomspace(0.78, 7.3, 6000),
                                   durations=np.array([0.03, 0.08, 0.12, 0.16, 0.2]))
    engine, cfg = BLSEngine.get(), SearchConfig("parity", objective="snr")
    out = []
    for beside in (1, 4):
        plan = engine.plan(batch, cfg, beside=beside)
        plan.execute()
        plan.check()
        out.append((plan.gathered()["counting"], plan.outputs))
        plan.close()
    assert out[0][0] == 0 and out[1][0] == nc * 6000
    for k, v in out[0][1].items():
        assert torch.equal(v, out[1][1][k]), k
