"""The kernels of a plan with look-up tables start before their predecessors have ended
(and wait for them): results in graphs, back to back and on several streams."""
import numpy as np
import pytest

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
