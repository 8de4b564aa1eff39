"""A server's slots have the graph of their whole pass before the first request."""
import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_first_large_batch_replays_a_graph(pst, dt):
    import torch
    pts = rand_points(50000, dt, seed=2)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    server = pst.Server(max_batch=256, slots_per_tree=1, out_budget_bytes=64 << 20)
    index = server.add_tree(tree)
    lo = np.linspace(900, 1000, 200).astype(pts["dim1"].dtype)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU,
                                            torch.profiler.ProfilerActivity.CUDA]) as prof:
        ids = server.submit(index, pst.make_queries([2] * 200, lo, lo, np.zeros(200), dt))
        server.drain(60000)
    calls = {e.key: e.count for e in prof.key_averages()}
    assert calls.get("cudaGraphLaunch", 0) == 1, sorted(calls)
    assert not any("GraphInstantiate" in k or "BeginCapture" in k for k in calls), sorted(calls)
    for rid, a in zip(ids[::50], lo[::50]):
        assert np.array_equal(np.sort(server.take(int(rid), np.uint32)), np.sort(pts["id"][pts["dim1"] >= a]))
    server.close()
    tree.close()
