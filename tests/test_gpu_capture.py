"""An asynchronous pass in a graph of the caller's: captured after passes outside it,
replayed, with its engine destroyed afterwards."""
import ctypes as C

import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,earlier", [(1, 0), (20, 2), (100, 2)])
def test_captured_pass(pst, oracle, nq, earlier):
    import torch
    lib = pst.pst.lib()
    pts = rand_points(20000, "f32", ids="random", seed=5)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    engine = pst.BatchEngine(tree, max_queries=nq)
    lo = np.linspace(pts["dim1"].min(), pts["dim1"].max(), nq + 1)[:-1].astype(np.float32)
    kinds = np.full(nq, 2)  # right queries
    batch = pst.make_queries(kinds, lo, lo, np.full(nq, np.median(pts["dim2"]), np.float32), "f32")
    want = [np.sort(pts["id"][(pts["dim1"] >= a) & (pts["dim2"] >= np.float32(np.median(pts["dim2"])))]) for a in lo]
    total = sum(map(len, want))
    q = torch.from_numpy(batch.view(np.uint8).copy()).cuda()
    out = torch.zeros(max(total, 1), dtype=torch.int32, device="cuda")
    offs = torch.zeros(nq + 1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for _ in range(earlier):
            engine.run(q, out, offs, queries_on_device=True, sync=False)
        assert engine.run(q, out, offs, queries_on_device=True) == (0, total)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            # (without a total: its copy would land in this call's host memory at every replay)
            assert lib.pst_batch_run(engine._h, C.c_void_p(q.data_ptr()), nq, 1, 0, C.c_void_p(out.data_ptr()), total,
                                     C.c_void_p(offs.data_ptr()), None, 0, C.c_void_p(stream.cuda_stream)) == 0
        for _ in range(2):
            out.zero_()
            offs.zero_()
            graph.replay()
            stream.synchronize()
            o, ids = offs.tolist(), out.cpu().numpy().view(np.uint32)
            assert o[-1] == total
            for i, w in enumerate(want):
                assert np.array_equal(np.sort(ids[o[i]:o[i + 1]]), w)
    engine.close()
    graph.reset()
    tree.close()
