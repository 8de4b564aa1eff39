"""A pass captured into a caller's graph is the pass that was captured: its queries, its
buffers and its frontier stay its own, whatever the engine is called with between the
replays, and whatever the engine did before the capture."""
import ctypes as C

import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


class Case:
    """A tree, an engine and right queries from `lo` on, with what they report."""

    def __init__(self, pst, lo, max_queries, n=20000, seed=5, **opts):
        import torch
        self.pst, self.pts = pst, rand_points(n, "f32", ids="random", seed=seed)
        self.tree = pst.StaticPSTGPU.from_numpy(self.pts, "f32")
        self.engine = pst.BatchEngine(self.tree, max_queries=max_queries, **opts)
        self.lo = np.quantile(self.pts["dim1"], lo).astype(np.float32)
        self.batch = self.queries(self.lo)
        self.want = [np.sort(self.pts["id"][self.pts["dim1"] >= a]) for a in self.lo]
        self.total = sum(map(len, self.want))
        self.q = torch.from_numpy(self.batch.view(np.uint8).copy()).cuda()
        self.out, self.offs = self.buffers()
        self.stream = torch.cuda.Stream()
        torch.cuda.synchronize()

    def queries(self, lo):
        low = np.full(len(lo), self.pts["dim2"].min(), np.float32)
        return self.pst.make_queries([2] * len(lo), lo, lo, low, "f32")

    def buffers(self):
        import torch
        return (torch.zeros(max(self.total, 1), dtype=torch.int32, device="cuda"),
                torch.zeros(len(self.lo) + 1, dtype=torch.int64, device="cuda"))

    def capture(self, out=None, offs=None, mode="thread_local"):
        import torch
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=self.stream, capture_error_mode=mode):
            st, _ = self.engine.run(self.q, self.out if out is None else out, self.offs if offs is None else offs,
                                    queries_on_device=True, sync=False, stream=self.stream)
        assert st == 0
        return graph

    def replayed(self, graph, out=None, offs=None):
        import torch
        out, offs = self.out if out is None else out, self.offs if offs is None else offs
        with torch.cuda.stream(self.stream):
            out.zero_()
            offs.zero_()
            graph.replay()
        self.stream.synchronize()
        o, ids = offs.tolist(), out.cpu().numpy().view(np.uint32)
        return o[-1] == self.total and all(
            np.array_equal(np.sort(ids[o[i]:o[i + 1]]), w) for i, w in enumerate(self.want))

    def close(self, *graphs):
        self.engine.close()
        for g in graphs:
            g.reset()
        self.tree.close()


@pytest.mark.parametrize("nq", [1, 20, 100])
def test_other_calls_between_replays(pst, nq):
    import torch
    c = Case(pst, np.linspace(0.9, 1, nq), nq)
    graph = c.capture()
    other = c.queries(c.lo[: max(nq // 2, 1)] - np.float32(3))
    out2, offs2 = c.buffers()
    for call in range(4):
        if call == 1:
            c.engine.count(other, stream=c.stream)
        if call == 2:
            c.engine.run(other, out2, offs2, stream=c.stream)
        if call == 3:  # queued just before the replay, with its own queries and buffers
            q2 = torch.from_numpy(other.view(np.uint8).copy()).cuda()
            torch.cuda.synchronize()
            c.engine.run(q2, out2, offs2, queries_on_device=True, sync=False, stream=c.stream)
        with torch.cuda.stream(c.stream):
            offs2.fill_(7)
        assert c.replayed(graph), call
        assert bool((offs2 == 7).all()), call
    # and a waiting call right behind a replay that has not run yet
    with torch.cuda.stream(c.stream):
        graph.replay()
        assert c.engine.run(c.batch, c.out, c.offs, stream=c.stream) == (0, c.total)
    assert c.replayed(graph)
    c.close(graph)


@pytest.mark.parametrize("earlier", [1, 6])
def test_capture_after_asynchronous_passes(pst, earlier):
    """Asynchronous passes right before the capture, and more of them than an engine launches
    kernel by kernel; then a second capture with nothing in between."""
    c = Case(pst, np.linspace(0.5, 1, 50), 50)
    for _ in range(earlier):
        c.engine.run(c.q, c.out, c.offs, queries_on_device=True, sync=False, stream=c.stream)
    first = c.capture()
    out2, offs2 = c.buffers()
    second = c.capture(out2, offs2)
    for _ in range(2):
        assert c.replayed(first) and c.replayed(second, out2, offs2)
    assert c.engine.run(c.batch, c.out, c.offs, stream=c.stream) == (0, c.total)
    c.close(first, second)


@pytest.mark.parametrize("nq", [30, 17000])  # (more than one CTA's scan of the offsets)
@pytest.mark.parametrize("mode", ["global", "relaxed"])
def test_capture_modes(pst, mode, nq):
    """Nothing in the call is refused in any mode, also as an engine's first call."""
    c = Case(pst, np.linspace(0.999, 1, nq), nq)
    graph = c.capture(mode=mode)
    assert c.replayed(graph) and c.replayed(graph)
    c.close(graph)


class _Handle:
    """A stream of another framework: all that the binding asks for is its handle."""

    def __init__(self, stream):
        self.cuda_stream = stream.cuda_stream


def test_total_of_a_captured_pass_is_left_alone(pst):
    import torch
    c = Case(pst, np.linspace(0.9, 1, 30), 30)
    st, total = c.engine.run(c.q, c.out, c.offs, queries_on_device=True, sync=False, stream=_Handle(c.stream))
    c.stream.synchronize()
    assert (st, total) == (0, c.total)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=c.stream, capture_error_mode="thread_local"):
        assert c.engine.run(c.q, c.out, c.offs, queries_on_device=True, sync=False, stream=_Handle(c.stream)) == (0, 0)
    assert c.replayed(graph)
    c.close(graph)


def test_frontier_grown_between_replays(pst):
    """The captured pass keeps its frontier when a later one needs a larger, and no other
    object is given that memory."""
    cap = 2048
    c = Case(pst, np.linspace(0.99, 1, 4), 100, task_capacity=cap)
    graph = c.capture()
    assert c.replayed(graph)
    wide = c.queries(np.full(100, c.pts["dim1"].min(), np.float32))
    assert c.engine.count(wide, stream=c.stream)[1] == 100 * len(c.pts)  # needs far more than cap records
    others = [Case(pst, np.linspace(0.9, 1, 4), 100, n=9000, seed=s, task_capacity=cap) for s in (6, 7)]
    for _ in range(2):
        for o in others:
            assert o.engine.run(o.batch, o.out, o.offs, stream=o.stream) == (0, o.total)
        assert c.replayed(graph)
        for o in others:
            ids, offs = o.out.cpu().numpy().view(np.uint32), o.offs.tolist()
            assert all(np.array_equal(np.sort(ids[offs[i]:offs[i + 1]]), w) for i, w in enumerate(o.want))
    for o in others:
        o.close()
    c.close(graph)


def test_host_queries_are_refused(pst):
    """Before anything is captured: the capture goes on."""
    import torch
    c = Case(pst, np.linspace(0.9, 1, 40), 40)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=c.stream, capture_error_mode="thread_local"):
        st = pst.pst.lib().pst_batch_run(c.engine._h, c.batch.ctypes.data_as(C.c_void_p), 40, 0, 0,
                                         C.c_void_p(c.out.data_ptr()), c.total, C.c_void_p(c.offs.data_ptr()), None, 0,
                                         C.c_void_p(c.stream.cuda_stream))
        c.out.add_(1)
    assert st == 5  # PST_ERR_UNSUPPORTED
    graph.replay()
    torch.cuda.synchronize()
    assert bool((c.out == 1).all())
    c.close(graph)
