"""Small batches through the one-CTA top pass: queries that come as kernel parameters,
from pinned memory or from a device array, results written by the pass itself or by the
emit (around the 16384 it writes), counts only, buffers one record too small, and trees
from one point on; exact against the query predicates over every point."""
import numpy as np
import pytest

from datagen import rand_points, rand_queries

pytestmark = pytest.mark.gpu


def _batch(pst, qs, dt):
    return pst.make_queries([pst.pst.KIND[q[0]] for q in qs], *[[q[k] for q in qs] for k in (1, 2, 3)], dt)


def _want(oracle, pts, dt, q):
    return pts[oracle.Orc.brute(pts, dt, *q).astype(np.int64)]


@pytest.mark.parametrize("dt", ["f32", "f64", "i32"])
@pytest.mark.parametrize("n", [1, 2, 5, 64, 300, 20011])
@pytest.mark.parametrize("nq", [1, 2, 31, 32, 33, 70])
def test_batches(pst, oracle, dt, n, nq):
    import torch
    pts = rand_points(n, dt, ids="random", dup=n == 300, seed=n + nq)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    engine = pst.BatchEngine(tree, max_queries=nq + 3, top_pass_queries=64, task_capacity=64)
    qs = rand_queries(pts, nq, seed=nq)
    want = [_want(oracle, pts, dt, q) for q in qs]
    batch = _batch(pst, qs, dt)
    total = sum(map(len, want))
    counts, tot = engine.count(batch)
    assert tot == total and counts.tolist() == [len(w) for w in want]
    for ret, rec in (("ids", np.uint32), ("points", pts.dtype)):
        size = np.dtype(rec).itemsize
        for on_device in (False, True):
            q = torch.from_numpy(batch.view(np.uint8).copy()).cuda() if on_device else batch
            out = torch.zeros(max(total, 1) * size, dtype=torch.uint8, device="cuda")
            offs = torch.empty(nq + 1, dtype=torch.int64, device="cuda")
            assert engine.run(q, out, offs, ret=ret, queries_on_device=on_device) == (0, total)
            o, got = offs.tolist(), out.cpu().numpy().view(rec)
            assert o == np.concatenate([[0], np.cumsum([len(w) for w in want])]).tolist()
            for i, w in enumerate(want):
                w = w["id"] if ret == "ids" else w
                assert np.array_equal(oracle.canon(got[o[i]:o[i + 1]]), oracle.canon(w)), (qs[i], ret, on_device)
    if total > 1:
        out = torch.full(((total - 1) * 4,), 0xAB, dtype=torch.uint8, device="cuda")
        assert engine.run(batch, out, offs) == (4, total)
        assert (out == 0xAB).all() and offs[-1] == total
    engine.close()
    tree.close()


@pytest.mark.parametrize("hits", [16383, 16384, 16385])
@pytest.mark.parametrize("ret", ["ids", "points"])
def test_where_the_pass_stops_writing(pst, oracle, hits, ret):
    import torch
    pts = rand_points(60000, "f32", seed=8)
    pts["dim1"] = np.random.default_rng(1).permutation(60000)
    pts["dim2"] = pts["dim1"]
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    q = ("three", 100, 99 + hits, 0)
    w = _want(oracle, pts, "f32", q)
    rec = np.dtype(np.uint32) if ret == "ids" else pts.dtype
    out = torch.full((hits * rec.itemsize + 16,), 0xCD, dtype=torch.uint8, device="cuda")
    assert tree.search_into(q[0], out, hits, *q[1:], ret=ret) == hits == len(w)
    got = out[: hits * rec.itemsize].cpu().numpy().view(rec)
    assert np.array_equal(oracle.canon(got), oracle.canon(w["id"] if ret == "ids" else w))
    assert (out[hits * rec.itemsize:] == 0xCD).all()
    out.fill_(0xCD)
    assert tree.search_into(q[0], out, hits - 1, *q[1:], ret=ret) == -hits and (out == 0xCD).all()
    tree.close()


@pytest.mark.parametrize("dt", ["f32", "f64"])
@pytest.mark.parametrize("nq,top", [(1, 1), (2, 1), (17, 4), (32, 1), (32, 32), (33, 1), (150, 1), (700, 1)])
@pytest.mark.parametrize("n", [3, 700, 9001, 150001])
def test_whole_passes(pst, oracle, dt, nq, top, n):
    """Batches above the engine's limit for the top pass, and asynchronous ones within it:
    the first levels by groups of queries, the rest by level kernels; waiting and asynchronous, again and again (the
    later passes from a graph), with other queries each time."""
    import torch
    pts = rand_points(n, dt, ids="random", dup=n == 700, seed=n + nq)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    engine = pst.BatchEngine(tree, max_queries=nq, top_pass_queries=top, task_capacity=256)
    for k in range(7):
        qs = rand_queries(pts, nq, seed=nq + k)
        batch = _batch(pst, qs, dt)
        off, idx = oracle.Orc.brute_multi(pts, dt, batch["kind"], *[[q[i] for q in qs] for i in (1, 2, 3)])
        total = int(off[-1])
        out = torch.zeros(max(total, 1), dtype=torch.int32, device="cuda")
        offs = torch.empty(nq + 1, dtype=torch.int64, device="cuda")
        if k % 3 == 2:
            assert engine.count(batch)[1] == total  # grows the frontier, which an asynchronous pass cannot
            engine.run(batch, out, offs, sync=False)
            torch.cuda.synchronize()
        else:
            assert engine.run(batch, out, offs) == (0, total)
            assert engine.last_stats()["points"] == total
        assert offs.cpu().numpy().astype(np.uint64).tolist() == off.tolist()
        ids = out.cpu().numpy().view(np.uint32)
        for i in range(nq):
            a, b = int(off[i]), int(off[i + 1])
            assert np.array_equal(np.sort(ids[a:b]), np.sort(pts["id"][idx[a:b].astype(np.int64)])), qs[i]
    engine.close()
    tree.close()
