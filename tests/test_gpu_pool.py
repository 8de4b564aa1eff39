"""The pool behind trees and engines: blocks reused between objects, threads and streams
never hold two objects' data at once, an asynchronous pass outlives the objects it was
queued on, and what is kept stays bounded."""
import threading

import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


def _check(pst, oracle, pts, dt, stream):
    import torch
    with torch.cuda.stream(stream):
        tree = pst.StaticPSTGPU.from_numpy(pts, dt)
        stream.synchronize()
        q = ("three", float(pts["dim1"][0]) - 40, float(pts["dim1"][0]) + 40, float(pts["dim2"].mean()) - 200)
        got = oracle.canon(tree.search(*q))
        tree.close()
    return np.array_equal(got, oracle.canon(pts["id"][oracle.Orc.brute(pts, dt, *q).astype(np.int64)]))


def test_threads_and_streams(pst, oracle):
    import torch
    sets = [(rand_points(n, dt, seed=n), dt) for n in (900, 5000, 70001) for dt in ("f32", "f64")]
    bad = []

    def work(pts, dt):
        stream = torch.cuda.Stream()
        for _ in range(4):
            if not _check(pst, oracle, pts, dt, stream):
                bad.append((len(pts), dt))

    threads = [threading.Thread(target=work, args=s) for s in sets]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("tree_first", [True, False])
def test_destroyed_under_an_asynchronous_pass(pst, oracle, tree_first):
    """The pass keeps its tree and workspace until it has run, whichever goes first, and
    whatever is built at once in the memory they leave."""
    import torch
    pts = rand_points(2_000_000, "f32", seed=5)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    qs = [("left", 0, 100 + 50 * i, 60) for i in range(16)]
    batch = pst.make_queries([1] * 16, [0] * 16, [q[2] for q in qs], [60] * 16, "f32")
    engine = pst.BatchEngine(tree, 16)
    total = engine.count(batch)[1]
    out = torch.empty(total, dtype=torch.int32, device="cuda")
    offs = torch.empty(17, dtype=torch.int64, device="cuda")
    dev = torch.from_numpy(batch.view(np.uint8).copy()).cuda()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    engine.run(dev, out, offs, queries_on_device=True, sync=False, stream=stream)
    for x in (tree, engine) if tree_first else (engine, tree):
        x.close()
    other = [pst.StaticPSTGPU.from_numpy(rand_points(1_900_000, "f32", seed=s), "f32") for s in (6, 7)]
    torch.cuda.synchronize()
    ids, o = out.cpu().numpy().view(np.uint32), offs.tolist()
    for i, q in enumerate(qs):
        want = pts["id"][oracle.Orc.brute(pts, "f32", *q).astype(np.int64)]
        assert np.array_equal(np.sort(ids[o[i]:o[i + 1]]), np.sort(want)), q
    for t in other:
        t.close()


def test_kept_memory_is_bounded(pst):
    """Trees of growing sizes, one after another: what stays is at most a 1/32 of the device."""
    import torch
    free0, total = torch.cuda.mem_get_info()
    for n in (1 << 20, 3 << 20, 9 << 20, 27 << 20, 60 << 20):
        pts = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
        pts[:, 2] = torch.arange(n, device="cuda", dtype=torch.int32)
        pst.StaticPSTGPU(pts, n).close()
        del pts
        torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info()[0] <= total // 32 + (512 << 20)
