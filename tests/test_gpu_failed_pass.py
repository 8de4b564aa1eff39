"""A waiting pass that fails leaves the caller's results and offsets as they were."""
import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ret", ["ids", "points"])
@pytest.mark.parametrize("nq", [2, 20, 33, 100, 17000])
def test_bad_kind(pst, nq, ret):
    import torch
    pts = rand_points(20000, "f32", seed=4)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    engine = pst.BatchEngine(tree, nq)
    lo = np.linspace(990, 1000, nq).astype(np.float32)
    batch = pst.make_queries([2] * nq, lo, lo, np.zeros(nq, np.float32), "f32")
    total = engine.count(batch)[1]
    assert total > 0
    out = torch.full((3 * total,), 77, dtype=torch.int32, device="cuda")
    offs = torch.full((nq + 1,), 77, dtype=torch.int64, device="cuda")
    bad = batch.copy()
    bad["kind"][nq // 2] = 9
    for on_device in (False, True):
        q = torch.from_numpy(bad.view(np.uint8).copy()).cuda() if on_device else bad
        with pytest.raises(pst.pst.PSTError) as e:
            engine.run(q, out, offs, ret=ret, queries_on_device=on_device)
        assert "kind" in str(e.value)
        torch.cuda.synchronize()
        assert bool((out == 77).all()) and bool((offs == 77).all())
    assert engine.run(batch, out, offs, ret=ret) == (0, total)
    assert offs[-1].item() == total
    engine.close()
    tree.close()
