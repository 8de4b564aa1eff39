"""A waiting call that has results and room for them, but no buffer, says so."""
import ctypes as C

import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq", [1, 40])
def test_no_buffer(pst, nq):
    import torch
    lib = pst.pst.lib()
    pts = rand_points(5000, "f32", seed=1)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    engine = pst.BatchEngine(tree, nq)
    lo = np.full(nq, 990, np.float32)
    batch = pst.make_queries([2] * nq, lo, lo, lo, "f32")
    total = engine.count(batch)[1]
    assert total > 0
    stream, got = C.c_void_p(torch.cuda.current_stream().cuda_stream), C.c_uint64()

    def run(capacity):
        return lib.pst_batch_run(engine._h, batch.ctypes.data_as(C.c_void_p), nq, 0, 0, None, capacity, None,
                                 C.byref(got), 1, stream)

    assert run(total) == 1 and run(total - 1) == 4 and got.value == total
    q = batch[:1].copy()
    count = tree.count("right", 990, 0, 990)
    assert lib.pst_search_into(tree.handle, q.ctypes.data_as(C.POINTER(pst.pst.Query)), 0, None, count, C.byref(got), stream) == 1
    assert lib.pst_search_into(tree.handle, q.ctypes.data_as(C.POINTER(pst.pst.Query)), 0, None, 0, C.byref(got), stream) == 4
    engine.close()
    tree.close()
