"""Query and offsets arrays that kernels cannot use where they are (not at a multiple of 8
bytes) give the results of aligned ones, on every path a batch can take."""
import ctypes as C

import numpy as np
import pytest

from datagen import rand_points, rand_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [4, 1])
@pytest.mark.parametrize("nq", [1, 20, 100])
def test_unaligned_arrays(pst, nq, shift):
    import torch
    lib = pst.pst.lib()
    pts = rand_points(30011, "f32", ids="random", seed=nq)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    k, a, b, m = zip(*rand_queries(pts, nq, seed=3))
    batch = pst.make_queries([pst.pst.KIND[x] for x in k], a, b, m, "f32")
    engine = pst.BatchEngine(tree, nq)
    offsets, ids = engine.search(batch)
    want = [np.sort(ids[offsets[i]:offsets[i + 1]]) for i in range(nq)]
    raw = batch.view(np.uint8).reshape(-1)
    for q_shift, o_shift in ((shift, 0), (0, shift), (shift, shift)):
        q = torch.zeros(raw.nbytes + 8, dtype=torch.uint8, device="cuda")
        q[q_shift:q_shift + raw.nbytes] = torch.from_numpy(raw.copy()).cuda()
        for sync in (1, 0):
            out = torch.zeros(max(len(ids), 1), dtype=torch.int32, device="cuda")
            offs = torch.full((8 * (nq + 1) + 16,), 255, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            st = lib.pst_batch_run(engine._h, C.c_void_p(q.data_ptr() + q_shift), nq, 1, 0,
                                   C.c_void_p(out.data_ptr()), len(ids), C.c_void_p(offs.data_ptr() + o_shift), None,
                                   sync, C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert st == 0
            torch.cuda.synchronize()
            o = offs.cpu().numpy()
            end = o_shift + 8 * (nq + 1)
            assert np.array_equal(o[o_shift:end].copy().view(np.uint64), offsets)
            assert (o[:o_shift] == 255).all() and (o[end:] == 255).all()
            got = out.cpu().numpy().view(np.uint32)
            assert all(np.array_equal(np.sort(got[offsets[i]:offsets[i + 1]]), want[i]) for i in range(nq))
        total = C.c_uint64()
        assert lib.pst_batch_count(engine._h, C.c_void_p(q.data_ptr() + q_shift), nq, 1, None, C.byref(total),
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert total.value == len(ids)
    engine.close()
    tree.close()
