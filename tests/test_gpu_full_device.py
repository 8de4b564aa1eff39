"""On a device that others fill, the memory that the library keeps for reuse is there for its
own allocations: results, a server's arena, the slabs of a volume read from a file."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n):
    import torch
    pts = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    pts[:, 0] = torch.arange(n, device="cuda", dtype=torch.int32)
    pts[:, 1] = pts[:, 0] + 5
    pts[:, 2] = pts[:, 0]
    return pts


def test_kept_memory_serves_the_library(pst, tmp_path):
    import torch
    n = 30_000_000
    tree = pst.StaticPSTGPU(_points(n), n, "i32")
    assert tree.count("right", 0, 0, 0) == n  # (the tree's own engine is made)
    big = 60_000_000
    pst.StaticPSTGPU(_points(big), big, "i32").close()  # leaves about a GB in the pool
    dims = (512, 256, 256)
    path = tmp_path / "volume.raw"
    volume = np.random.default_rng(3).standard_normal(dims[::-1]).astype(np.float32)
    volume.tofile(path)
    want, _ = pst.formMetacellTags(torch.from_numpy(volume).cuda(), dims, (4, 4, 4))
    want = want.cpu()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()

    def filled():
        """All free device memory but 64 MB."""
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")

    def refill():
        pst.StaticPSTGPU(_points(big), big, "i32").close()

    fill = filled()
    ptr, count = tree.search_device("right", 0, 0, 0)  # 120 MB
    assert count == n
    pst.free_device(ptr)
    del fill
    refill()
    fill = filled()
    server = pst.Server(out_budget_bytes=200 << 20, keep_results=0)
    server.close()
    del fill
    refill()
    out = torch.empty(want.numel(), dtype=torch.uint8, device="cuda")
    fill = filled()
    lib, P, M = pst.pst.lib(), (pst.pst.C.c_uint32 * 3)(*dims), (pst.pst.C.c_uint32 * 3)(4, 4, 4)
    st = lib.pst_form_metacells_from_file(str(path).encode(), 0, 1, P, M, pst.pst.C.c_void_p(out.data_ptr()), 128 << 20,
                                          pst.pst._stream())
    assert st == 0, lib.pst_last_error()
    torch.cuda.synchronize()
    assert torch.equal(out.cpu(), want)
    del fill
    tree.close()
