"""pst_trim_memory gives back what the library keeps, and leaves what is in use alone."""
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


def test_trim(pst, oracle):
    import torch
    pts = rand_points(50000, "f32", ids="random", seed=9)
    tree = pst.StaticPSTGPU.from_numpy(pts, "f32")
    q = ("three", 300, 320, 310)
    want = oracle.canon(tree.search(*q))
    n = 20_000_000
    big = torch.zeros((n, 3), dtype=torch.int32, device="cuda")
    big[:, 2] = torch.arange(n, device="cuda", dtype=torch.int32)
    pst.trim_memory()
    free = torch.cuda.mem_get_info()[0]
    other = pst.StaticPSTGPU(big, n)
    assert len(other.search("left", 0, 0, 0)) == n  # (a result of 80 MB, freed by now)
    other.close()
    kept = free - torch.cuda.mem_get_info()[0]
    assert kept > 500 << 20
    torch.cuda.empty_cache()
    pst.trim_memory()
    assert free - torch.cuda.mem_get_info()[0] < 32 << 20
    assert (oracle.canon(tree.search(*q)) == want).all()
    tree.close()
