"""Marching cubes over cubic metacells of 2, 4 and 8 cells a side (a warp per group of
metacells, offsets by one pass with look-back): bit for bit the CPU restatement, in the
given order, from one metacell to many counting tiles (ids repeat, so each metacell's
triangles are computed on the CPU once), on volumes that cut the last metacells."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import marching_cubes as mc  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,dims", [(2, (9, 7, 5)), (2, (8, 6, 4)), (4, (17, 13, 9)), (4, (16, 11, 6)), (4, (3, 3, 3)),
                                       (8, (17, 9, 9)), (8, (14, 12, 6))])
@pytest.mark.parametrize("n", [1, 3, 31, 64, 65, 2049, 9001])
def test_cubic_equals_cpu(pst, side, dims, n):
    import torch
    rng = np.random.default_rng(n + side)
    vol = rng.random(dims[::-1]).astype(np.float32)
    vol[0, 0, :2] = (np.nan, 0.5)  # a value equal to the isovalue is inside, a NaN outside
    grid = [-(-(d - 1) // side) for d in dims]
    each = [mc.metacell_triangles(vol, (side,) * 3, np.array([i], np.uint32), 0.5)
            for i in range(grid[0] * grid[1] * grid[2])]
    ids = rng.integers(0, len(each), n).astype(np.uint32)
    want = np.concatenate([each[i] for i in ids])
    got = pst.marchingCubes(torch.from_numpy(vol.reshape(-1)).cuda(), dims, (side,) * 3,
                            torch.from_numpy(ids.view(np.int32)).cuda(), 0.5).cpu().numpy()
    assert got.shape == want.shape
    same = (got.view(np.uint32) == want.view(np.uint32)) | ((got != got) & (want != want))
    assert same.all()
