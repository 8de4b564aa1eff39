"""Whole points packed per block on their way out: every value type, with and without
ids, on trees whose levels end just below, at and above whole 64-slot blocks, one query
at a time and batched, exact against the query predicates over every point."""
import numpy as np
import pytest

from datagen import rand_points, rand_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["f32", "f64", "i32"])
@pytest.mark.parametrize("ids", ["arange", "none"])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 4095, 4097, 40009])
def test_points_of_partial_blocks(pst, oracle, dt, ids, n):
    pts = rand_points(n, dt, ids=ids, seed=n + 3)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    qs = rand_queries(pts, 40, seed=n)
    want = [oracle.canon(pts[oracle.Orc.brute(pts, dt, *q).astype(np.int64)]) for q in qs]
    for q, w in zip(qs[:6], want):
        assert np.array_equal(oracle.canon(tree.search(*q, ret="points")), w), q
    engine = pst.BatchEngine(tree, max_queries=len(qs))
    batch = pst.make_queries([pst.pst.KIND[q[0]] for q in qs], *[[q[k] for q in qs] for k in (1, 2, 3)], dt)
    offs, res = engine.search(batch, ret="points")
    for i, w in enumerate(want):
        assert np.array_equal(oracle.canon(res[offs[i]:offs[i + 1]]), w), qs[i]
    engine.close()
    tree.close()
