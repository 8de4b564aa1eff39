"""The construction's radix sort over a few tiles (4096 keys) and steps of its look-back
(four tiles), every digit in use or all keys on few of them: whole trees bit for bit
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [4096 * t + r for t in (2, 3, 4, 5, 9, 21) for r in (-1, 1)] + [4096 * 8, 4096 * 700 + 33]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt,spread", [("f32", "wide"), ("f64", "wide"), ("i32", "wide"), ("f64", "few"), ("i32", "few")])
def test_tree_over_sort_tiles(pst, oracle, n, dt, spread):
    rng = np.random.default_rng(n)
    t = {"f32": np.float32, "f64": np.float64, "i32": np.int32}[dt]
    if spread == "few":
        # two digits in use, of very unequal counts
        d1 = np.where(rng.random(n) < 0.999, 7, 7 + (rng.integers(0, 3, n) << 20))
        d2 = rng.integers(0, 2, n) << 12
    else:
        d1 = rng.integers(-(1 << 31), 1 << 31, n)
        d2 = rng.integers(-(1 << 31), 1 << 31, n)
    ids = rng.permutation(n)  # decreasing somewhere: the ids are sorted too, from the identity
    pts = oracle.make_points(d1.astype(t), d2.astype(t), ids.astype(np.uint32), dt)
    ref = oracle.Orc.build(pts, dt)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    got = tree.export()
    for f in ("dim1", "dim2", "med", "bitcodes", "ids"):
        assert got[f].tobytes() == getattr(ref, f).tobytes(), f
    tree.close()
