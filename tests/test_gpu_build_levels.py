"""Wide-level construction at the edges of its tiles (512 positions), groups of tiles
(16384) and of a warp or a CTA per node, on data whose maxima lie anywhere, all at one
end, or tie: whole trees bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [512, 513, 514, 1023, 1024, 1025, 1537, 16383, 16385, 32769, 49153, 524289, 1250003]


def _points(oracle, n, dt, shape):
    rng = np.random.default_rng(n)
    t = {"f32": np.float32, "f64": np.float64, "i32": np.int32}[dt]
    d1 = rng.permutation(n) if shape != "ties" else rng.integers(0, 50, n)
    d2 = {"random": rng.integers(0, 1 << 20, n), "rising": d1, "falling": n - d1, "ties": rng.integers(0, 3, n)}[shape]
    ids = np.arange(n) if n % 2 else rng.permutation(n)
    return oracle.make_points(d1.astype(t), d2.astype(t), ids.astype(np.uint32), dt)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dt,shape", [("f32", "random"), ("f64", "random"), ("i32", "rising"), ("f32", "falling"),
                                      ("i32", "ties"), ("f64", "ties")])
def test_tree_at_tile_edges(pst, oracle, n, dt, shape):
    pts = _points(oracle, n, dt, shape)
    ref = oracle.Orc.build(pts, dt)
    tree = pst.StaticPSTGPU.from_numpy(pts, dt)
    got = tree.export()
    for f in ("dim1", "dim2", "med", "bitcodes", "ids"):
        assert got[f].tobytes() == getattr(ref, f).tobytes(), f
    tree.close()
