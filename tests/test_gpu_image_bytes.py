"""Equal trees give equal images, whatever used the memory before: a tree of more points and
the same number of levels leaves its last level behind."""
import numpy as np
import pytest

from datagen import rand_points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 5, 33, 70, 300, 1025, 40000, 70001])
@pytest.mark.parametrize("dt,ids", [("f32", "arange"), ("f64", "random"), ("i32", "none")])
def test_equal_trees_equal_images(pst, tmp_path, n, dt, ids):
    pts = rand_points(n, dt, ids=ids, seed=3)
    levels = n.bit_length()
    full = rand_points((1 << levels) - 1, dt, ids=ids, seed=4, lo=500.0)

    def images():
        tree = pst.StaticPSTGPU.from_numpy(pts, dt)
        image = tree.to_bytes()
        tree.save(tmp_path / "tree.pstb")
        back = pst.StaticPSTGPU.from_bytes(image)
        got = oracle_fields(back.export())
        want = oracle_fields(tree.export())
        tree.close()
        back.close()
        return image, (tmp_path / "tree.pstb").read_bytes(), got, want

    def oracle_fields(e):
        return [e[k].tobytes() for k in ("dim1", "dim2", "med", "bitcodes")]

    pst.trim_memory()
    first, first_file, _, want = images()
    for _ in range(3):
        pst.StaticPSTGPU.from_numpy(full, dt).close()
        image, file, got, again = images()
        assert image == first and file == first_file == first
        assert got == want and again == want
