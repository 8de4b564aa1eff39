"""Metacells of any sides over odd volumes, with the values whose order in a fold shows
(-0.0, NaN) among them: bit for bit what a fold vertex after vertex, plane by plane,
gives, keeping the first of equal values and never replacing by a NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NP = {"f32": np.float32, "f64": np.float64, "i32": np.int32}


def _fold(values):
    lo = hi = values[0]
    for v in values[1:]:
        lo = v if v < lo else lo
        hi = v if v > hi else hi
    return lo, hi


def _metacells(vol, mc, by_rows):
    grid = [-(-(s - 1) // m) for s, m in zip(vol.shape, mc)]
    out = []
    for at in np.ndindex(*grid):
        z, y, x = [range(i * m, min(i * m + m, s - 1) + 1) for i, m, s in zip(at, mc, vol.shape)]
        planes = []
        for k in z:
            rows = [vol[k, j, x.start:x.stop] for j in y]
            if by_rows:
                rows = [_fold(r) for r in rows]
                planes.append((_fold([r[0] for r in rows])[0], _fold([r[1] for r in rows])[1]))
            else:
                planes.append(_fold(np.concatenate(rows)))
        out.append((_fold([p[0] for p in planes])[0], _fold([p[1] for p in planes])[1]))
    return np.array(out, vol.dtype)


@pytest.mark.parametrize("dims,mc", [((13, 11, 9), (1, 1, 1)), ((13, 11, 9), (2, 2, 2)), ((27, 13, 10), (4, 4, 4)),
                                     ((28, 13, 10), (4, 4, 4)), ((35, 18, 17), (8, 8, 8)), ((17, 10, 11), (3, 5, 2)),
                                     ((12, 10, 11), (4, 3, 5)), ((515, 3, 5), (2, 4, 8)), ((1030, 3, 3), (600, 1, 2)),
                                     ((520, 4, 3), (511, 2, 1)), ((2, 2, 2), (8, 8, 8)), ((514, 2, 34), (4, 1, 1))])
@pytest.mark.parametrize("dt", ["f32", "f64", "i32"])
@pytest.mark.parametrize("special", [False, True])
def test_any_sides(pst, dims, mc, dt, special):
    import torch
    rng = np.random.default_rng(sum(dims) + sum(mc))
    shape = dims[::-1]
    if dt == "i32":
        vol = rng.integers(-9, 9, shape).astype(np.int32)
    else:
        vol = rng.standard_normal(shape).astype(NP[dt])
        if special:
            some = np.array([-0.0, 0.0, 0.0, 1.0, np.nan, np.inf, -np.inf, -1.0], NP[dt])
            vol = np.where(rng.random(shape) < 0.5, rng.choice(some, shape), vol)
            vol[:, :, : dims[0] // 2] = rng.choice(np.array([0.0, -0.0, 2.0], NP[dt]), (*shape[:2], dims[0] // 2))
    want = _metacells(vol, mc[::-1], by_rows=dt != "f64" and mc[0] == 4 and dims[0] % 4 == 0)
    out, n = pst.formMetacellTags(torch.from_numpy(vol.reshape(-1).copy()).cuda(), dims, mc, dt, True)
    rec = out.cpu().numpy().view(pst.point_dtype(dt, True))
    assert n == len(want) and np.array_equal(rec["id"], np.arange(n))
    bits = f"u{want.itemsize}"
    for k, f in enumerate(("dim1", "dim2")):
        got, w = rec[f], np.ascontiguousarray(want[:, k])
        same = (got.view(bits) == w.view(bits)) | ((got != got) & (w != w))  # (a NaN's payload is its vertex's)
        assert same.all(), (f, np.nonzero(~same)[0][:5])
