"""Metacells on both sides of the rule that chooses between a thread per metacell and a
thread per vertex column, against max pooling: flat ones (few vertices to a column) on
volumes that fill the device and on small ones."""
import pytest

pytestmark = pytest.mark.gpu


def _pooled(vol, mc):
    import torch
    v = vol.double()[None, None]
    kernel, stride = tuple(m + 1 for m in mc[::-1]), tuple(mc[::-1])
    pool = torch.nn.functional.max_pool3d
    return -pool(-v, kernel, stride).reshape(-1), pool(v, kernel, stride).reshape(-1)


def _fields(pst, out, dt):
    import torch
    size = 8 if dt == "f64" else 4
    rec = out.view(-1, pst.point_dtype(dt, True).itemsize)
    typ = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32}[dt]
    return [rec[:, k * size:(k + 1) * size].contiguous().view(typ).view(-1) for k in (0, 1)]


@pytest.mark.parametrize("mc", [(2, 1, 1), (5, 5, 1), (5, 6, 1), (8, 1, 2), (9, 1, 2), (2, 2, 2), (5, 2, 3), (5, 7, 1), (6, 3, 2),
                                (3, 1, 3), (4, 1, 1), (4, 1, 2)])
@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("dt", ["f32", "f64", "i32"])
def test_flat_and_deep(pst, dt, big, mc):
    import torch
    torch.manual_seed(sum(mc))
    want_dims = (515, 240, 130) if big else (70, 33, 19)
    dims = tuple(-(-(d - 1) // m) * m + 1 for d, m in zip(want_dims, mc))
    typ = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32}[dt]
    vol = (torch.randn(dims[::-1], device="cuda") * 1000).to(typ)
    out, n = pst.formMetacellTags(vol, dims, mc, dt, True)
    lo, hi = _fields(pst, out, dt)
    a, b = _pooled(vol, mc)
    assert n == len(a) and torch.equal(lo.double(), a) and torch.equal(hi.double(), b)
