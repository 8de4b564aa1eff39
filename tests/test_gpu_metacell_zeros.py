"""Metacells of fields clipped at zero, whose zeros have one sign: max pooling gives the
same, and a zero of a result has the sign of the field's."""
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


@pytest.mark.parametrize("minus", [False, True])
@pytest.mark.parametrize("above", [False, True])
@pytest.mark.parametrize("mc", [(2, 2, 2), (4, 4, 4), (3, 5, 2)])
@pytest.mark.parametrize("dt", ["f32", "f64"])
def test_zeros_of_one_sign(pst, dt, mc, above, minus):
    """A field clipped at zero from above or below: every zero of a result has the field's."""
    import torch
    torch.manual_seed(7)
    dims = (61, 41, 31)
    typ = {"f32": torch.float32, "f64": torch.float64}[dt]
    vol = torch.randn(dims[::-1], device="cuda").to(typ)
    zero = torch.full_like(vol, -0.0 if minus else 0.0)
    vol = torch.where(vol > 0 if above else vol < 0, zero, vol)
    out, _ = pst.formMetacellTags(vol, dims, mc, dt, True)
    lo, hi = _fields(pst, out, dt)
    if all((d - 1) % m == 0 for d, m in zip(dims, mc)):
        a, b = _pooled(vol, mc)
        assert torch.equal(lo.double(), a) and torch.equal(hi.double(), b)
    for v in (lo, hi):
        zeros = v[v == 0]
        assert bool((torch.signbit(zeros) == minus).all())
    assert bool(((hi if above else lo) == 0).any())
