"""The CRT scan's scale factors (GPU): one power of two while 2^-e is a normal double, two outside,
and rows of subnormal entries only.  Scaling a row of op(A) by a power of two and op(B) back
changes no bit of the product as long as the entries keep their digits."""
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def crt_method():
    eb.set_dgemm_method(eb.METHOD_CRT)
    yield
    eb.set_dgemm_method(eb.METHOD_AUTO)


def _scale(x, e):
    # in steps whose factors are normal doubles
    while e:
        s = max(-1000, min(1000, e))
        x = x * 2.0 ** s
        e -= s
    return x


@pytest.mark.parametrize("e", [-1066, -1030, -1023, -1022, -1021, -1, 0, 1, 1020, 1021, 1022, 1023])
@pytest.mark.parametrize("rows,k", [(1, 1), (33, 127), (40, 300)])
def test_scaled_rows(e, rows, k):
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    if e > -1021:
        a = torch.rand((k, rows), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        # entries whose last bit stays above the subnormals after the scaling
        a = torch.where(a.abs() < 0.125, torch.full_like(a, 0.75), a) if e < 0 else a
        a = a * 0.5 if e == 1023 else a
    else:  # |a| an integer below 2^7, over 2^8: exact down to 2^-1074
        a = torch.randint(-127, 128, (k, rows), device="cuda", generator=g).double() / 256
    b = torch.rand((8, k), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    b = torch.where(b.abs() < 0.125, torch.full_like(b, 0.5), b)
    shift = 500 if e < 0 else -500
    out = []
    for ea, eb_ in ((0, 0), (e, shift)):
        c = torch.empty((8, rows), dtype=torch.float64, device="cuda")
        x, y = _scale(a, ea), _scale(b, eb_)
        assert eb.dgemm_device("N", "N", rows, 8, k, 1.0, x, rows, y, k, 0.0, c, rows) == eb.EB2_OK
        out.append(c)
    assert torch.isfinite(out[1]).all()
    assert torch.equal(out[1], _scale(out[0], e + shift))
