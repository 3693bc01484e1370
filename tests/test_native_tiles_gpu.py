"""The native FP64 kernel's output tiles (GPU): sizes at the edges of the 32, 64 and 128 tiles and
on both sides of the tile choice, every transpose, odd and even leading dimensions.  The sum of an
output has one order whatever tile it lies in, so a product equals the same block of a larger
product bit for bit; against FP64 sums of the absolute values it stays within k u."""
import time

import numpy as np
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.fixture(autouse=True)
def native_method():
    eb.set_dgemm_method(eb.METHOD_NATIVE)
    yield
    eb.set_dgemm_method(eb.METHOD_AUTO)


def product(ta, tb, m, n, k, a, lda, b, ldb, ldc, alpha=1.0, beta=0.0, c=None):
    c = torch.full((n, ldc), float("nan"), dtype=torch.float64, device="cuda") if c is None else c.clone()
    assert eb.dgemm_device(ta, tb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc) == eb.EB2_OK
    return c


# (rows, columns): one tile, edges of 32 / 64 / 128, and shapes the choice gives to each tile side
SIZES = [(1, 1), (31, 33), (64, 65), (127, 129), (200, 190), (512, 500), (768, 760), (1000, 1531), (1540, 1500)]


@pytest.mark.parametrize("m,n", SIZES)
@pytest.mark.parametrize("ta,tb,pad", [("N", "N", 0), ("T", "N", 1), ("N", "T", 8), ("T", "T", 3)])
def test_tiles_agree_with_a_larger_product(m, n, ta, tb, pad):
    k = 37
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    big_m, big_n = 2100, 1700  # 128 x 128 tiles
    rows_a, cols_a = (big_m, k) if ta == "N" else (k, big_m)
    rows_b, cols_b = (k, big_n) if tb == "N" else (big_n, k)
    lda, ldb = rows_a + pad, rows_b + pad
    a = torch.rand((cols_a, lda), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    b = torch.rand((cols_b, ldb), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    whole = product(ta, tb, big_m, big_n, k, a, lda, b, ldb, big_m)
    part = product(ta, tb, m, n, k, a, lda, b, ldb, m + pad)
    assert torch.equal(part[:, :m], whole[:n, :m])
    if pad:
        assert torch.isnan(part[:, m:]).all()  # the padding rows are not touched
    # |computed - exact| <= k u sum |a||b|, and the reference's own sum is as far off
    opa = (a[:, :m].T if ta == "N" else a[:m, :k]).cpu().numpy()
    opb = (b[:n, :k].T if tb == "N" else b[:, :n]).cpu().numpy()
    ref = opa @ opb
    bound = 2 * k * U * (np.abs(opa) @ np.abs(opb))
    assert (np.abs(part[:, :m].T.cpu().numpy() - ref) <= bound).all()


@pytest.mark.parametrize("m,n", [(33, 70), (300, 130), (770, 765)])
def test_tiles_update_c(m, n):
    k = 21
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.rand((k, m), dtype=torch.float64, device="cuda", generator=g)
    b = torch.rand((n, k), dtype=torch.float64, device="cuda", generator=g)
    c = torch.rand((n, m + 1), dtype=torch.float64, device="cuda", generator=g)
    plain = product("N", "N", m, n, k, a, m, b, k, m)
    got = product("N", "N", m, n, k, a, m, b, k, m + 1, alpha=1.5, beta=0.5, c=c)
    # 1.5 p is rounded once and 0.5 c + that once more
    want = 0.5 * c[:, :m] + 1.5 * plain
    assert torch.equal(got[:, :m], want) and torch.equal(got[:, m], c[:, m])


def test_fallback_of_a_checked_call_takes_the_tile_that_fits():
    # a call that reads the flags on the host launches the fallback knowing that it will run: 16 tiles of
    # 32 x 32; behind the flag it is one of 128 x 128, on one SM
    m = n = 128
    k = 8192
    a = torch.rand((k, m), dtype=torch.float64, device="cuda")
    b = torch.rand((n, k), dtype=torch.float64, device="cuda")
    a[7, 3] = float("nan")
    c = {flag: torch.zeros((n, m), dtype=torch.float64, device="cuda") for flag in (True, False)}

    def call(check):
        assert eb.dgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c[check], m, check_accuracy=check) == eb.EB2_OK
        torch.cuda.synchronize()

    def best(check):
        times = []
        for _ in range(8):
            t0 = time.perf_counter()
            call(check)
            times.append(time.perf_counter() - t0)
        return min(times)

    eb.set_dgemm_method(eb.METHOD_CRT)
    try:
        call(True)
        assert eb.last_call_info()["nonfinite"] == 1
        checked, flagged = best(True), best(False)
    finally:
        eb.set_dgemm_method(eb.METHOD_AUTO)
    assert torch.equal(torch.nan_to_num(c[True], nan=-1.0), torch.nan_to_num(c[False], nan=-1.0))
    assert torch.isnan(c[True][:, 3]).all() and torch.isnan(c[True]).sum() == n
    assert checked < 0.7 * flagged, (checked, flagged)
