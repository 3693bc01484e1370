"""Split-BF16 SGEMM with K ranges (GPU): tiles of the last, partly filled round of CTAs are summed
over several K ranges.  Grids below one round, at a round's edges and past it, every tile
configuration, ragged K chunks, alpha / beta and padded leading dimensions."""
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def emulated():
    eb.set_sgemm_method(eb.METHOD_EMULATED)
    yield
    eb.set_sgemm_method(eb.METHOD_AUTO)
    eb.set_tile_n(0)


# m, n, k, tile, whether K is cut: few tiles with long K; 149 tiles of 128 x 128 (one past a round of
# 148); 148 (a full round); one chunk only; 3 x 148 + 12 tiles
CASES = [(300, 517, 1100, 256, True), (100, 100, 4000, 128, True), (64, 70, 513, 512, True),
         (149 * 128, 100, 700, 128, True), (148 * 128, 128, 700, 128, False), (300, 300, 256, 256, False),
         (38 * 128, 12 * 128, 600, 128, True), (900, 1300, 2048, 512, True)]


@pytest.mark.parametrize("m,n,k,tile,cut", CASES)
@pytest.mark.parametrize("pieces", [3, 2])
def test_ranges_sum_to_the_product(m, n, k, tile, cut, pieces):
    eb.set_tile_n(tile)
    eb.set_sgemm_pieces(pieces)
    g = torch.Generator(device="cuda").manual_seed(m + k)
    a = torch.rand((k, m + 3), device="cuda", generator=g) * 2 - 1
    b = torch.rand((n, k + 1), device="cuda", generator=g) * 2 - 1
    c0 = torch.rand((n, m + 2), device="cuda", generator=g)
    c = c0.clone()
    try:
        assert eb.sgemm_device("N", "N", m, n, k, 1.5, a, m + 3, b, k + 1, 0.5, c, m + 2) == eb.EB2_OK
        info = eb.last_call_info()
    finally:
        eb.set_sgemm_pieces(3)
    assert info["tile_n"] == tile and (info["splits"] > 1) == cut, info
    assert torch.equal(c[:, m:], c0[:, m:])
    A, B = a[:, :m].T.double(), b[:, :k].T.double()
    exact = 1.5 * (A @ B) + 0.5 * c0[:, :m].T.double()
    # dropped piece products: 3 2^-24 of a term with three pieces, 3 2^-16 with two; the sums of
    # 256-deep chunks truncate in FP32, chunks and ranges add with rounding; two more for alpha, beta
    drop = 3 * 2.0 ** -24 if pieces == 3 else 3 * 2.0 ** -16
    bound = (drop + (16 + k / 256 + 2) * 2.0 ** -24) * 1.5 * (A.abs() @ B.abs()) + 2.0 ** -23
    assert ((c[:, :m].T.double() - exact).abs() <= bound).all()


def test_non_finite_entry_leaves_c_to_the_fallback():
    eb.set_tile_n(256)
    m, n, k = 90, 70, 1500
    a = torch.rand((k, m), device="cuda")
    b = torch.rand((n, k), device="cuda")
    a[1499, 89] = float("inf")
    c0 = torch.rand((n, m), device="cuda")
    c, want = c0.clone(), c0.clone()
    assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.5, c, m) == eb.EB2_OK
    assert eb.last_call_info()["splits"] > 1
    eb.set_sgemm_method(eb.METHOD_NATIVE)
    assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.5, want, m) == eb.EB2_OK
    torch.cuda.synchronize()
    assert torch.equal(c, want)
