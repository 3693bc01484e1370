"""The split of FP32 operands into BF16 pieces (GPU): both storage directions, aligned and unaligned
leading dimensions, ragged edges, and the NaN/Inf test at every place of a tile."""
import numpy as np
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def emulated():
    eb.set_sgemm_method(eb.METHOD_EMULATED)
    yield
    eb.set_sgemm_method(eb.METHOD_AUTO)


def _call(ta, tb, m, n, k, a, lda, b, ldb):
    c = torch.zeros((n, m), dtype=torch.float32, device="cuda")
    assert eb.sgemm_device(ta, tb, m, n, k, 1.0, a, lda, b, ldb, 0.0, c, m) == eb.EB2_OK
    return c


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 70, 65), (128, 64, 64), (95, 257, 130), (160, 96, 1000)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_product_of_the_pieces(m, n, k, ta, tb, pad):
    g = torch.Generator(device="cuda").manual_seed(k)
    rows_a, cols_a = (m, k) if ta == "N" else (k, m)
    rows_b, cols_b = (k, n) if tb == "N" else (n, k)
    lda, ldb = rows_a + pad, rows_b + pad
    a = torch.rand((cols_a, lda), device="cuda", generator=g) * 2 - 1
    b = torch.rand((cols_b, ldb), device="cuda", generator=g) * 2 - 1
    c = _call(ta, tb, m, n, k, a, lda, b, ldb)
    opa = (a[:, :m].T if ta == "N" else a[:, :k]).double()
    opb = (b[:, :k].T if tb == "N" else b[:, :n]).double()
    exact = opa @ opb
    # dropped piece products 3 2^-24 per term, FP32 sums of 256-deep chunks that truncate (8 bits of
    # chunk depth) and of the chunks
    bound = (3 + 16 + k / 256) * 2.0 ** -24 * (opa.abs() @ opb.abs())
    assert ((c.T.double() - exact).abs() <= bound).all()


@pytest.mark.parametrize("ta", ["N", "T"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf"), 3.4e38])
def test_non_finite_entries_are_seen(ta, bad):
    m, n, k = 40, 24, 72
    for r, l in [(0, 0), (39, 71), (17, 63), (31, 64), (32, 1), (5, 38)]:
        a = torch.full((k, m) if ta == "N" else (m, k), 0.5, device="cuda")
        a[(l, r) if ta == "N" else (r, l)] = bad
        b = torch.ones((n, k), device="cuda")
        got = _call(ta, "N", m, n, k, a, m if ta == "N" else k, b, k)
        eb.set_sgemm_method(eb.METHOD_NATIVE)
        want = _call(ta, "N", m, n, k, a, m if ta == "N" else k, b, k)
        eb.set_sgemm_method(eb.METHOD_EMULATED)
        torch.cuda.synchronize()
        # 3.4e38 rounds up to infinity as a BF16 piece: the FP32 kernel takes it too
        assert torch.equal(torch.nan_to_num(got, nan=1.25), torch.nan_to_num(want, nan=1.25))
