"""The one-launch FP32 kernel of small products (GPU): sizes around its 32 x 32 tiles and 64-deep K
tiles, both sides of the line to split-BF16, every transpose, padded leading dimensions; NaN beside
the operands must not reach C, and inside them must."""
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def _operands(ta, tb, m, n, k, pad, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + m + n + k)
    ar, ac = (m, k) if ta == "N" else (k, m)
    br, bc = (k, n) if tb == "N" else (n, k)
    a = torch.full((ac + 1, ar + pad), float("nan"), device="cuda")
    b = torch.full((bc + 1, br + pad), float("nan"), device="cuda")
    a[:ac, :ar] = torch.rand((ac, ar), device="cuda", generator=g) * 2 - 1
    b[:bc, :br] = torch.rand((bc, br), device="cuda", generator=g) * 2 - 1
    A = a[:ac, :ar].T if ta == "N" else a[:ac, :ar]
    B = b[:bc, :br].T if tb == "N" else b[:bc, :br]
    return a, b, A.double(), B.double()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 63), (32, 32, 64), (33, 31, 65), (100, 70, 257), (5, 400, 129),
                                   (380, 390, 300), (500, 510, 600), (32, 4096, 1024)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "N"), ("N", "T"), ("T", "T")])
@pytest.mark.parametrize("pad", [0, 3])
def test_small_products(m, n, k, ta, tb, pad):
    a, b, A, B = _operands(ta, tb, m, n, k, pad)
    c0 = torch.rand((n, m + 1), device="cuda")
    c = c0.clone()
    assert eb.sgemm_device(ta, tb, m, n, k, 1.5, a, a.shape[1], b, b.shape[1], 0.5, c, m + 1) == eb.EB2_OK
    info = eb.last_call_info()
    assert info["method"] == eb.METHOD_NATIVE and info["config"] == 6 and info["launches"] == 1, info
    assert torch.equal(c[:, m], c0[:, m])
    exact = 1.5 * (A @ B) + 0.5 * c0[:, :m].T.double()
    # chains of at most 32 FMAs, K / 256 running sums and 8 shares, alpha and beta
    bound = (32 + k / 256 + 1 + 8 + 2) * U * (1.5 * (A.abs() @ B.abs()) + 0.5 * c0[:, :m].T.double().abs())
    assert ((c[:, :m].T.double() - exact).abs() <= bound).all()


def test_the_line_to_split_bf16():
    # one round of 148 tiles: K = 1200 is the last small one; two rounds halve it
    for m, n, k, small in [(148 * 32, 32, 1200, True), (148 * 32, 32, 1201, False), (149 * 32, 32, 600, True),
                           (149 * 32, 32, 601, False)]:
        a, b, A, B = _operands("N", "N", m, n, k, 0)
        c = torch.zeros((n, m), device="cuda")
        assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m) == eb.EB2_OK
        assert (eb.last_call_info()["method"] == eb.METHOD_NATIVE) == small
        exact = A @ B
        err = float((c.T.double() - exact).norm() / exact.norm())
        assert err <= 2.5e-7  # both paths: a few units of 2^-24


def test_non_finite_entries():
    m, n, k = 70, 40, 100
    a, b, A, B = _operands("N", "N", m, n, k, 0)
    a[99, 69] = float("inf")
    b[0, 0] = float("nan")
    c = torch.zeros((n, m), device="cuda")
    assert eb.sgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m) == eb.EB2_OK
    torch.cuda.synchronize()
    bad = ~torch.isfinite(c)
    want = torch.zeros_like(bad)
    want[0, :] = True
    want[:, 69] = True
    assert torch.equal(bad, want)


def test_alpha_zero_and_empty():
    a = torch.full((4, 4), float("nan"), device="cuda")
    c = torch.ones((4, 4), device="cuda")
    assert eb.sgemm_device("N", "N", 4, 4, 4, 0.0, a, 4, a, 4, 0.5, c, 4) == eb.EB2_OK
    assert eb.sgemm_device("N", "N", 4, 4, 0, 1.0, a, 4, a, 4, 0.5, c, 4) == eb.EB2_OK
    torch.cuda.synchronize()
    assert torch.equal(c, torch.full_like(c, 0.25))


@pytest.mark.parametrize("m,n,k", [(9, 103, 39), (70, 40, 200), (33, 31, 1000)])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("T", "T")])
def test_sums_that_overflow(m, n, k, ta, tb):
    # products beyond the FP32 range with both signs: one chain of FMAs stays at the infinity it reaches
    # first, as the FFMA kernel's does, and never turns to NaN
    a, b, A, B = _operands(ta, tb, m, n, k, 2)
    ar, ac = (m, k) if ta == "N" else (k, m)
    a[:ac, :ar] *= 1e30
    b[: b.shape[0] - 1, : b.shape[1] - 2] *= 1e20
    a[:ac, :ar][torch.rand((ac, ar), device="cuda") < 0.5] *= 1e-30  # and some that stay in range
    out = []
    for method in (eb.METHOD_AUTO, eb.METHOD_NATIVE):
        c = torch.zeros((n, m), device="cuda")
        eb.set_sgemm_method(method)
        try:
            assert eb.sgemm_device(ta, tb, m, n, k, 1.0, a, a.shape[1], b, b.shape[1], 0.0, c, m) == eb.EB2_OK
        finally:
            eb.set_sgemm_method(eb.METHOD_AUTO)
        out.append(c)
    torch.cuda.synchronize()
    small, ffma = out
    assert torch.isinf(ffma).any() and not torch.isnan(ffma).any()
    bad = ~torch.isfinite(small)
    assert torch.equal(bad, torch.isinf(ffma))
    assert torch.equal(small[bad], ffma[bad])
