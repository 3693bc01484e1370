"""The CRT product's residue planes (GPU): four neighbouring columns of a row share a word, and the
256 x 256 tile hands its accumulator back one row half after the other.  Sizes around groups of
four columns and around whole tiles, every tile configuration, triangles, K beyond one INT32
unit, more than 16 moduli, split K: all give the bits of the 128 x 256 tile, and those the exact
product of the scaled operands."""
import numpy as np
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def crt_method():
    eb.set_dgemm_method(eb.METHOD_CRT)
    yield
    eb.set_dgemm_method(eb.METHOD_AUTO)
    eb.set_tile_n(0)
    eb.set_dgemm_moduli(0)
    eb.set_config(-1)


def _operands(m, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.rand((k, m), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    b = torch.rand((n, k), dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    return a, b


def _product(a, b, beta=0.0, c0=None):
    k, m = a.shape
    n = b.shape[0]
    c = torch.full((n, m + 2), 7.0, dtype=torch.float64, device="cuda") if c0 is None else c0.clone()
    assert eb.dgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, beta, c, m + 2) == eb.EB2_OK
    return c


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 3, 130), (32, 4, 128), (33, 5, 129), (256, 255, 300), (257, 258, 64),
                                   (511, 513, 200), (520, 1027, 100)])
@pytest.mark.parametrize("moduli", [16, 11, 20])
def test_tiles_agree(m, n, k, moduli):
    a, b = _operands(m, n, k, m + n)
    eb.set_dgemm_moduli(moduli)
    c0 = torch.rand((n, m + 2), dtype=torch.float64, device="cuda")
    eb.set_tile_n(256)
    base, upd = _product(a, b), _product(a, b, 0.5, c0)
    assert torch.equal(base[:, m:], torch.full_like(base[:, m:], 7.0))
    for tile in (512, 1024):
        eb.set_tile_n(tile)
        assert torch.equal(_product(a, b), base)
        assert torch.equal(_product(a, b, 0.5, c0), upd)
    if moduli >= 16:
        # b >= 62 bits per row of the operands: the product's own rounding is what is left
        exact = (b.cpu().numpy().astype(np.longdouble) @ a.cpu().numpy().astype(np.longdouble))
        got = base[:, :m].cpu().numpy()
        assert np.all(np.abs(got - exact) <= 2.0 ** -52 * np.abs(exact) + 2.0 ** -58 * np.sqrt(k))


@pytest.mark.parametrize("tile", [512, 1024])
def test_long_k_adds_units(tile):
    # 1023 blocks of 128 fill one INT32 unit: three units, a ragged last one
    a, b = _operands(70, 9, 128 * 1023 * 2 + 777, 3)
    eb.set_tile_n(256)
    base = _product(a, b)
    eb.set_tile_n(tile)
    assert torch.equal(_product(a, b), base)


def test_split_k_agrees():
    a, b = _operands(300, 70, 6000, 4)
    base = _product(a, b)
    eb.set_config(5)
    assert torch.equal(_product(a, b), base)
    assert eb.last_call_info()["splits"] > 1


@pytest.mark.parametrize("uplo", ["U", "L"])
@pytest.mark.parametrize("n", [30, 259, 700])
def test_triangle_writes_its_side_only(uplo, n):
    a, _ = _operands(n, 1, 200, n)
    full = torch.full((n, n), 3.0, dtype=torch.float64, device="cuda")
    assert eb.dgemm_device("N", "T", n, n, 200, 1.0, a, n, a, n, 0.0, full, n) == eb.EB2_OK
    c = torch.full((n, n), 3.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    eb.level3("dsyrk", uplo, "N", n, 200, 1.0, a, n, 0.0, c, n)
    i = torch.arange(n, device="cuda")
    kept = (i[None, :] <= i[:, None]) if uplo == "U" else (i[None, :] >= i[:, None])  # c[j, i]
    assert torch.equal(c[kept], full[kept]) and (c[~kept] == 3.0).all()


@pytest.mark.parametrize("check", [True, False])
@pytest.mark.parametrize("which", ["a", "b", "none"])
def test_non_finite_operand_takes_the_fp64_kernel(check, which):
    a, b = _operands(260, 130, 150, 9)
    if which == "a":
        a[149, 259] = float("inf")
    if which == "b":
        b[129, 0] = float("nan")
    c0 = torch.rand((130, 260), dtype=torch.float64, device="cuda")
    c, want = c0.clone(), c0.clone()
    assert eb.dgemm_device("N", "N", 260, 130, 150, 1.5, a, 260, b, 150, 0.5, c, 260, check_accuracy=check) == eb.EB2_OK
    torch.cuda.synchronize()
    if which != "none":
        eb.set_dgemm_method(eb.METHOD_NATIVE)
        assert eb.dgemm_device("N", "N", 260, 130, 150, 1.5, a, 260, b, 150, 0.5, want, 260) == eb.EB2_OK
        assert torch.equal(torch.nan_to_num(c, nan=5e300), torch.nan_to_num(want, nan=5e300))
    else:
        assert torch.isfinite(c).all()


def test_rows_without_a_nonzero():
    a, b = _operands(100, 60, 300, 8)
    a[:, 3] = 0.0
    b[7, :] = 0.0
    a[:, 50] *= 2.0 ** -900
    c = _product(a, b)
    assert (c[:, 3] == 0).all() and (c[7, :100] == 0).all()
    exact = b.cpu().numpy().astype(np.longdouble) @ a.cpu().numpy().astype(np.longdouble)
    got = c[:, :100].cpu().numpy()
    rows = np.abs(a.cpu().numpy()).max(axis=0)
    assert np.all(np.abs(got - exact) <= 2.0 ** -52 * np.abs(exact) + 2.0 ** -54 * rows[None, :])
