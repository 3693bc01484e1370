"""The diagonal-block solve of ?trsm_ (GPU) at the sizes where it changes: blocks around its 16-row
sub-blocks and the largest block, vector counts around the 16, 32 and 64 vectors a CTA takes, every
side, triangle and transpose.  The triangle that the routine must not read, and the diagonal of a
unit triangle, hold NaN."""
import numpy as np
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


def _solve(dtype, side, uplo, trans, diag, m, n, alpha=1.0):
    td = torch.float64 if dtype == "d" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n)
    order = m if side == "L" else n
    full = (torch.rand((order, order), dtype=td, device="cuda", generator=g) * 2 - 1) / order ** 0.5
    full.diagonal().copy_(1 + torch.rand(order, dtype=td, device="cuda", generator=g))
    tri = torch.triu(full) if uplo == "U" else torch.tril(full)  # row-major view of the matrix
    ref = tri.clone()
    if diag == "U":
        ref.diagonal().fill_(1.0)
    stored = torch.where(tri != 0, tri, torch.full_like(tri, float("nan")))
    if diag == "U":
        stored.diagonal().fill_(float("nan"))
    lda, ldb = order + 3, m + 1
    a = torch.full((order, lda), float("nan"), dtype=td, device="cuda")
    a[:, :order] = stored.T  # column-major
    b = torch.rand((n, ldb), dtype=td, device="cuda", generator=g) * 2 - 1
    x = b.clone()
    torch.cuda.synchronize()
    eb.level3("dtrsm" if dtype == "d" else "strsm", side, uplo, trans, diag, m, n, alpha, a, lda, x, ldb)
    assert eb.last_error()[0] == eb.EB2_OK, eb.last_error()
    assert torch.equal(x[:, m:], b[:, m:])
    op = (ref if trans == "N" else ref.T).double()
    X, B = x[:, :m].T.double(), b[:, :m].T.double() * alpha
    res = (op @ X if side == "L" else X @ op) - B
    # substitution is backward stable: |op(A) X - B| <= order u |op(A)| |X|, entry by entry (one
    # more u for alpha, and the residual's own FP64 sums)
    u = 2.0 ** -53 if dtype == "d" else 2.0 ** -24
    scale = op.abs() @ X.abs() if side == "L" else X.abs() @ op.abs()
    bound = (2 * order + 4) * u * scale + 4 * u * B.abs()
    assert (res.abs() <= bound).all(), float((res.abs() / bound).max())


@pytest.mark.parametrize("dtype", ["d", "s"])
@pytest.mark.parametrize("order", [1, 15, 16, 17, 100, 255, 256])
@pytest.mark.parametrize("side,uplo,trans,diag", [("L", "L", "N", "N"), ("L", "U", "N", "U"), ("R", "L", "T", "N"),
                                                  ("R", "U", "N", "N"), ("L", "L", "T", "U")])
def test_block_edges(dtype, order, side, uplo, trans, diag):
    m, n = (order, 37) if side == "L" else (37, order)
    _solve(dtype, side, uplo, trans, diag, m, n, alpha=1.5)


@pytest.mark.parametrize("dtype", ["d", "s"])
@pytest.mark.parametrize("count", [1, 16 * 148, 16 * 148 + 1, 32 * 148 + 1, 9001])
@pytest.mark.parametrize("side", ["L", "R"])
def test_vectors_per_block(dtype, count, side):
    m, n = (40, count) if side == "L" else (count, 40)
    _solve(dtype, side, "L", "N", "N", m, n)


@pytest.mark.parametrize("dtype", ["d", "s"])
@pytest.mark.parametrize("count", [37, 16 * 148 + 1, 32 * 148 + 1])
def test_block_error(dtype, count):
    """A vector entry is rounded at its own size once per 16-row sub-block above it (8 on average in 256
    rows), by half of its own sub-block's 15 updates, its reciprocal and its product: about 17.5
    independent roundings, each of variance at most u^2 / 3 of the entry.  (Rounded by every one of
    the 128 rows above it on average, the error would be 2.4 times the bound.)"""
    td = torch.float64 if dtype == "d" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(count)
    order = 256
    a = (torch.rand((order, order), dtype=td, device="cuda", generator=g) * 2 - 1) / 16
    a.diagonal().uniform_(1, 2, generator=g)
    b = torch.rand((count, order), dtype=td, device="cuda", generator=g) * 2 - 1
    x = b.clone()
    torch.cuda.synchronize()
    eb.level3("dtrsm" if dtype == "d" else "strsm", "L", "L", "N", "N", order, count, 1.0, a, order, x, order)
    low = np.tril(a.cpu().numpy().T).astype(np.longdouble)
    ref = b.cpu().numpy().T[:, :32].astype(np.longdouble)
    for c in range(order):
        ref[c] /= low[c, c]
        ref[c + 1:] -= low[c + 1:, c:c + 1] * ref[c]
    err = np.sqrt((((x.cpu().numpy().T[:, :32] - ref) ** 2).sum()) / (ref ** 2).sum())
    u = 2.0 ** -53 if dtype == "d" else 2.0 ** -24
    assert err <= u * np.sqrt(17.5 / 3)
