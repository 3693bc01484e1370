"""The CRT reconstruction's runs of columns (GPU): shapes around the blocks' runs (few or many row
blocks, a last run that is short, fewer columns than runs, more than one 32-column sum of the error
estimate per run), with and without the accuracy check, beta != 0 and a padded C."""
import pytest
import torch

import eigen_b200 as eb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def crt_method():
    eb.set_dgemm_method(eb.METHOD_CRT)
    yield
    eb.set_dgemm_method(eb.METHOD_AUTO)


@pytest.mark.parametrize("m,n", [(1, 1), (1, 2367), (255, 2369), (256, 593), (257, 600), (1025, 149), (5000, 9),
                                 (40000, 5), (300, 20003)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("check", [False, True])
def test_runs(m, n, beta, check):
    k = 24
    g = torch.Generator(device="cuda").manual_seed(m + n)
    # integers below 2^15, so that the product and beta C are exact in FP64
    a = torch.randint(-(2 ** 15), 2 ** 15, (k, m), device="cuda", generator=g).double()
    b = torch.randint(-(2 ** 15), 2 ** 15, (n, k), device="cuda", generator=g).double()
    c = torch.randint(-64, 64, (n, m + 3), device="cuda", generator=g).double() * 2
    ref = beta * c[:, :m] + b @ a
    pad = c[:, m:].clone()
    rc = eb.dgemm_device("N", "N", m, n, k, 1.0, a, m, b, k, beta, c, m + 3, check_accuracy=check)
    torch.cuda.synchronize()
    assert rc == eb.EB2_OK
    assert torch.equal(c[:, :m], ref)
    assert torch.equal(c[:, m:], pad)
