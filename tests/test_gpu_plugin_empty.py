"""The BLAS-shaped plugin without a product (k = 0, or alpha = 0): the uplo triangle becomes beta C (zero for
beta = 0, even over NaN), with a real diagonal for zherk and zher2k, and the other triangle stays."""
import numpy as np
import pytest

from hybridhsdla_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = api.Context()
    yield c
    c.close()


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("op", ["zherk", "zher2k", "zherkx"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("k,alpha", [(0, 1.0), (0, 0.5), (3, 0.0)])
@pytest.mark.parametrize("beta", [0.0, 1.0, -0.75])
@pytest.mark.parametrize("where", ["device", "host"])
def test_beta_c_without_a_product(ctx, precision, op, uplo, k, alpha, beta, where):
    import torch
    n, ld = 45, 47
    rng = np.random.default_rng(3)
    C0 = rng.standard_normal((ld, n)) + 1j * rng.standard_normal((ld, n))
    tri = np.tril(np.ones((n, n), bool)) if uplo == "L" else np.triu(np.ones((n, n), bool))
    if beta == 0.0:
        C0[:n][tri] = np.nan                 # beta = 0 never reads C
    want = C0.copy()
    want[:n][tri] = 0.0 if beta == 0.0 else beta * C0[:n][tri]
    if op != "zherkx":
        d = np.arange(n)
        want[d, d] = want[d, d].real
    C = torch.from_numpy(np.ascontiguousarray(C0.T))
    A = torch.zeros((n, max(k, 1)), dtype=torch.complex128)
    if where == "device":
        C, A = C.cuda(), A.cuda()
    args = (uplo, "C", n, k, alpha, A, max(k, 1)) + (() if op == "zherk" else (A, max(k, 1)))
    getattr(ctx, op)(*args, beta, C, ld, precision=precision)
    got = C.cpu().numpy().T
    assert np.array_equal(got, want, equal_nan=True)
