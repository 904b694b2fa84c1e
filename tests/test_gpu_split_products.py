"""Complex Ozaki products whose last wave of tiles is cut over the idle CTA pairs (csrc/ozaki.cu).

Sizes: fewer tiles than pairs (one tile to 66), a whole wave and a remainder (2999 columns: 78 tiles
on 76 pairs), contractions of one k-block (not cut) to many; every part of a tile and the slabs' sum
against numpy, against a capped context (which never cuts) and against a second run, bit for bit.
Tolerance: 1e-13 (relative Frobenius and max-norm of the lower triangle), that of the digit products
with 11 digits; the cut only reorders FP64 additions, a few 1e-16."""
import numpy as np
import pytest

import oracle
from hybridhsdla_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no GPU")
    return t


@pytest.mark.parametrize("n,k,slices", [(1, 2000, 11), (130, 128, 11), (255, 700, 12), (257, 1025, 11), (700, 3000, 11),
                                        (1100, 640, 10), (2600, 300, 11), (2999, 450, 11), (3000, 100, 11)])
def test_split_matches_whole(torch, n, k, slices):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    P, Q = (torch.complex(torch.randn((n, k), generator=g, device="cuda", dtype=torch.float64),
                          torch.randn((n, k), generator=g, device="cuda", dtype=torch.float64)) for _ in range(2))
    ctx, capped = api.Context(), api.Context()
    try:
        capped.set_mem_cap(1 << 34)
        w = torch.rand(k, generator=g, device="cuda", dtype=torch.float64) + 0.5
        a = ctx.zherkx_lower(P, Q, w, precision="ozaki", num_slices=slices).cpu().numpy()
        b = ctx.zherkx_lower(P, Q, w, precision="ozaki", num_slices=slices).cpu().numpy()
        c = capped.zherkx_lower(P, Q, w, precision="ozaki", num_slices=slices).cpu().numpy()
    finally:
        ctx.close()
        capped.close()
    assert np.array_equal(a, b)
    Pn, Qn, wn = P.cpu().numpy().T, Q.cpu().numpy().T, w.cpu().numpy()
    R = Pn.conj().T @ (wn[:, None] * Qn)
    tol = 1e-13 if slices >= 11 else 32e-13
    for X in (a.T, c.T):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < tol and mx < tol, (n, k, fro, mx)
