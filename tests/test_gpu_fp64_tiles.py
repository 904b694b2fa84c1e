"""The complex FP64 products (csrc/contract_fp64.cu) on both tile shapes: small launches on 16 x 16 tiles with the
contraction split over four warps, large ones on 32 x 32.  Ends of tiles and of the contraction's steps of four
(and fewer steps than warps), with and without row weights, against numpy.  Tolerance: 1e-13 (relative
Frobenius and max-norm of the lower triangle), as for every FP64 product here."""
import numpy as np
import pytest

import oracle
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


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n,k", [(1, 1), (15, 3), (16, 4), (17, 13), (31, 162), (33, 98), (250, 17), (481, 242),
                                 (1552, 6), (1601, 33), (2113, 50)])
def test_fp64_tiles(ctx, n, k, weighted):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + k)
    P, Q = (torch.complex(torch.randn((n, k), generator=g, device="cuda", dtype=torch.float64),
                          torch.randn((n, k), generator=g, device="cuda", dtype=torch.float64)) for _ in range(2))
    w = torch.rand(k, generator=g, device="cuda", dtype=torch.float64) + 0.5 if weighted else None
    X = ctx.zherkx_lower(P, Q, w, precision="fp64").cpu().numpy().T
    Pn, Qn = P.cpu().numpy().T, Q.cpu().numpy().T
    R = Pn.conj().T @ (w.cpu().numpy()[:, None] * Qn if weighted else Qn)
    fro, mx = oracle.lower_errors(X, R)
    assert fro < 1e-13 and mx < 1e-13, (n, k, fro, mx)
    assert not np.triu(X, 1).any()


@pytest.mark.parametrize("sf", ["1", "0"])
def test_groups_sum_in_one_order(ctx, monkeypatch, sf):
    """Three k-points whose launches take 32 x 32 tiles together and would take split ones alone: the same bits in one
    group and in groups of one k-point."""
    import torch
    from hybridhsdla_gb300 import synth
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=2, types=1, rmt=2.0, min_sep=3.9, lmax=2,
               kpts=[(0.1, 0.2, 0.3), (0.0, 0.25, -0.1), (0.4, 0.1, 0.2)], n_g=700, seed=3)
    s = synth.make_system(cfg)
    monkeypatch.setenv("HSDLA_SF", sf)
    monkeypatch.setenv("HSDLA_TYPE_BATCH", "1")
    monkeypatch.setenv("HSDLA_PANELS", "1")
    outs = []
    for budget in (None, "1"):
        if budget:
            monkeypatch.setenv("HSDLA_WORKSPACE_BUDGET", budget)
        pl = ctx.plan(s, precision="fp64")
        o = pl.alloc_outputs()
        pl.execute(o)
        torch.cuda.synchronize()
        outs.append([(h.cpu().numpy(), v.cpu().numpy()) for h, v in o])
        pl.close()
    for (h1, s1), (h2, s2) in zip(*outs):
        assert np.array_equal(h1, h2) and np.array_equal(s1, s2)


@pytest.mark.parametrize("lmax,n_g", [(4, 2017), (3, 3903)])
def test_weighted_rows_of_whole_tiles(ctx, lmax, n_g):
    """T applications on 32 x 32 tiles (1216 of them on 152 SMs), which also write the weighted rows of S."""
    from hybridhsdla_gb300 import synth
    cfg = dict(cell=(14.0, 14.5, 15.0), atoms=5, types=5, rmt=2.0, min_sep=4.1, lmax=lmax, kpts=[(0.1, 0.2, 0.3)], n_g=n_g,
               seed=n_g)
    s = synth.make_system(cfg)
    ((H, S),), rep = ctx.create_hs(s, precision="fp64")
    assert rep["num_row_sets"] == 5
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (nm, lmax, n_g, fro, mx)
