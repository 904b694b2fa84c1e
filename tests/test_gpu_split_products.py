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


@pytest.mark.parametrize("lmax,types,n_g", [(1, 2, 40), (3, 3, 257), (7, 2, 300), (8, 2, 130), (10, 2, 513)])
def test_t_application_on_pair_tiles(torch, monkeypatch, lmax, types, n_g):
    """T applied per type and per atom on 256 x 256 tiles that reach past a type's 2L rows (8, 32, 128, 162 and 242:
    the rows of the next type or plane, or past the last)."""
    from hybridhsdla_gb300 import synth
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=5, types=types, rmt=2.0, min_sep=3.9, lmax=lmax,
               kpts=[(0.1, 0.2, 0.3)], n_g=n_g, seed=lmax)
    ctx = api.Context()
    try:
        for rot in (False, True):
            s = synth.make_system(cfg)
            s = synth.with_rotations(s) if rot else s
            monkeypatch.setenv("HSDLA_SF", "0")
            monkeypatch.setenv("HSDLA_CLASSES", "0")
            ((H, S),), rep = ctx.create_hs(s, precision="ozaki", num_slices=11)
            assert rep["num_row_sets"] == 0
            Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
            for X, R in ((H, Hr), (S, Sr)):
                fro, mx = oracle.lower_errors(X, R)
                assert fro < 1e-13 and mx < 1e-13, (lmax, rot, fro, mx)
    finally:
        ctx.close()


@pytest.mark.parametrize("lmax,atoms,G", [(1, 1, 9), (6, 1, 200), (8, 2, 300), (9, 7, 257), (10, 3, 600)])
def test_contraction_with_split_t(torch, lmax, atoms, G):
    """T applications of few tiles cut over the pairs (one and two k-blocks), then S and H, against the oracle, a
    capped context (nothing cut) and a second call, bit for bit."""
    from hybridhsdla_gb300 import flapw_data
    L = (lmax + 1) ** 2
    rng = np.random.default_rng(lmax * 1000 + G)
    cx = lambda *sh: rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    blocks = []
    for _ in range(atoms):
        aa, bb = cx(L, L), cx(L, L)
        blocks.append((aa + aa.conj().T, cx(L, L), bb + bb.conj().T))
    d = flapw_data.DataIn(L, atoms, G, np.asfortranarray(cx(L * atoms, G)), np.asfortranarray(cx(L * atoms, G)), blocks,
                          np.full(atoms, lmax, np.int32), lmax, np.sqrt(rng.uniform(0.1, 1.0, (atoms, lmax + 1))))
    ctx, capped = api.Context(), api.Context()
    try:
        capped.set_mem_cap(1 << 34)
        H, S, _ = ctx.contract_ab(d, precision="ozaki", num_slices=11)
        H2, S2, _ = ctx.contract_ab(d, precision="ozaki", num_slices=11)
        Hc, Sc, _ = capped.contract_ab(d, precision="ozaki", num_slices=11)
    finally:
        ctx.close()
        capped.close()
    assert np.array_equal(H, H2) and np.array_equal(S, S2)
    Hr, Sr = oracle.stripped_v2(d.L, d.a, d.A, d.B, d.blocks, d.lmaxs, d.max_lmax, d.sqrt_u_norms)
    for X, R in ((H, Hr), (S, Sr), (Hc, Hr), (Sc, Sr)):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (lmax, atoms, G, fro, mx)
