"""Calls that fit a memory cap: the device bytes of a plain FP64 structure-factor call are its T blocks as given and in
real form, H and S, each once, and a workspace of the rows, their T application and the products (or of two of the
per-atom row matrices, which every plan's holds)."""
import numpy as np
import pytest

import oracle
from hybridhsdla_gb300 import api, synth

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = api.Context()
    yield c
    c.close()


@pytest.mark.parametrize("types,lmax,n_g", [(6, 12, 40), (1, 14, 60), (2, 8, 300)])
def test_fp64_call_within_its_own_bytes(ctx, types, lmax, n_g):
    cfg = dict(cell=(11.0, 11.5, 12.0), atoms=max(types, 2), types=types, rmt=2.0, min_sep=3.9, lmax=lmax,
               kpts=[(0.1, 0.2, 0.3)], n_g=n_g, seed=2)
    s = synth.make_system(cfg)
    L, rows = s.L, 2 * s.L * types
    blocks = types * (3 * 16 * L * L + 2 * 8 * (2 * L) ** 2)
    ws = max(8 * rows * n_g * 4 + 3 * 8 * types * n_g * n_g, 2 * 16 * 2 * L * s.num_atoms * n_g)
    rest = ws + 2 * 16 * n_g * n_g
    half = 2 * np.abs(s.kpoints[0].g).max(axis=0)
    tables = 16 * types * int(np.prod(2 * half + 1)) + 16 * s.num_atoms * int((2 * half + 1).sum())
    ctx.set_mem_cap(blocks + rest + tables + MB // 4)
    ((H, S),), _ = ctx.create_hs(s, precision="fp64")
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (nm, fro, mx)
