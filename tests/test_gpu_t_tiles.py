"""The complex T application on both tile shapes (csrc/ozaki.cu, pair_t_tiles): on each side of the lines by columns (16, 64)
and k-blocks (2L = 98, 162, 338: one, two, three), and more tiles than a wave."""
import pytest

import oracle
from hybridhsdla_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = api.Context()
    yield c
    c.close()


@pytest.mark.parametrize("rot", [False, True])
@pytest.mark.parametrize("atoms,lmax,n_g", [(1, 1, 7), (2, 6, 16), (2, 6, 17), (3, 8, 64), (3, 8, 65), (2, 12, 40), (2, 12, 300),
                                            (30, 12, 260), (60, 2, 700)])
def test_t_application_tiles(ctx, monkeypatch, rot, atoms, lmax, n_g):
    monkeypatch.setenv("HSDLA_SF", "0")
    edge = (125.0 * max(atoms, 2)) ** (1.0 / 3.0)
    s = synth.make_system(dict(cell=(edge, edge, edge), atoms=atoms, types=min(atoms, 2), rmt=2.0, min_sep=3.6, lmax=lmax,
                               kpts=[(0.1, 0.2, 0.3)], n_g=n_g, seed=atoms + n_g))
    if rot:
        s = synth.with_rotations(s)
    ((H, S),), rep = ctx.create_hs(s, precision="ozaki", num_slices=11)
    assert rep["contracted_sets"] == 0
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (nm, fro, mx)
