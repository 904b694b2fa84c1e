"""The structure factors' fixed points (csrc/structure.cu, sf_fixed_points): row sets of very different atom
counts keep their bits beside each other, and their order in the combine is not that of the types."""
import numpy as np
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


def _system(counts, lmax, n_g, nk=1, seed=4):
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=len(counts), types=len(counts), rmt=2.0, min_sep=1.0, lmax=lmax,
               kpts=[(0.1 + 0.1 * i, 0.2, 0.3) for i in range(nk)], n_g=n_g, seed=seed)
    s = synth.make_system(cfg)
    rng = np.random.default_rng(seed)
    s.atom_type = rng.permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)
    s.atom_pos = rng.uniform(0.0, 1.0, (s.atom_type.size, 3))
    return s


@pytest.mark.parametrize("many", [7, 8, 127, 30000])
def test_one_atom_beside_many(ctx, many):
    """All but the whole of H and S comes from a type of one atom (the other's matching rows are 1e-12 of its); its
    structure factors are numbers of magnitude one, held to 2^-53: 12 digits agree with plain FP64 to 2e-14 (FP64 sums of
    2L = 8 terms and the digits: a few 1e-15; a fixed point of 30000 atoms would leave 2^-41 = 4.5e-13)."""
    s = _system([many, 1], 1, 40)
    for x in (s.u, s.u_dr, s.dE_u, s.dE_u_dr):
        x[0] *= 1e12
    ((H, S),), rep = ctx.create_hs(s, precision="ozaki", num_slices=12)
    ((Hd, Sd),), _ = ctx.create_hs(s, precision="fp64")
    assert rep["num_row_sets"] == 2
    for X, R, nm in ((H, Hd, "H"), (S, Sd, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 2e-14 and mx < 2e-14, (nm, many, fro, mx)


@pytest.mark.parametrize("counts", [[1, 9, 1, 40, 2, 300, 1, 5, 80, 3], [2, 3, 2, 3, 2], [1, 1, 1, 1, 8, 8, 8, 8, 64, 64, 64, 64],
                                    [64, 1, 1, 1, 1, 1, 1, 1, 1, 1], [1] * 9 + [500]])
def test_sets_out_of_order(ctx, monkeypatch, counts):
    """Classes of equal and of mixed counts, items cut at their ends, batches that begin inside them.  12 digits: with
    radial data this uneven the truncation of 11 alone comes to 1e-13."""
    s = _system(counts, 2, 45, nk=2)
    whole, _ = ctx.create_hs(s, precision="ozaki", num_slices=12)
    monkeypatch.setenv("HSDLA_TYPE_BATCH", "3")
    cut, _ = ctx.create_hs(s, precision="ozaki", num_slices=12)
    for (H, S), (Hc, Sc), kp in zip(whole, cut, s.kpoints):
        Hr, Sr = oracle.reference_hs(s, kp)
        for X, C, R, nm in ((H, Hc, Hr, "H"), (S, Sc, Sr, "S")):
            for Y in (X, C):
                fro, mx = oracle.lower_errors(Y, R)
                assert fro < 1e-13 and mx < 1e-13, (nm, counts, fro, mx)
