"""The real digit products of the structure-factor form (csrc/real_products.cu): one real product for
S and two for H over the real and imaginary parts of the matching rows, against the oracle.

Sizes where the kernels change course: contraction lengths 2L = 2 (lmax + 1)^2 on both sides of the
64-digit chunks and with one or two K steps in the last (lmax 1: 8, 3: 32, 5: 72, 7: 128, 9: 200, 11:
288, 14: 450), basis sizes around the 128-column and 256-row tiles, 10, 11 and 12 digits (bands of one
and of two diagonals first, every fold of the fixed-point sums).  Tolerance: 1e-13 (relative
Frobenius and max-norm of the lower triangles) for 11 and 12 digits; a digit less multiplies the
truncation error by 2^5, so 32e-13 for 10."""
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


@pytest.mark.parametrize("lmax,n_g,slices", [
    (1, 1, 11), (1, 128, 11), (2, 129, 12), (3, 255, 11), (4, 256, 10), (5, 257, 11), (5, 130, 12), (7, 385, 11),
    (8, 127, 11), (9, 513, 11), (10, 300, 12), (10, 261, 11), (11, 200, 11), (14, 150, 12), (14, 140, 10)])
def test_real_products_match_oracle(ctx, lmax, n_g, slices):
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=5, types=2, rmt=2.0, min_sep=3.9, lmax=lmax,
               kpts=[(0.1, 0.2, 0.3), (-0.2, 0.35, 0.15)], n_g=n_g, seed=100 * lmax + n_g)
    s = synth.make_system(cfg)
    if lmax > 1:
        s.type_lmax = np.asarray([lmax, lmax - 1], np.int32)      # rows above a type's lmax are zero
        s.type_lmax_nonsph = s.type_lmax.copy()
    res, rep = ctx.create_hs(s, precision="ozaki", num_slices=slices)
    assert rep["num_row_sets"] == 2
    tol = 1e-13 if slices >= 11 else 32e-13
    for (H, S), kp in zip(res, s.kpoints):
        Hr, Sr = oracle.reference_hs(s, kp)
        for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
            fro, mx = oracle.lower_errors(X, R)
            assert fro < tol and mx < tol, (nm, lmax, n_g, slices, fro, mx)


@pytest.mark.parametrize("lmax,n_g,types", [(1, 1, 1), (1, 15, 2), (2, 17, 1), (3, 33, 2), (4, 100, 3), (8, 241, 2),
                                            (10, 47, 1), (5, 801, 4), (7, 1000, 2)])
def test_fp64_real_products_match_oracle(ctx, lmax, n_g, types):
    """Plain FP64 on both tile shapes: small launches (16 x 16 tiles, the contraction split over four
    warps; contraction lengths 8 to 242 are not multiples of its steps) and large ones (32 x 32)."""
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=5, types=types, rmt=2.0, min_sep=3.9, lmax=lmax,
               kpts=[(0.1, 0.2, 0.3)], n_g=n_g, seed=7 + n_g)
    s = synth.make_system(cfg)
    ((H, S),), rep = ctx.create_hs(s, precision="fp64")
    assert rep["num_row_sets"] == types
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (nm, lmax, n_g, fro, mx)


@pytest.mark.parametrize("precision", ["ozaki", "fp64"])
@pytest.mark.parametrize("atoms,lmax,n_g", [(1, 2, 40), (3, 6, 130), (18, 3, 257), (35, 1, 300)])
def test_every_atom_its_own_rotation_on_row_sets(ctx, monkeypatch, precision, atoms, lmax, n_g):
    """Every atom a row set of its own (one atom; more sets than a combine batch of 16, with a partial
    last batch; more rotations than the rows kernel's 16 at a time): the oracle, and the per-atom form."""
    edge = (125.0 * max(atoms, 2)) ** (1.0 / 3.0)
    cfg = dict(cell=(edge, edge, edge), atoms=atoms, types=min(atoms, 2), rmt=2.0, min_sep=3.6, lmax=lmax,
               kpts=[(0.1, 0.2, 0.3), (0.0, 0.0, 0.0)], n_g=n_g, seed=31 + atoms)
    s = synth.with_rotations(synth.make_system(cfg))
    res, rep = ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0)
    assert rep["num_row_sets"] == 0 and rep["rotation_classes"] == 0
    monkeypatch.setenv("HSDLA_CLASSES", "0")
    per_atom, rep_pa = ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0)
    for (H, S), (Hp, Sp), kp in zip(res, per_atom, s.kpoints):
        Hr, Sr = oracle.reference_hs(s, kp)
        for X, P, R, nm in ((H, Hp, Hr, "H"), (S, Sp, Sr, "S")):
            fro, mx = oracle.lower_errors(X, R)
            assert fro < 1e-13 and mx < 1e-13, (nm, atoms, lmax, fro, mx)
            assert oracle.lower_errors(X, P)[0] < 1e-13


@pytest.mark.parametrize("precision", ["ozaki", "fp64"])
@pytest.mark.parametrize("types", [1, 2, 3, 4, 5, 6, 7, 8, 9, 13, 16, 17])
def test_combine_over_type_counts(ctx, monkeypatch, precision, types):
    """Every chunk of the combine (4, 2 and 1 types) and sums of more than the eight types that the
    integers hold, whole and cut into batches of three types; a ragged basis of one and a half tiles,
    and many atoms of one type beside single ones (the structure factors' fixed point)."""
    atoms = types + 14
    edge = (125.0 * atoms) ** (1.0 / 3.0)
    cfg = dict(cell=(edge, edge * 1.05, edge * 0.95), atoms=atoms, types=types, rmt=2.0, min_sep=3.6, lmax=3,
               kpts=[(0.1, 0.2, 0.3), (-0.25, 0.0, 0.5)], n_g=49, seed=53 + types)
    s = synth.make_system(cfg)
    first = np.arange(types)
    s.atom_type = np.concatenate([first, np.full(14, types - 1)]).astype(s.atom_type.dtype)
    n_slices = 11 if precision == "ozaki" else 0
    whole, rep = ctx.create_hs(s, precision=precision, num_slices=n_slices)
    assert rep["num_row_sets"] == types
    monkeypatch.setenv("HSDLA_TYPE_BATCH", "3")
    cut, _ = ctx.create_hs(s, precision=precision, num_slices=n_slices)
    for (H, S), (Hc, Sc), kp in zip(whole, cut, s.kpoints):
        Hr, Sr = oracle.reference_hs(s, kp)
        for X, C, R, nm in ((H, Hc, Hr, "H"), (S, Sc, Sr, "S")):
            fro, mx = oracle.lower_errors(X, R)
            assert fro < 1e-13 and mx < 1e-13, (nm, types, fro, mx)
            fro, mx = oracle.lower_errors(C, R)
            assert fro < 1e-13 and mx < 1e-13, (nm, types, fro, mx)


@pytest.mark.parametrize("slices", [2, 3, 4, 6, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("halves,merge", [("2", "1"), ("2", "0"), ("1", "1"), ("1", "0")])
def test_bands_and_issuers(ctx, monkeypatch, slices, halves, merge):
    """Every number of digits (bands of one and two diagonals, odd and even counts of them, chunks in
    which an issuer has no band) with one accumulator and with all of them: the tolerance grows by 2^5 per
    digit left out."""
    monkeypatch.setenv("HSDLA_PAIR_HALVES", halves)
    monkeypatch.setenv("HSDLA_MERGE", merge)
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=5, types=2, rmt=2.0, min_sep=3.9, lmax=5,
               kpts=[(0.1, 0.2, 0.3)], n_g=700, seed=slices)
    s = synth.make_system(cfg)
    ((H, S),), rep = ctx.create_hs(s, precision="ozaki", num_slices=slices)
    assert rep["tile_halves"] == int(halves) and rep["merged_units"] == int(merge)
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    tol = 1e-13 * 32.0 ** max(0, 11 - slices)
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < tol and mx < tol, (nm, slices, fro, mx)
