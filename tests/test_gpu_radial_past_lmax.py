"""Radial values past a type's own lmax are not part of the input (the library checks those up to lmax
only): NaN and infinities there change nothing, in both precisions, with types, with (type, rotation)
classes, with a rotation per atom, and in the per-atom form."""
import numpy as np
import pytest

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


def _system(rot):
    cfg = dict(cell=(11.0, 11.5, 12.0), atoms=8, types=2, rmt=2.0, min_sep=3.9, lmax=5, kpts=[(0.1, 0.2, 0.3)],
               n_g=150, seed=5)
    s = synth.make_system(cfg)
    s.type_lmax = np.asarray([5, 3], np.int32)
    s.type_lmax_nonsph = s.type_lmax.copy()
    if rot == "classes":
        return synth.with_class_rotations(s, per_type=2)
    return synth.with_rotations(s) if rot == "own" else s


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("rot,sf", [("none", "1"), ("classes", "1"), ("own", "1"), ("none", "0"), ("own", "0")])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_values_past_a_types_lmax_are_ignored(ctx, monkeypatch, precision, rot, sf, value):
    monkeypatch.setenv("HSDLA_SF", sf)
    s = _system(rot)
    tm = api.prepare_tmats(s)
    args = dict(precision=precision, num_slices=11 if precision == "ozaki" else 0, tmats=tm)
    (clean,), _ = ctx.create_hs(s, **args)
    for x in (s.u, s.u_dr, s.dE_u, s.dE_u_dr, s.dE_u_norm):
        x[1, 4:] = value
    (marked,), _ = ctx.create_hs(s, **args)
    for X, Y in zip(marked, clean):
        assert np.array_equal(X, Y)
