"""The report says which form ran: ``contracted_sets`` row sets (structure-factor form), or 0 (per-atom form)."""
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


def _system(rot):
    cfg = dict(cell=(11.0, 11.5, 12.0), atoms=8, types=2, rmt=2.0, min_sep=3.9, lmax=4, kpts=[(0.1, 0.2, 0.3)],
               n_g=130, seed=6)
    s = synth.make_system(cfg)
    if rot == "classes":
        return synth.with_class_rotations(s, per_type=2)
    return synth.with_rotations(s) if rot == "own" else s


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("rot,env,sets,shared,classes", [
    ("none", {}, 2, 2, 0), ("classes", {}, 4, 4, 1), ("own", {}, 8, 0, 0), ("none", {"HSDLA_SF": "0"}, 0, 0, 0),
    ("classes", {"HSDLA_CLASSES": "0"}, 0, 0, 0), ("own", {"HSDLA_CLASSES": "0"}, 0, 0, 0)])
def test_report_names_the_form(ctx, monkeypatch, precision, rot, env, sets, shared, classes):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    s = _system(rot)
    ((H, S),), rep = ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0)
    assert rep["contracted_sets"] == sets
    assert rep["num_row_sets"] == shared and rep["rotation_classes"] == classes
    # (the digit form's band configuration exists in the structure-factor form only)
    assert (rep["tile_halves"] > 0) == (sets > 0 and precision == "ozaki")
    Hr, Sr = oracle.reference_hs(s, s.kpoints[0])
    for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (nm, fro, mx)
