"""Atoms with rotations of their own: row sets of one atom where they fit, else the per-atom form, which streams its
contraction in atom panels: by the workspace budget and by the context's memory cap.  A cap that the per-atom form
fits never refuses the call, whatever the row sets would have taken."""
import pytest

import oracle
from hybridhsdla_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _context():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    return api.Context()


def _system(atoms, lmax, n_g):
    edge = (125.0 * atoms) ** (1.0 / 3.0)
    cfg = dict(cell=(edge, edge, edge), atoms=atoms, types=2, rmt=2.0, min_sep=3.6, lmax=lmax, kpts=[(0.1, 0.2, 0.3)],
               n_g=n_g, seed=11)
    return synth.with_rotations(synth.make_system(cfg))


def _check(res, s):
    for (H, S), kp in zip(res, s.kpoints):
        Hr, Sr = oracle.reference_hs(s, kp)
        for X, R, nm in ((H, Hr, "H"), (S, Sr, "S")):
            fro, mx = oracle.lower_errors(X, R)
            assert fro < 1e-13 and mx < 1e-13, (nm, fro, mx)


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("budget,sets", [(1 << 30, 12), (1 << 20, 0)])
def test_by_workspace_budget(monkeypatch, precision, budget, sets):
    monkeypatch.setenv("HSDLA_WORKSPACE_BUDGET", str(budget))
    ctx = _context()
    s = _system(12, 5, 150)
    res, rep = ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0)
    assert rep["contracted_sets"] == sets
    assert (rep["num_panels"] > 1) == (precision == "ozaki" and not sets)
    _check(res, s)
    ctx.close()


def _accepted(s, cap, **args):
    ctx = _context()
    ctx.set_mem_cap(cap)
    try:
        return ctx.create_hs(s, **args)
    except api.HsdlaError as e:
        assert e.code == -3, e
        return None
    finally:
        ctx.close()


@pytest.mark.parametrize("atoms,lmax,n_g,slices", [(12, 5, 150, 11), (24, 8, 300, 11), (6, 10, 60, 0)])
def test_by_memory_cap(monkeypatch, atoms, lmax, n_g, slices):
    s = _system(atoms, lmax, n_g)
    args = dict(precision="ozaki", num_slices=slices, tmats=api.prepare_tmats(s))
    forms = set()
    for mb in (4, 6, 8, 11, 14, 18, 23, 29, 36, 45, 56, 70, 88, 110, 140, 180, 230, 300, 400):
        got = _accepted(s, mb << 20, **args)
        if got is None:
            with monkeypatch.context() as m:
                m.setenv("HSDLA_CLASSES", "0")
                assert _accepted(s, mb << 20, **args) is None, mb
        else:
            forms.add(got[1]["contracted_sets"])
            _check(got[0], s)
    # (with the slice count tuned, the tuner's buffers are the most that either form holds)
    assert atoms in forms and (0 in forms or slices == 0)
