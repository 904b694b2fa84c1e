"""Plain FP64: a k-point's H and S do not depend on the k-points it is computed with (the tile shape, and
with it the order of the sums, is its own): the same bits alone, in a mesh of its like, and in a mesh of small
and large ones.  Basis sizes on both sides of the tile shapes' line (1216 tiles of 32 on 152 SMs), alone and
together."""
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


def _system(types, lmax, sizes, rot):
    cfg = dict(cell=(11.0, 11.5, 12.0), atoms=6, types=types, rmt=2.0, min_sep=3.9, lmax=lmax, kpts=[], n_g=1, seed=9)
    s = synth.make_system(cfg)
    for i, n in enumerate(sizes):
        k = np.array([0.1 + 0.03 * i, 0.2, 0.3 - 0.05 * i])
        s.kpoints.append(synth.KPoint(k=k, g=synth.g_vectors(s.bmat, k, n)))
    return synth.with_rotations(s) if rot else s


@pytest.mark.parametrize("form", ["row sets", "own rotations", "per atom", "per atom with rotations"])
@pytest.mark.parametrize("types,lmax,sizes", [(1, 3, [700, 701, 699]), (3, 2, [45, 1100, 300, 460]), (2, 4, [1]),
                                              (2, 4, [610, 33])])
def test_alone_and_in_a_mesh(ctx, monkeypatch, form, types, lmax, sizes):
    s = _system(types, lmax, sizes, "rotations" in form)
    if form.startswith("per atom"):
        monkeypatch.setenv("HSDLA_SF", "0")
    mesh, _ = ctx.create_hs(s, precision="fp64")
    for kp, (H, S) in zip(s.kpoints, mesh):
        ((Ha, Sa),), _ = ctx.create_hs(s, kpoints=[kp], precision="fp64")
        assert np.array_equal(H, Ha) and np.array_equal(S, Sa), kp.n_g
