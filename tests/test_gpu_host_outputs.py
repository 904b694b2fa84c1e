"""Host arrays of the host entry points: pages of pageable outputs that are not in memory yet, and
contraction inputs uploaded through the output buffer."""
import numpy as np
import pytest

import oracle
from hybridhsdla_gb300 import api, flapw_data, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = api.Context()
    yield c
    c.close()


@pytest.mark.parametrize("precision", ["fp64", "ozaki"])
@pytest.mark.parametrize("n_g,pad", [(1, 0), (37, 0), (513, 1), (700, 3), (300, 20000), (1100, 9000)])
def test_untouched_outputs(ctx, n_g, pad, precision):
    """Fresh (never touched) outputs, dense and with columns many pages apart: the same H and S as in
    outputs that are in memory, nothing written outside the lower triangles' column blocks."""
    cfg = dict(cell=(10.0, 10.5, 11.0), atoms=5, types=2, rmt=2.0, min_sep=3.9, lmax=2,
               kpts=[(0.1, 0.2, 0.3)], n_g=n_g, seed=n_g)
    s = synth.make_system(cfg)
    held = tuple(np.full((n_g, n_g), 7.0 + 0j, order="F") for _ in range(2))
    for m in held:
        m[:] = 0.0
    ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0, out=[held])
    fresh = tuple(np.zeros((n_g + pad, n_g), np.complex128, order="F") for _ in range(2))
    ctx.create_hs(s, precision=precision, num_slices=11 if precision == "ozaki" else 0, out=[fresh])
    for a, b in zip(held, fresh):
        assert np.array_equal(np.tril(a), np.tril(b[:n_g]))
        assert not b[n_g:].any()


@pytest.mark.parametrize("lmax,atoms,G", [(0, 1, 1), (2, 3, 1), (2, 5, 3), (3, 7, 12), (4, 9, 20), (1, 2, 40), (5, 3, 70)])
def test_contract_inputs_in_pieces(ctx, lmax, atoms, G):
    """A and B copied strided (bases too small), in several pieces with a partial last one, and whole.
    Tolerance: 1e-13 (relative Frobenius and max-norm), as for every contraction of the oracle."""
    L = (lmax + 1) ** 2
    rng = np.random.default_rng(100 * lmax + G)
    cx = lambda *sh: rng.standard_normal(sh) + 1j * rng.standard_normal(sh)
    blocks = []
    for _ in range(atoms):
        aa, bb = cx(L, L), cx(L, L)
        blocks.append((aa + aa.conj().T, cx(L, L), bb + bb.conj().T))
    d = flapw_data.DataIn(L, atoms, G, np.asfortranarray(cx(L * atoms, G)), np.asfortranarray(cx(L * atoms, G)), blocks,
                          np.full(atoms, lmax, np.int32), lmax, np.sqrt(rng.uniform(0.1, 1.0, (atoms, lmax + 1))))
    H, S, _ = ctx.contract_ab(d, precision="fp64")
    Hr, Sr = oracle.stripped_v2(d.L, d.a, d.A, d.B, d.blocks, d.lmaxs, d.max_lmax, d.sqrt_u_norms)
    for X, R in ((H, Hr), (S, Sr)):
        fro, mx = oracle.lower_errors(X, R)
        assert fro < 1e-13 and mx < 1e-13, (fro, mx)
