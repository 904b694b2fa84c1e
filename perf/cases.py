"""What the speed of this framework is judged by: the H/S generation path over its real range,
through the entry points a user's program calls.

Kinds of case (``case["kind"]``):

* ``plan``      device-resident: a ``Plan`` kept by the caller, ``execute`` into device H and S
                (what an eigensolver on the same GPU reads next);
* ``host``      the drop-in ``create_hs``: plain arrays in, host H and S out, one call per k-point
                (``pinned``: page-locked outputs, as a program that keeps its buffers has them);
* ``contract``  the contraction-only drop-in ``contract_ab``: caller-built A, B and T blocks;
* ``plugin``    the BLAS-shaped backend (``zherk``, ``zher2k``, ``zherkx``) on device matrices;
* ``pack``      the packed hand-off ``pack_lower`` of a device H.

Cells follow the repository's synthetic configurations (``synth.CONFIGS``): ~125 bohr^3 per atom,
R_MT 2.0, seeded radial data and T blocks, shifted k-points.  One library context per process.
"""
import math

import numpy as np
import torch

from hybridhsdla_gb300 import api, flapw_data, synth

_CTX = None


def _ctx():
    global _CTX
    if _CTX is None:
        _CTX = api.Context(0)
    return _CTX


def _hs(name, kind, precision, n_g, atoms, types, lmax, rot="none", nk=1, graph=False, pinned=False):
    return {"name": name, "kind": kind, "precision": precision, "n_g": n_g, "atoms": atoms, "types": types,
            "lmax": lmax, "rot": rot, "nk": nk, "graph": graph, "pinned": pinned}


def _blas(name, op, precision, n, k, uplo, trans):
    return {"name": name, "kind": "plugin", "op": op, "precision": precision, "n": n, "k": k, "uplo": uplo,
            "trans": trans}


def listed():
    return [
        # the reference's own sample: two atoms of two types, lmax 8, 235 plane waves, plain FP64
        _hs("two_atoms_host_fp64", "host", "fp64", 235, 2, 2, 8),
        # a small cell inside a self-consistency loop: latency and launches
        _hs("small_plan_ozaki", "plan", "ozaki", 501, 4, 2, 6),
        # medium cell, the drop-in with page-locked buffers, odd basis size
        _hs("medium_host_ozaki", "host", "ozaki", 2999, 32, 4, 8, pinned=True),
        # medium cell in plain FP64 on the device
        _hs("medium_plan_fp64", "plan", "fp64", 3000, 32, 4, 8),
        # the headline size: 128 atoms of 8 types, lmax 10
        _hs("headline_plan_ozaki", "plan", "ozaki", 8000, 128, 8, 10),
        # the largest: a basis of 12001 plane waves
        _hs("large_plan_ozaki", "plan", "ozaki", 12001, 128, 8, 10),
        # a k-mesh in one captured plan, uneven basis sizes (~6000-6600), 64 atoms of 4 types
        _hs("kmesh_graph_ozaki", "plan", "ozaki", 6300, 64, 4, 8, nk=4, graph=True),
        # a dump with symmetry: each type's atoms in two rotation classes
        _hs("symmetry_classes_ozaki", "plan", "ozaki", 3001, 32, 4, 8, rot="classes"),
        # every atom its own rotation: the general form
        _hs("own_rotations_ozaki", "plan", "ozaki", 2003, 32, 4, 8, rot="own"),
        # the contraction-only drop-in on the caller's host arrays
        {"name": "contract_host_ozaki", "kind": "contract", "precision": "ozaki", "n_g": 1501, "atoms": 8, "lmax": 8},
        # the contraction backend: H = B^H X + X^H B of a medium cell
        _blas("zher2k_device_ozaki", "zher2k", "ozaki", 2999, 2592, "L", "C"),
        # hand-off of a finished H to a packed eigensolver
        {"name": "pack_device", "kind": "pack", "n": 8000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "host", "host", "contract", "plugin", "plugin", "pack"])
    if kind == "pack":
        return {"kind": "pack", "n": _log(rng, 100, 12000)}
    if kind == "plugin":
        precision = rng.choice(["ozaki", "ozaki", "fp64"])
        top = 3000 if precision == "ozaki" else 1200
        return {"kind": "plugin", "op": rng.choice(["zherk", "zher2k", "zherkx"]), "precision": precision,
                "n": _log(rng, 100, top), "k": _log(rng, 100, top), "uplo": rng.choice("LU"), "trans": rng.choice("NC")}
    if kind == "contract":
        return {"kind": "contract", "precision": rng.choice(["ozaki", "fp64"]), "n_g": _log(rng, 100, 1500),
                "atoms": rng.randint(1, 8), "lmax": rng.randint(4, 10)}
    precision = rng.choice(["ozaki", "ozaki", "ozaki", "fp64"])
    lmax = rng.randint(4, 10)
    types = rng.randint(1, 8)
    per = rng.randint(1, 16)
    rot = rng.choice(["none", "none", "none", "classes", "own"])
    nk = rng.choice([1, 1, 1, 2, 3])
    graph = kind == "plan" and rng.random() < 0.3
    if precision == "fp64":
        n_g = _log(rng, 150, 2500)
    elif rot == "own":
        n_g = _log(rng, 150, 2500)
    else:
        n_g = _log(rng, 150, 8000)
    if kind == "host":
        n_g = min(n_g, 4000)
    if rot == "own":
        per = min(per, 8)
    return {"kind": kind, "precision": precision, "n_g": n_g, "atoms": per * types, "types": types, "lmax": lmax,
            "rot": rot, "nk": nk, "graph": graph, "pinned": kind == "host" and rng.random() < 0.5}


# ------------------------------------------------------------------------------- inputs
def _system(case, seed):
    atoms = case["atoms"]
    edge = (125.0 * max(atoms, 2)) ** (1.0 / 3.0)
    rng = np.random.default_rng([seed, 17])
    n_g, nk = case["n_g"], case.get("nk", 1)
    cfg = dict(cell=(edge, edge, edge), atoms=atoms, types=case.get("types", atoms), rmt=2.0,
               min_sep=4.0 if atoms > 2 else 3.6, lmax=case["lmax"], kpts=[], n_g=n_g, seed=seed)
    s = synth.make_system(cfg)
    # shifted k-points; a mesh's basis sizes spread over 0.95 to 1.05 of n_g
    for i in range(nk):
        k = rng.uniform(0.05, 0.45, 3)
        size = n_g if nk == 1 else int(n_g * (0.95 + 0.1 * ((i + 1) * 0.618 % 1.0)))
        s.kpoints.append(synth.KPoint(k=k, g=synth.g_vectors(s.bmat, k, size)))
    if case.get("rot") == "classes":
        s = synth.with_class_rotations(s, per_type=2, seed=seed)
    elif case.get("rot") == "own":
        s = synth.with_rotations(s, seed=seed)
    return s


def _contract_input(case, seed):
    a, lmax, G = case["atoms"], case["lmax"], case["n_g"]
    L = (lmax + 1) ** 2
    rng = np.random.default_rng([seed, 23])
    # matching coefficients fall off with l, as A and B of a plane wave do
    decay = np.repeat(0.6 ** np.arange(lmax + 1), 2 * np.arange(lmax + 1) + 1)

    def rows():
        z = rng.standard_normal((a, L, G)) + 1j * rng.standard_normal((a, L, G))
        return np.asfortranarray((z * decay[None, :, None]).reshape(a * L, G))

    def herm():
        x = (rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L))) / math.sqrt(L)
        return 0.5 * (x + x.conj().T)

    A, B = rows(), rows()
    blocks = [(herm(), (rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L))) / math.sqrt(L), herm())
              for _ in range(a)]
    un = np.sqrt(rng.uniform(0.01, 1.0, (a, lmax + 1)))
    return flapw_data.DataIn(L, a, G, A, B, blocks, np.full(a, lmax, np.int32), lmax, un)


def _device_normal(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.complex(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64),
                         torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))


def _plugin_input(case, seed):
    # column-major rows x cols, as a tensor of shape (cols, rows)
    shape = (case["n"], case["k"]) if case["trans"] == "C" else (case["k"], case["n"])
    A = _device_normal(shape, 2 * seed + 1)
    B = _device_normal(shape, 2 * seed + 2) if case["op"] != "zherk" else None
    return A, B, (0.75 if case["op"] == "zherk" else 0.6 - 0.8j)


def prepare(case, seed):
    kind = case["kind"]
    ctx = _ctx()
    if kind == "pack":
        n = case["n"]
        return {"case": case, "M": _device_normal((n, n), seed),
                "out": torch.empty(n * (n + 1) // 2, dtype=torch.complex128, device="cuda")}
    if kind == "plugin":
        A, B, alpha = _plugin_input(case, seed)
        n = case["n"]
        return {"case": case, "A": A, "B": B, "alpha": alpha,
                "C": torch.zeros((n, n), dtype=torch.complex128, device="cuda")}
    if kind == "contract":
        return {"case": case, "d": _contract_input(case, seed)}
    s = _system(case, seed)
    tmats = api.prepare_tmats(s)
    if kind == "plan":
        pl = ctx.plan(s, precision=case["precision"], tmats=tmats, use_graph=case["graph"])
        return {"case": case, "plan": pl, "outs": pl.alloc_outputs()}
    outs, keep = [], []
    for kp in s.kpoints:
        pair = []
        for _ in range(2):
            t = torch.zeros((kp.n_g, kp.n_g), dtype=torch.complex128)
            t = t.pin_memory() if case["pinned"] else t
            keep.append(t)
            pair.append(t.numpy().T)
        outs.append(tuple(pair))
    return {"case": case, "sys": s, "tmats": tmats, "outs": outs, "keep": keep}


def run(state):
    case = state["case"]
    kind = case["kind"]
    ctx = _ctx()
    if kind == "plan":
        state["plan"].execute(state["outs"])
        return state["outs"]
    if kind == "host":
        res, _ = ctx.create_hs(state["sys"], precision=case["precision"], tmats=state["tmats"], out=state["outs"])
        return res
    if kind == "contract":
        H, S, _ = ctx.contract_ab(state["d"], precision=case["precision"])
        return H, S
    if kind == "plugin":
        n, k, ld = case["n"], case["k"], state["A"].shape[1]
        if case["op"] == "zherk":
            ctx.zherk(case["uplo"], case["trans"], n, k, state["alpha"], state["A"], ld, 0.0, state["C"], n,
                      precision=case["precision"])
        else:
            getattr(ctx, case["op"])(case["uplo"], case["trans"], n, k, state["alpha"], state["A"], ld, state["B"],
                                     ld, 0.0, state["C"], n, precision=case["precision"])
        return state["C"]
    return ctx.pack_lower(state["M"], out=state["out"])


def _row_sets(case):
    """Sets of matching rows that differ: types, (type, rotation) pairs, or atoms."""
    atoms, types = case["atoms"], case.get("types", case["atoms"])
    if case["kind"] == "contract" or case.get("rot") == "own":
        return atoms
    return min(atoms, 2 * types) if case.get("rot") == "classes" else types


def work(case):
    """Inputs once, outputs (lower triangles) once; operations of the products regrouped over the
    distinct row sets (S and H), of the T application and of the sums over the row sets."""
    if case["kind"] == "pack":
        n = case["n"]
        return {"bytes": 2 * 16 * n * (n + 1) // 2, "flops": 0}
    if case["kind"] == "plugin":
        n, k = case["n"], case["k"]
        two = 2 if case["op"] == "zher2k" else 1
        mats = 1 if case["op"] == "zherk" else 2
        return {"bytes": 16 * (mats * n * k + n * (n + 1) // 2), "flops": 8 * two * k * n * (n + 1) // 2}
    n, L, sets, nk = case["n_g"], (case["lmax"] + 1) ** 2, _row_sets(case), case.get("nk", 1)
    tri = n * (n + 1) // 2
    types = case.get("types", case["atoms"])
    inputs = 16 * 3 * types * L * L + 12 * n * nk
    if case["kind"] == "contract":
        inputs += 2 * 16 * L * case["atoms"] * n
    flops = nk * (2 * 8 * tri * 2 * L * sets + 8 * (2 * L) ** 2 * n * sets + 16 * tri * sets)
    return {"bytes": inputs + nk * 2 * 16 * tri, "flops": flops}


# ------------------------------------------------------- the same results in plain 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _bessel(lmax, x):
    """j_l(x) for l = 0 .. lmax + 1 (numpy, x > 0): a power series below 1/2, else Miller's
    downward recursion."""
    n = lmax + 2
    out = np.zeros((n,) + x.shape)
    small = x < 0.5
    xs = np.where(small, x, 0.1)
    dfact = 1.0
    for l in range(n):
        dfact *= 2 * l + 1
        term = np.ones_like(xs)
        tot = np.ones_like(xs)
        for k in range(1, 12):
            term = term * (-0.5 * xs * xs) / (k * (2 * l + 2 * k + 1))
            tot += term
        out[l] = xs ** l / dfact * tot
    xb = np.where(small, 1.0, x)
    hi, cur = np.zeros_like(xb), np.full_like(xb, 1e-150)
    down = np.zeros((n,) + x.shape)
    for l in range(int(x.max()) + 45, -1, -1):
        if l < n:
            down[l] = cur
        hi, cur = cur, (2 * l + 1) / xb * cur - hi
    j0, j1 = np.sin(xb) / xb, np.sin(xb) / xb ** 2 - np.cos(xb) / xb
    q = np.where(np.abs(j0) > np.abs(j1), j0 / down[0], j1 / down[1])
    return np.where(small[None], out, down * q[None])


def _harmonics(lmax, v):
    """Y_lm of unit vectors v (n, 3), Condon-Shortley phase, as (L, n) complex."""
    n = v.shape[0]
    cth = v[:, 2]
    rho = np.sqrt(v[:, 0] ** 2 + v[:, 1] ** 2)
    e = np.where(rho > 1e-13, (v[:, 0] + 1j * v[:, 1]) / np.where(rho > 1e-13, rho, 1.0), 1.0)
    Y = np.zeros(((lmax + 1) ** 2, n), complex)
    pmm = np.full(n, math.sqrt(1.0 / (4.0 * math.pi)))
    for m in range(lmax + 1):
        if m > 0:
            pmm = -math.sqrt((2 * m + 1) / (2.0 * m)) * rho * pmm
        a, b = np.zeros(n), pmm
        for l in range(m, lmax + 1):
            if l > m:
                f = math.sqrt((4.0 * l * l - 1) / (l * l - m * m))
                g = math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1)) if l - 1 > m else 0.0
                a, b = b, f * (cth * b - g * a)
            Y[l * (l + 1) + m] = b * e ** m
            Y[l * (l + 1) - m] = (-1) ** m * np.conj(Y[l * (l + 1) + m])
    return Y


def _rows(s, kp, t, rot):
    """[A; B] of type t with rotation matrix rot, without the structure phase: (2L, n) complex."""
    lmax = s.max_lmax
    K = kp.k[None, :] + kp.g
    kn = np.sqrt(((K @ s.bmat.T) ** 2).sum(axis=1))
    d = K @ rot
    d /= np.sqrt((d ** 2).sum(axis=1))[:, None]
    x = s.type_rmt[t] * kn
    j = _bessel(lmax, x)
    Yc = np.conj(_harmonics(lmax, d)) * (4 * math.pi / math.sqrt(s.vol_cell))
    A, B = np.zeros_like(Yc), np.zeros_like(Yc)
    for l in range(lmax + 1):
        dj = -j[1] if l == 0 else j[l - 1] - (l + 1) / x * j[l]
        u, ud, v, vd = s.u[t, l], s.u_dr[t, l], s.dE_u[t, l], s.dE_u_dr[t, l]
        w = 1.0 / (v * ud - u * vd)
        q = slice(l * l, (l + 1) ** 2)
        A[q] = Yc[q] * (w * (v * kn * dj - vd * j[l]))
        B[q] = Yc[q] * (w * (-u * kn * dj + ud * j[l]))
    return np.concatenate([A, B])


def _full_t(s, t):
    """The type's Hermitian 2L x 2L block with the energy and normalisation terms."""
    L = s.L
    ls = np.repeat(np.arange(s.max_lmax + 1), 2 * np.arange(s.max_lmax + 1) + 1)
    low = np.tril(np.ones((L, L), bool))

    def herm(x):
        return np.where(low, x, np.conj(x.T))

    aa = herm(s.taa_raw[t]) + np.diag(s.energies[t][ls])
    bb = herm(s.tbb_raw[t]) + np.diag((s.energies[t] * s.dE_u_norm[t])[ls])
    ab = s.tab_raw[t] + 0.5 * np.eye(L)
    return np.block([[aa, ab], [ab.conj().T, bb]]), np.concatenate([np.ones(L), s.dE_u_norm[t][ls]])


def _exact_hs(s, kp):
    dev, n = _dev(), kp.g.shape[0]
    K = kp.k[None, :] + kp.g
    H = torch.zeros((n, n), dtype=torch.complex128, device=dev)
    S = torch.zeros_like(H)
    sets = {}
    for a in range(s.num_atoms):
        R = s.bmat if s.atom_rotmat is None else s.atom_rotmat[a]
        sets.setdefault((int(s.atom_type[a]), R.tobytes()), (R, []))[1].append(a)
    for (t, _), (R, atoms) in sets.items():
        M = torch.from_numpy(_rows(s, kp, t, R)).to(dev)
        T, w = (torch.from_numpy(x).to(dev) for x in _full_t(s, t))
        ph = torch.from_numpy(np.exp(2j * math.pi * (s.atom_pos[atoms] @ K.T))).to(dev)
        sf = ph.conj().T @ ph
        Mh = M.conj().T.contiguous()
        S += sf * (Mh @ (w[:, None] * M))
        H += sf * (Mh @ (T @ M))
        del sf
    return H, S


def exact(case, seed):
    kind = case["kind"]
    if kind == "pack":
        n = case["n"]
        M = _device_normal((n, n), seed)
        r, c = torch.tril_indices(n, n, device=M.device)
        return M[c, r]
    if kind == "plugin":
        A, B, alpha = _plugin_input(case, seed)
        # op(X)^H as (n, k) rows: stored columns for 'C', stored rows (conjugated) for 'N'
        XA = A.conj() if case["trans"] == "C" else A.T
        XB = XA if B is None else B.conj() if case["trans"] == "C" else B.T
        P = alpha * (XA @ XB.conj().T)
        if case["op"] == "zher2k":
            P = P + P.conj().T
        P = torch.tril(P) if case["uplo"] == "L" else torch.triu(P)
        if case["op"] != "zherkx":
            P = P - 1j * torch.diag(torch.diagonal(P).imag)
        return P.T.contiguous()
    if kind == "contract":
        d = _contract_input(case, seed)
        dev, L, un2 = _dev(), d.L, d.sqrt_u_norms ** 2
        ls = np.repeat(np.arange(d.max_lmax + 1), 2 * np.arange(d.max_lmax + 1) + 1)
        H = torch.zeros((d.G, d.G), dtype=torch.complex128, device=dev)
        S = torch.zeros_like(H)
        for j in range(d.a):
            C = torch.from_numpy(np.concatenate([d.A[j * L:(j + 1) * L], d.B[j * L:(j + 1) * L]])).to(dev)
            aa, ab, bb = d.blocks[j]
            T = torch.from_numpy(np.block([[aa, ab], [ab.conj().T, bb]])).to(dev)
            w = torch.from_numpy(np.concatenate([np.ones(L), un2[j][ls]])).to(dev)
            S += C.conj().T @ (w[:, None] * C)
            H += C.conj().T @ (T @ C)
        return torch.tril(H), torch.tril(S)
    s = _system(case, seed)
    out = []
    for kp in s.kpoints:
        H, S = _exact_hs(s, kp)
        H, S = torch.tril(H), torch.tril(S)
        # device outputs are column-major tensors (tensor[col, row]); host outputs Fortran arrays
        out.append((H.T.contiguous(), S.T.contiguous()) if kind == "plan" else (H.cpu().numpy(), S.cpu().numpy()))
    return out
