"""Performance cases of the library: the calls a host program makes, over the
range of systems it makes them for.

A host program builds a Context per structure, prepares the operators once
(OLCAOsetup), then iterates: potential coefficients in, eigenvalues out, and
from the eigenvectors the density matrix and its traces.  After convergence
it runs band paths.  The cases follow that: set-up passes, SCF iterations in
both forms and precisions, the density step, a band path, and the single
layers a host calls with arrays of its own (assembly and solve of packed
operators, products).

Structures are the repository's own kinds (silicon diamond supercells,
two-atom carbon and silicon cells, graphite, a two-atom oxide with f
functions); the basis is fixed per kind, the geometry's displacements, the
potential coefficients and the other inputs come from the seed.

A case is a dict:
  call    setup | scf | mixed | fused | density | band | secular | product
  kind    structure: c2, si2, graphite, sif, si (diamond supercell)
  rx, ry, rz   repetitions of the conventional silicon cell (kind si)
  kx, ky, kz   Monkhorst-Pack mesh (shifted by half a step)
  core    0: valence functions only (kind si)
  rel     1: with the mass-velocity term
and per call: states, spin, electrons, points, m, n, k.

The mixed-precision calls ask for eigenvalues alone: their eigenvectors carry
FP32-grade components, an arbitrary phase and arbitrary mixing inside nearly
degenerate levels, so two correct solvers differ in every element.  The step
with vectors is measured in FP64 through the density matrix, which has
neither freedom.
"""

import math

import numpy as np
import torch

from olcao_gb300 import api
from olcao_gb300 import band
from olcao_gb300 import system as S


# ---------------------------------------------------------------------------
# structures
# ---------------------------------------------------------------------------
SI8 = ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0),
       (.25, .25, .25), (.25, .75, .75), (.75, .25, .75), (.75, .75, .25))


def _structure(case):
    """(cell vectors as columns, positions, types, site types, potentials,
    potential type of each atom type), before displacement."""
    kind = case["kind"]
    basis = np.random.default_rng(6)
    if kind in ("c2", "si2"):
        a = (3.567 if kind == "c2" else 5.431) * S.ANGSTROM
        vec = 0.5 * a * np.array([[0, 1, 1], [1, 0, 1], [1, 1, 0]], float)
        pos = np.array([[0.0, 0, 0], [0.25 * a] * 3])
        if kind == "c2":
            return vec, pos, [S.carbon_type(basis)], [0, 0], [S.carbon_pot()], [0]
        return vec, pos, [S.silicon_type(basis)], [0, 0], [S.silicon_pot()], [0]
    if kind == "graphite":
        a, c = 2.46 * S.ANGSTROM, 6.71 * S.ANGSTROM
        vec = np.array([[a, 0, 0], [-0.5 * a, 0.5 * math.sqrt(3) * a, 0], [0, 0, c]]).T
        frac = np.array([[0, 0, .25], [0, 0, .75], [1 / 3, 2 / 3, .25], [2 / 3, 1 / 3, .75]])
        return (vec, frac @ vec.T, [S.carbon_type(basis, vale_l=(0, 1, 0, 1), core_l=())], [0] * 4,
                [S.carbon_pot()], [0])
    if kind == "sif":
        a = 4.2 * S.ANGSTROM
        vec = np.array([[a, 0, 0], [0.1 * a, a, 0], [0.2 * a, 0.1 * a, 1.05 * a]]).T
        pos = np.array([[0.1, 0.2, 0.3], [1.4, 1.3, 1.8]]) * S.ANGSTROM
        t1 = S.make_type(basis, 1, 18, 0.12, 1.0e6, (18, 18, 12, 8), (0, 1, 2, 3, 0, 1), (0, 0, 1, 3))
        t2 = S.make_type(basis, 2, 18, 0.12, 1.0e6, (18, 18, 12, 0), (0, 1, 0, 1, 2), (0,))
        pots = [S.silicon_pot(1), S.PotSpec(2, 8.0, 20.0, S.even_tempered(16, 0.1, 1.0e6))]
        return vec, pos, [t1, t2], [0, 1], pots, [0, 1]
    a = 5.431 * S.ANGSTROM
    reps = (case["rx"], case["ry"], case["rz"])
    pos = np.array([[i + f[0], j + f[1], k + f[2]] for i in range(reps[0]) for j in range(reps[1])
                    for k in range(reps[2]) for f in SI8]) * a
    return (a * np.diag(np.array(reps, float)), pos, [S.silicon_type(basis, core=bool(case.get("core", 1)))],
            [0] * len(pos), [S.silicon_pot()], [0])


def _system(case, seed):
    """The structure with this seed's displacements (sigma 0.02 A) and
    potential coefficients (2 % around the kind's own)."""
    vec, pos, types, site, pots, pot_of = _structure(case)
    rng = np.random.default_rng([int(seed), 17])
    pos = pos + rng.normal(0.0, 0.02 * S.ANGSTROM, pos.shape)
    npot = sum(len(p.alphas) for p in pots)
    base = 0.1 * np.random.default_rng(60).standard_normal(npot)
    coeffs = base * (1.0 + 0.02 * rng.standard_normal(npot))
    site = np.array(site, np.int32)
    ptype = np.array([pot_of[t] for t in site], np.int32)
    order = np.argsort(ptype, kind="stable")
    mesh = S.mp_mesh((case.get("kx", 1), case.get("ky", 1), case.get("kz", 1)), (0.5, 0.5, 0.5))
    return S.System(name=case["kind"], real_vectors=vec, types=types, site_type=site, site_pos=pos, pots=pots,
                    pot_site_type=ptype[order], pot_site_pos=pos[order], kpoints_abc=mesh, pot_coeffs=coeffs,
                    seed=int(seed), rel=int(case.get("rel", 0)))


def _dims(case):
    """(basis functions n, core functions, potential terms, k-points)."""
    vec, pos, types, site, pots, _ = _structure(case)
    n = sum(types[t].num_vale_states for t in site)
    nc = sum(types[t].num_core_states for t in site)
    return n, nc, sum(len(p.alphas) for p in pots), case.get("kx", 1) * case.get("ky", 1) * case.get("kz", 1)


def _states(case):
    """Eigenvalues asked for: all, or the doubly occupied ones of silicon's
    four valence electrons per atom."""
    n = _dims(case)[0]
    return n if case.get("states", "all") == "all" else 16 * case["rx"] * case["ry"] * case["rz"]


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    si = {"kind": "si", "rx": 1, "ry": 1, "rz": 1}
    si64 = {"kind": "si", "rx": 2, "ry": 2, "rz": 2}
    return [
        # one whole SCF step of the smallest cell: iteration with vectors, occupations, density matrix
        # and traces; latency and launches
        {"name": "scf_diamond_216k", "call": "scf", "kind": "c2", "kx": 6, "ky": 6, "kz": 6, "electrons": 8.0},
        # the same for a layered cell on a dense mesh: thousands of small pencils
        {"name": "scf_graphite_8192k", "call": "scf", "kind": "graphite", "kx": 32, "ky": 32, "kz": 8,
         "electrons": 16.0},
        # mixed-precision iterations on resident operators (graph replay): the conventional cell on a dense
        # mesh, valence only; the 64-atom supercell; the 216-atom supercell
        dict(si, name="mixed_si8_512k", call="mixed", core=0, kx=8, ky=8, kz=8, states="all"),
        dict(si64, name="mixed_si64_64k", call="mixed", kx=4, ky=4, kz=4, states="occupied"),
        {"name": "mixed_si216_8k", "call": "mixed", "kind": "si", "rx": 3, "ry": 3, "rz": 3, "kx": 2, "ky": 2,
         "kz": 2, "states": "occupied"},
        # an iteration that recomputes the potential integrals instead of keeping every term resident
        dict(si64, name="fused_si64_8k", call="fused", kx=2, ky=2, kz=2, states="occupied"),
        # OLCAOsetup: every stored operator of a small two-type cell with f functions and the relativistic
        # term, and of the 64-atom supercell
        {"name": "setup_oxide_f_8k", "call": "setup", "kind": "sif", "kx": 2, "ky": 2, "kz": 2, "rel": 1},
        dict(si64, name="setup_si64_8k", call="setup", kx=2, ky=2, kz=2),
        # a converged potential's band path, the whole call
        {"name": "band_si2_61", "call": "band", "kind": "si2", "points": 61},
        # density matrix and operator traces of given vectors, both spin channels
        dict(si64, name="density_si64_27k", call="density", kx=3, ky=3, kz=3, spin=2),
        # assembly and FP64 solve of packed operators that the host holds
        {"name": "secular_si2_343k", "call": "secular", "kind": "si2", "kx": 7, "ky": 7, "kz": 7},
        # the two tensor-core products on matrices of the host's own
        {"name": "product_1248", "call": "product", "m": 1248, "n": 1248, "k": 1248},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, most):
    """A mesh with at most `most` points, spread over the logarithm."""
    nk = _log(rng, 1, most)
    kx = max(1, _log(rng, 1, max(1, round(nk ** 0.6))))
    ky = max(1, _log(rng, 1, max(1, nk // kx)))
    return {"kx": kx, "ky": ky, "kz": max(1, nk // (kx * ky))}


def _cells(rng, most):
    while True:
        r = sorted(rng.randint(1, 3) for _ in range(3))
        rng.shuffle(r)
        if r[0] * r[1] * r[2] <= most:
            return {"kind": "si", "rx": r[0], "ry": r[1], "rz": r[2]}


def draw(rng):
    call = rng.choice(["scf", "mixed", "mixed", "mixed", "fused", "setup", "setup", "band", "density", "secular",
                       "product"])
    if call == "scf":
        kind = rng.choice(["c2", "si2", "graphite"])
        return dict({"call": call, "kind": kind, "electrons": 16.0 if kind == "graphite" else 8.0},
                    **_mesh(rng, 4096))
    if call == "mixed":
        c = _cells(rng, 27)
        n = 104 * c["rx"] * c["ry"] * c["rz"]
        most = min(512, max(1, int(8 * (2808 / n) ** 3)))
        core = rng.choice([0, 1]) if n == 104 else 1
        return dict(c, call=call, core=core, states="all" if n <= 208 else "occupied", **_mesh(rng, most))
    if call == "fused":
        c = _cells(rng, 8)
        return dict(c, call=call, states="occupied", **_mesh(rng, max(1, 64 // (c["rx"] * c["ry"] * c["rz"]))))
    if call == "setup":
        kind = rng.choice(["c2", "si2", "graphite", "sif", "si", "si"])
        if kind != "si":
            return dict({"call": call, "kind": kind, "rel": rng.choice([0, 0, 1])}, **_mesh(rng, 64))
        c = _cells(rng, 8)
        return dict(c, call=call, **_mesh(rng, max(1, 64 // (c["rx"] * c["ry"] * c["rz"]))))
    if call == "band":
        return {"call": call, "kind": rng.choice(["c2", "si2", "graphite"]), "points": _log(rng, 10, 200)}
    if call == "density":
        c = _cells(rng, 8)
        return dict(c, call=call, spin=rng.choice([1, 2]),
                    **_mesh(rng, max(1, 216 // (c["rx"] * c["ry"] * c["rz"]))))
    if call == "secular":
        kind = rng.choice(["c2", "si2", "graphite", "si"])
        c = {"kind": "si", "rx": 1, "ry": 1, "rz": 1} if kind == "si" else {"kind": kind}
        return dict(c, call=call, **_mesh(rng, 64 if kind == "si" else 1024))
    return {"call": call, "m": _log(rng, 48, 2000), "n": _log(rng, 48, 2000), "k": _log(rng, 48, 2000)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rand_c(seed, *shape, dtype=torch.complex128):
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    return torch.randn(*shape, dtype=dtype, device="cuda", generator=g)


def _density_inputs(case, seed):
    """Occupied-state vectors with norms near 1 and occupations x k weight,
    some of the highest states partly filled or empty."""
    n, _, _, nk = _dims(case)
    spin, ns = case["spin"], 16 * case["rx"] * case["ry"] * case["rz"]
    vec = _rand_c(seed, spin, nk, ns, n) / math.sqrt(n)
    rng = np.random.default_rng([int(seed), 23])
    occ = np.full((spin, nk, ns), 2.0 / (nk * spin))
    occ[:, :, ns - ns // 8:] *= rng.uniform(0.0, 1.0, (spin, nk, ns // 8))
    occ[:, :, ns - 1] = 0.0
    eig = np.sort(rng.uniform(-1.0, 0.5, (spin, nk, ns)), axis=2)
    return vec, occ, eig


def _secular_inputs(case, seed):
    """Packed Hermitian operators as a host holds them: a well-conditioned
    overlap near the identity, a kinetic-like and a nuclear-like term and
    smaller potential terms, [nk, plen, 2]."""
    n, _, pd, nk = _dims(case)
    plen = n * (n + 1) // 2
    col = torch.arange(n, device="cuda").repeat_interleave(torch.arange(1, n + 1, device="cuda"))
    row = torch.arange(plen, device="cuda") - col * (col + 1) // 2
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 104729 + 5)
    fall = torch.exp(-0.05 * (col - row).double())[None, :, None]
    diag = (row == col)

    def op(scale, centre):
        x = scale / math.sqrt(n) * fall * torch.randn(nk, plen, 2, dtype=torch.float64, device="cuda", generator=g)
        x[:, diag, 1] = 0.0
        x[:, diag, 0] += centre
        return x

    level = torch.linspace(0.2, 3.0, n, dtype=torch.float64, device="cuda")
    packed = {"S": op(0.15, 1.0), "KE": op(0.3, level), "NP": op(0.3, -1.0)}
    for j in range(pd):
        packed["V%d" % j] = op(0.2, 0.3 / (j + 1))
    rng = np.random.default_rng([int(seed), 29])
    return packed, 0.1 * rng.standard_normal(pd)


def _product_inputs(case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    return (_rand_c(seed, m, k), _rand_c(seed + 1, k, n), _rand_c(seed + 2, k, m, dtype=torch.complex64),
            _rand_c(seed + 3, k, n, dtype=torch.complex64))


# high-symmetry points of the face-centred and of the hexagonal cell (fractional)
_FCC = [[0.5, 0.5, 0.5], [0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.25, 0.625, 0.625], [0.375, 0.75, 0.375],
        [0.0, 0.0, 0.0]]
_HEX = [[0.0, 0.0, 0.0], [0.5, 0.0, 0.0], [1 / 3, 1 / 3, 0.0], [0.0, 0.0, 0.0], [0.0, 0.0, 0.5]]


def prepare(case, seed):
    call = case["call"]
    if call == "product":
        ctx = api.Context(_system({"kind": "c2"}, seed))
        return {"call": call, "ctx": ctx, "ops": _product_inputs(case, seed)}
    sysm = _system(case, seed)
    if call == "band":
        return {"call": call, "system": sysm, "points": case["points"],
                "path": [np.array(_HEX if case["kind"] == "graphite" else _FCC)]}
    ctx = api.Context(sysm)
    state = {"call": call, "ctx": ctx, "system": sysm}
    if call == "scf":
        ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
        state["electrons"] = case["electrons"]
        state["vectors"] = torch.zeros(ctx.nk, ctx.vale_dim, ctx.vale_dim, dtype=torch.complex128, device="cuda")
    elif call == "mixed":
        ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
        state["states"] = _states(case)
    elif call == "fused":
        ctx.scf_prepare(api.PREC_MIXED, api.FORM_FUSED)
        state["states"] = _states(case)
    elif call == "density":
        ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
        state["vectors"], state["occ"], state["eig"] = _density_inputs(case, seed)
    elif call == "secular":
        state["packed"], state["coeffs"] = _secular_inputs(case, seed)
    return state


def run(state):
    call = state["call"]
    if call == "setup":
        return state["ctx"].packed_operators()
    if call == "scf":
        ctx, sysm = state["ctx"], state["system"]
        eig = ctx.scf_iteration(sysm.pot_coeffs, ctx.vale_dim, precision=api.PREC_FP64, vectors=state["vectors"])
        occ, fermi = api.populate_states(eig, sysm.kpoint_weights(), state["electrons"], thermal_sigma=0.01)
        traces, energy, rho = ctx.make_valence_rho(occ, state["vectors"], eig, rho=True)
        return eig, occ, fermi, traces, energy, rho
    if call == "mixed":
        return state["ctx"].scf_iteration(state["system"].pot_coeffs, state["states"], precision=api.PREC_MIXED,
                                          graph=True)
    if call == "fused":
        return state["ctx"].scf_iteration(state["system"].pot_coeffs, state["states"], precision=api.PREC_MIXED)
    if call == "band":
        return band.band_structure(state["system"], state["path"], state["points"])
    if call == "density":
        return state["ctx"].make_valence_rho(state["occ"], state["vectors"], state["eig"], rho=True)
    if call == "secular":
        ctx = state["ctx"]
        h = ctx.assemble_hamiltonian(state["packed"], state["coeffs"])
        eig, _, info = ctx.solve_zhegv(h, state["packed"]["S"], ctx.vale_dim)
        return h, eig, info
    a, b, a32, b32 = state["ops"]
    return state["ctx"].split_zgemm(a, b), state["ctx"].split_cgemm32(a32, b32, conj_a=True)


# ---------------------------------------------------------------------------
# work of one pass, and 64-bit results
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: each input and each output once.  Flops: the complex products
    and solves of the mathematical statement, 8 per complex multiply-add
    (solve with vectors 23 n^3 complex-real flops); the integrals' own
    arithmetic depends on the screening and is left out."""
    call = case["call"]
    if call == "product":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 24.0 * (m * k + k * n + m * n), "flops": 16.0 * m * n * k}
    n, nc, pd, nk = _dims(case)
    if call == "band":
        nk = case["points"]
    rel = case.get("rel", 0)
    plen = n * (n + 1) // 2
    ortho = 8.0 * nk * (2.0 * nc * n * n + 1.0 * nc * nc * n)
    solve = 23.0 * nk * float(n) ** 3
    if call == "setup":
        nop = 3 + rel + pd
        return {"bytes": 16.0 * nk * plen * nop, "flops": nop * ortho}
    if call in ("mixed", "scf"):
        by, fl = 16.0 * nk * plen * (3 + pd) + 8.0 * nk * _states(case), solve
        if call == "scf":
            by += 16.0 * nk * (plen * (4 + pd) + 2.0 * n * n)
            fl += 8.0 * nk * n * n * min(n, case["electrons"])
        return {"bytes": by, "flops": fl}
    if call == "fused":
        return {"bytes": 16.0 * nk * (2.0 * n * n + 2.0 * nc * n) + 8.0 * nk * _states(case), "flops": ortho + solve}
    if call == "band":
        return {"bytes": 8.0 * nk * n, "flops": 3 * ortho + solve}
    if call == "density":
        ns = 16 * case["rx"] * case["ry"] * case["rz"]
        s = case["spin"]
        return {"bytes": 16.0 * nk * (plen * (3 + pd) + s * (ns * n + plen)),
                "flops": s * nk * (4.0 * n * n * ns + 4.0 * plen * (3 + pd))}
    return {"bytes": 16.0 * nk * plen * (5 + pd) + 8.0 * nk * n, "flops": solve}


def _unpack(p, n):
    """Packed [nk, plen, 2] -> full Hermitian [nk, n, n]."""
    col = torch.arange(n, device="cuda").repeat_interleave(torch.arange(1, n + 1, device="cuda"))
    row = torch.arange(n * (n + 1) // 2, device="cuda") - col * (col + 1) // 2
    z = torch.view_as_complex(p)
    full = torch.zeros(p.shape[0], n, n, dtype=torch.complex128, device="cuda")
    full[:, col, row] = z.conj()
    full[:, row, col] = z
    return full


def exact(case, seed):
    call = case["call"]
    if call == "product":
        a, b, a32, b32 = _product_inputs(case, seed)
        return a @ b, a32.to(torch.complex128).conj().t() @ b32.to(torch.complex128)
    if call == "density":
        vec, occ, eig = _density_inputs(case, seed)
        n = _dims(case)[0]
        f = torch.from_numpy(occ).cuda()
        rho = torch.einsum("skj,skja,skjb->skab", f.to(torch.complex128), vec, vec.conj())
        if case["spin"] == 2:
            rho = torch.stack([rho[0] + rho[1], rho[0] - rho[1]])
        col = torch.arange(n, device="cuda").repeat_interleave(torch.arange(1, n + 1, device="cuda"))
        row = torch.arange(n * (n + 1) // 2, device="cuda") - col * (col + 1) // 2
        return None, (occ * eig).sum(axis=(1, 2)), torch.view_as_real(rho[:, :, row, col].contiguous())
    if call == "secular":
        packed, co = _secular_inputs(case, seed)
        n = _dims(case)[0]
        h = packed["NP"] + packed["KE"]
        for j, c in enumerate(co):
            h = h + c * packed["V%d" % j]
        inv = torch.linalg.inv(torch.linalg.cholesky(_unpack(packed["S"], n)))
        red = inv @ _unpack(h, n) @ inv.mH
        return h, torch.from_numpy(np.linalg.eigvalsh(red.cpu().numpy())), None
    return None
