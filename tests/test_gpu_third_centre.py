"""The third-centre kernels' image lists and moment transformation (gpu).

Nuclear and electronic-potential blocks against the oracle where the lists,
the screen and the transformation can go wrong: a flat and a strongly skewed
cell (many lattice planes within the radius in one direction), potential
sites far outside the home cell, two types of one element with different
exponents (the screen's centre is then not the pair's centre), two potential
types, and every class pair s..f.  Bar: the integrals' 1e-10 of the block's
largest magnitude.  The mixed-precision sum (far images in FP32) is held to
the FP64 one at 1e-10 of it: an FP32 rounding (6e-8) of terms suppressed
below exp(-22) = 3e-10.
"""

import numpy as np
import pytest

import oracle as orc
from olcao_gb300 import system as S

RTOL = 1e-10


def _sites(vec, pos, types, site, pots, ptype, mesh=(2, 1, 1), seed=3, shift=None):
    rng = np.random.default_rng(seed)
    ptype = np.asarray(ptype, np.int32)
    order = np.argsort(ptype, kind="stable")
    ppos = pos if shift is None else pos + shift
    return S.System(name="t", real_vectors=vec, types=types, site_type=np.asarray(site, np.int32), site_pos=pos,
                    pots=pots, pot_site_type=ptype[order], pot_site_pos=ppos[order],
                    kpoints_abc=S.mp_mesh(mesh, (0.5, 0.5, 0.5)),
                    pot_coeffs=0.1 * rng.standard_normal(sum(len(p.alphas) for p in pots)), seed=seed)


def _type(rng, element, amin, orb=(8, 8, 5, 0), vale=(0, 1, 2), core=(0,)):
    return S.make_type(rng, element, 8, amin, 2.0e3, orb, vale, core)


def _flat():
    rng = np.random.default_rng(5)
    vec = np.array([[3.0, 0, 0], [0, 11.0, 0], [0, 0, 7.0]])
    pos = np.array([[0.1, 0.2, 0.3], [1.4, 5.1, 3.9]])
    return _sites(vec, pos, [_type(rng, 1, 0.4)], [0, 0], [S.PotSpec(1, 6.0, 20.0, S.even_tempered(4, 0.3, 1e3))],
                  [0, 0])


def _skew():
    rng = np.random.default_rng(6)
    vec = np.array([[5.0, 0, 0], [4.5, 5.5, 0], [-4.0, 4.8, 6.0]]).T
    pos = np.array([[0.1, 0.2, 0.3], [2.0, 3.1, 2.2], [9.0, -7.0, 4.0]])
    shift = vec @ np.array([[3.0, -2.0, 4.0]]).T        # whole lattice vectors
    return _sites(vec, pos, [_type(rng, 1, 0.4)], [0, 0, 0],
                  [S.PotSpec(1, 6.0, 20.0, S.even_tempered(4, 0.3, 1e3))], [0, 0, 0], shift=shift.T)


def _one_element():
    rng = np.random.default_rng(7)
    vec = np.diag([6.5, 7.0, 6.0])
    pos = np.array([[0.1, 0.2, 0.3], [3.0, 3.1, 2.9]])
    return _sites(vec, pos, [_type(rng, 1, 0.4), _type(rng, 1, 0.55)], [0, 1],
                  [S.PotSpec(1, 6.0, 20.0, S.even_tempered(4, 0.3, 1e3)),
                   S.PotSpec(2, 8.0, 15.0, S.even_tempered(3, 0.5, 1e2))], [0, 1])


def _f_types():
    rng = np.random.default_rng(8)
    vec = np.diag([7.5, 7.0, 8.0])
    pos = np.array([[0.1, 0.2, 0.3], [3.2, 3.6, 3.1]])
    return _sites(vec, pos, [_type(rng, 1, 0.5, (8, 8, 5, 3), (0, 1, 2, 3), (0, 3)), _type(rng, 2, 0.5)], [0, 1],
                  [S.PotSpec(1, 6.0, 20.0, S.even_tempered(4, 0.4, 1e3)),
                   S.PotSpec(2, 8.0, 20.0, S.even_tempered(2, 0.4, 1e2))], [0, 1])


SYSTEMS = {"flat": _flat, "skew": _skew, "one_element": _one_element, "f_types": _f_types}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_third_centre_blocks(gpu_lib, name):
    from olcao_gb300 import api
    sysm = SYSTEMS[name]()
    o, ctx = orc.Oracle(sysm), api.Context(sysm)
    runs = [(api.OP_NUCLEAR, 0)] + [(api.OP_ELECPOT, j) for j in range(ctx.pot_dim)]
    total = None
    for op, term in runs:
        got = [b.cpu().numpy() for b in ctx.gauss_overlap(op, term)]
        ref = o.operator(op, term)
        for g, r, what in zip(got, ref, ("vv", "cv", "cc")):
            scale = np.abs(r).max()
            assert np.abs(g - r).max() <= RTOL * scale + 1e-14, f"{name} op {op} term {term} {what}"
        if op == api.OP_ELECPOT:
            part = [sysm.pot_coeffs[term] * r for r in ref]
            total = part if total is None else [x + y for x, y in zip(total, part)]
    # all terms in one pass, FP64 and with the far images in FP32
    fixed = [o.operator(op) for op in (api.OP_KINETIC, api.OP_NUCLEAR)]
    want = [t + a + b for t, a, b in zip(total, *fixed)]
    for prec in (api.PREC_FP64, api.PREC_MIXED):
        got = ctx.gauss_overlap(api.OP_HAMILTONIAN, 0, sysm.pot_coeffs, precision=prec)
        for g, r, what in zip(got, want, ("vv", "cv", "cc")):
            scale = np.abs(r).max()
            assert np.abs(g.cpu().numpy() - r).max() <= RTOL * scale + 1e-14, f"{name} H precision {prec} {what}"
    ctx.close()
