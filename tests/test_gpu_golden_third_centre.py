"""The kernels that sum third-centre primitives over lattice images (gpu) against
the blocks of tests/golden/primitives.npz: two atoms of one exponent each and one
potential site in a cell so large that the image in the home cell is the only one
whose contribution is not zero to rounding, so that a block of the operator is one
primitive.  Every class pair s..f, as one term and as a sum over terms; bars of
tests/test_gpu_primitives.py.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S

# angular normalisation of the harmonics (l m), in the order of the states
NORM = np.array([0.2820947917738782] + 3 * [0.4886025119029199] + 3 * [1.0925484305920790] +
                [0.5462742152960396, 0.3153915652525200, 2.8906114426405543, 1.4453057213202771] +
                2 * [0.5900435899266435] + [0.3731763325901154] + 2 * [0.4570457994644657])
CLASS = {1: 0, 4: 1, 9: 2, 16: 3}


def _block(api, kind, p, lm):
    a1, a2, a3 = p[:3]
    types = []
    for q, a in ((0, a1), (1, a2)):
        l = CLASS[int(lm[q])]
        types.append(S.TypeSpec(element=q + 1, alphas=np.array([a]), num_orb_alphas=tuple([1] * (l + 1) + [0] * (3 - l)),
                                vale_l=list(range(l + 1)), core_l=[], vale_coeff=np.ones((l + 1, 1)),
                                core_coeff=np.zeros((0, 1))))
    pos = np.array([p[3:6], p[6:9]])
    # pairs and images one cell away are suppressed below exp(-800)
    rho = (a1 + a2) * a3 / (a1 + a2 + a3)
    size = 4.0 * np.abs(p[3:12]).max() + np.sqrt(800.0 / min(rho, a1 * a2 / (a1 + a2)))
    sysm = S.System(name="g", real_vectors=size * np.eye(3), types=types, site_type=np.array([0, 1], np.int32),
                    site_pos=pos, pots=[S.PotSpec(3, 1.0, a3, np.array([a3]))], pot_site_type=np.zeros(1, np.int32),
                    pot_site_pos=p[None, 9:12].copy(), kpoints_abc=np.zeros((1, 3)), pot_coeffs=np.ones(1), thresh=1e-300)
    ctx = api.Context(sysm)
    n1, n2 = int(lm[0]), int(lm[1])
    out = []
    if kind == 3:
        out.append(-ctx.gauss_overlap(api.OP_NUCLEAR)[0].cpu().numpy())
    else:
        out.append(ctx.gauss_overlap(api.OP_ELECPOT, 0)[0].cpu().numpy())
        # the sum over terms: a coefficient beside which the fixed operators vanish
        out.append(ctx.gauss_overlap(api.OP_HAMILTONIAN, 0, np.array([2.0 ** 900]))[0].cpu().numpy() * 2.0 ** -900)
    ctx.close()
    return [o[0, n1:n1 + n2, :n1].real.T / (NORM[:n1, None] * NORM[None, :n2]) for o in out]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [3, 4])
def test_golden_blocks(gpu_lib, golden, kind):
    from olcao_gb300 import api
    sel = golden["kind"] == kind
    tol = 1e-9 if kind == 3 else 1e-12
    for i, (p, lm, ref) in enumerate(zip(golden["params"][sel], golden["lmalpha"][sel], golden["sh"][sel])):
        r = ref[:lm[0], :lm[1]]
        for got in _block(api, kind, p, lm):
            err = np.abs(got - r).max() / max(np.abs(r).max(), 1e-280)
            assert err <= tol, f"kind {kind} item {i} lm {lm}: rel err {err:.2e}"
