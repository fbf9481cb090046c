"""Third-centre items shared by up to 32 lanes (gpu): the blocks at a k-point do
not depend on how many items the system has.  A cell with one atom gives
classes of a few items (32 lanes each), its supercells of 2, 4 and 12 cells
give items that 16 lanes down to one share; the supercell's Gamma block folds the
cell's k-points, so the trace of its potential and nuclear blocks equals the
sum of the cell's over the folded k-points.  Bar: 1e-10 of that sum, the
integrals' own."""

import numpy as np
import pytest

from olcao_gb300 import system as S


def _cell(reps, kpoints):
    rng = np.random.default_rng(8)
    t = S.make_type(rng, 1, 6, 0.35, 2.0e3, (6, 6, 4, 0), (0, 1, 2), (0,))
    a = np.diag([6.0, 6.5, 7.0])
    pos = np.array([[0.3 + 6.0 * i, 0.2, 0.1] for i in range(reps)])
    n = len(pos)
    return S.System(name="t", real_vectors=a @ np.diag([float(reps), 1, 1]), types=[t], site_type=np.zeros(n, np.int32),
                    site_pos=pos, pots=[S.PotSpec(1, 6.0, 20.0, S.even_tempered(3, 0.3, 1e3))],
                    pot_site_type=np.zeros(n, np.int32), pot_site_pos=pos, kpoints_abc=np.asarray(kpoints, float),
                    pot_coeffs=np.array([0.3, -0.2, 0.1]))


def _diagonals(sysm):
    from olcao_gb300 import api
    ctx = api.Context(sysm)
    out = []
    for op, term in ((3, 0), (4, 0), (4, 2)):
        vv = ctx.gauss_overlap(op, term)[0].cpu().numpy()
        out.append(np.einsum("kii->k", vv).real)
    ctx.close()
    return np.array(out)


@pytest.mark.gpu
@pytest.mark.parametrize("reps", [2, 4, 12])
def test_supercell_trace(gpu_lib, reps):
    folded = [[i / reps, 0.0, 0.0] for i in range(reps)]
    cell = _diagonals(_cell(1, folded)).sum(axis=1)
    super_ = _diagonals(_cell(reps, [[0.0, 0.0, 0.0]]))[:, 0]
    assert np.abs(super_ - cell).max() <= 1e-10 * np.abs(cell).max()
