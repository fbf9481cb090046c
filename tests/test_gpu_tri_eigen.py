"""The batched tridiagonal eigen-solve (gpu): the common grid of Sturm shifts,
the multisection and the inverse iteration at the edges of a warp.  The mixed
solver's eigenvalues at a k-point do not depend on how many k-points are
solved beside it (1 x 104 eigenvalues leave a partly filled warp, 4 x 104 none,
188 x 104 more than a warp a sub-partition).  Bar: the mixed path's 1e-6 Ha."""

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("nk", [1, 3, 4, 188])
def test_eigenvalues_independent_of_batch(gpu_lib, nk):
    from olcao_gb300 import api
    kp = np.random.default_rng(nk).uniform(-0.5, 0.5, (nk, 3))

    def eigenvalues(points, precision):
        sysm = S.silicon_supercell(1, mesh=(1, 1, 1))
        sysm.kpoints_abc = points
        ctx = api.Context(sysm)
        ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
        assert ctx.vale_dim == 104
        w = ctx.scf_iteration(sysm.pot_coeffs, 104, precision=precision)
        w = w if isinstance(w, np.ndarray) else w.cpu().numpy()
        ctx.close()
        return w

    few = eigenvalues(kp[[0, nk - 1]], api.PREC_FP64)
    assert np.abs(eigenvalues(kp, api.PREC_MIXED)[[0, nk - 1]] - few).max() <= 1e-6
