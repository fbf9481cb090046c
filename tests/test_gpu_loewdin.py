"""The orthonormalisation step of the mixed solver over tile edges (gpu): its
Hermitian products form lower tiles only, and the basis is transformed only
where eigenvectors are asked for.  Neither may show: eigenvalues with and
without vectors are the same numbers, and the vectors stay orthonormal in the
prepared overlap to the FP32 grade of the basis (1e-4, as the solver's own
comparison with the FP64 path takes it)."""

import numpy as np
import pytest

from olcao_gb300 import system as S

SYSTEMS = {"104": lambda: S.silicon_supercell(1, mesh=(1, 1, 2)), "117": lambda: S.quartz(reps=1)}


@pytest.mark.gpu
@pytest.mark.parametrize("n", sorted(SYSTEMS))
def test_vectors_do_not_change_eigenvalues(gpu_lib, n):
    import torch
    from olcao_gb300 import api
    sysm = SYSTEMS[n]()
    ctx = api.Context(sysm)
    ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
    nv = ctx.vale_dim
    assert nv == int(n)
    alone = ctx.scf_iteration(sysm.pot_coeffs, nv, precision=api.PREC_MIXED)
    vec = torch.zeros(ctx.nk, nv, nv, dtype=torch.complex128, device="cuda")
    both = ctx.scf_iteration(sysm.pot_coeffs, nv, precision=api.PREC_MIXED, vectors=vec)
    assert (alone == both).all()
    _, s = ctx.scf_matrices(sysm.pot_coeffs, 0)
    x = vec[0].cpu().numpy().T                                   # columns are vectors
    err = np.abs(x.conj().T @ s @ x - np.eye(nv)).max()
    ctx.close()
    assert err <= 1e-4
