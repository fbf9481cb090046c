"""Orthogonalisation and packing over tile edges (gpu): random blocks against
the three-product form in FP64, O_vv - (S^H O_cv + O_cv^H S) + S^H O_cc S.

The products keep 53 bits below their row's (column's) largest magnitude:
with entries of at most 6 in S and O_cv and 6 nc in O_cc S (FP64 rounding of
the same sums in the reference form included) an element of the result is off
by at most 16 nc^2 36 2^-52, far above what is seen and far below 1e-6.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S

SYSTEMS = {
    "one partial tile (10)": lambda: S.small_test_system("c2", nk=(2, 1, 1)),
    "one partial tile (26)": lambda: S.small_test_system("si2", nk=(2, 1, 2)),
    "two ragged tiles (33)": lambda: S.small_test_system("sif", nk=(1, 1, 1)),
    "four tiles, ragged (104)": lambda: S.silicon_supercell(1, mesh=(1, 1, 2)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_ortho_pack_random(gpu_lib, name, overlap):
    import torch
    from olcao_gb300 import api
    ctx = api.Context(SYSTEMS[name]())
    nk, n, nc = ctx.nk, ctx.vale_dim, ctx.core_dim
    rng = np.random.default_rng(n + overlap)

    def rand(*shape):
        x = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        return np.clip(x.real, -4, 4) + 1j * np.clip(x.imag, -4, 4)

    # column-major blocks: [k][column][row]
    vv, scv, ocv, cc = rand(nk, n, n), rand(nk, n, nc), rand(nk, n, nc), rand(nk, nc, nc)
    cc = cc + cc.conj().transpose(0, 2, 1)
    vv = vv + vv.conj().transpose(0, 2, 1)
    if overlap:
        ocv = scv
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (vv, ocv, cc, scv)]
    packed = ctx.ortho_pack(overlap, *dev).cpu().numpy()
    ctx.close()
    s, o = scv.transpose(0, 2, 1), ocv.transpose(0, 2, 1)          # [k][row][column]
    sh = s.conj().transpose(0, 2, 1)
    x = sh @ o
    ref = vv.transpose(0, 2, 1) - x - x.conj().transpose(0, 2, 1) + sh @ cc.transpose(0, 2, 1) @ s
    col, row = np.tril_indices(n)
    want = ref[:, row, col]
    got = packed[..., 0] + 1j * packed[..., 1]
    tol = 16.0 * nc * nc * 36.0 * 2.0 ** -52 + 1e-10
    assert np.abs(got - want).max() <= tol
    assert not got[:, row == col].imag.any()
