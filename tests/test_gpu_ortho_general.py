"""Orthogonalisation of blocks whose core block is not Hermitian (gpu): it enters as it
is, O_vv - (S^H O_cv + O_cv^H S) + S^H O_cc S, on the stored triangle.  Bound of
tests/test_gpu_ortho.py; one k-point's core block alone, or only by a small part, is off.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S

SYSTEMS = {
    "one partial tile (10)": lambda: S.small_test_system("c2", nk=(2, 1, 1)),
    "two ragged tiles (33)": lambda: S.small_test_system("sif", nk=(1, 1, 1)),
    "four tiles, ragged (104)": lambda: S.silicon_supercell(1, mesh=(1, 1, 2)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("part", [1.0, 1e-9])
@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_core_block_not_hermitian(gpu_lib, name, overlap, part):
    import torch
    from olcao_gb300 import api
    ctx = api.Context(SYSTEMS[name]())
    nk, n, nc = ctx.nk, ctx.vale_dim, ctx.core_dim
    rng = np.random.default_rng(n + overlap)

    def rand(*shape):
        x = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        return np.clip(x.real, -4, 4) + 1j * np.clip(x.imag, -4, 4)

    vv, scv, ocv, cc = rand(nk, n, n), rand(nk, n, nc), rand(nk, n, nc), rand(nk, nc, nc)
    cc = cc + cc.conj().transpose(0, 2, 1)
    k = nk - 1
    cc[k] += part * rand(nc, nc)
    if overlap:
        ocv = scv
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (vv, ocv, cc, scv)]
    packed = ctx.ortho_pack(overlap, *dev).cpu().numpy()
    ctx.close()
    s, o = scv.transpose(0, 2, 1), ocv.transpose(0, 2, 1)          # [k][row][column]
    sh = s.conj().transpose(0, 2, 1)
    x = sh @ o
    ref = vv.transpose(0, 2, 1) - x - x.conj().transpose(0, 2, 1)
    i = np.arange(n)
    ref[:, i, i] = ref[:, i, i].real                                # the rank update leaves a real diagonal
    ref = ref + sh @ cc.transpose(0, 2, 1) @ s
    col, row = np.tril_indices(n)
    want, got = ref[:, row, col], packed[..., 0] + 1j * packed[..., 1]
    assert np.abs(got - want).max() <= 16.0 * nc * nc * 36.0 * 2.0 ** -52 + 1e-10
