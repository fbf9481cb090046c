"""Both forms of the tridiagonalisation (gpu) where only they differ: orders above 192,
the one with fixed-point sums (OLC_TRD_DET=1) and the one with FP32 atomics (0), even
and odd (a padding row, a last strip of one to seven columns, blocks of 32 rows that end
ragged).  Eigenvalues against the FP64 path at the mixed path's 1e-6 Ha.  And the
largest order that the path takes.
"""

import ctypes as C

import numpy as np
import pytest

from olcao_gb300 import system as S


def _chain(natoms, extra):
    """Silicon atoms in a row, the last `extra` of a type with one s function less."""
    rng = np.random.default_rng(6)
    pos = np.array([[4.6 * i, 0.0, 0.0] for i in range(natoms)]) + rng.normal(0, 0.1, (natoms, 3))
    types = [S.silicon_type(rng), S.make_type(rng, 2, 18, 0.12, 1.0e6, (18, 18, 12, 0), (0, 1, 2, 1), (0, 0, 1))]
    site = np.array([0] * (natoms - extra) + [1] * extra, np.int32)
    pots = [S.silicon_pot(), S.silicon_pot(2)]
    return S.System(name="chain", real_vectors=np.diag([4.6 * natoms, 9.0, 9.0]), types=types, site_type=site,
                    site_pos=pos, pots=pots, pot_site_type=site.copy(), pot_site_pos=pos,
                    kpoints_abc=S.mp_mesh((1, 1, 2), (0.5, 0.5, 0.5)),
                    pot_coeffs=0.1 * np.random.default_rng(60).standard_normal(32))


@pytest.mark.gpu
@pytest.mark.parametrize("natoms,extra", [(15, 0), (16, 1), (17, 3), (25, 2)])
def test_orders(gpu_lib, monkeypatch, natoms, extra):
    from olcao_gb300 import api
    sysm = _chain(natoms, extra)
    ctx = api.Context(sysm)
    n = ctx.vale_dim
    assert n == 13 * natoms - extra and n > 192
    ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
    want = ctx.scf_iteration(sysm.pot_coeffs, n, precision=api.PREC_FP64)
    for det in ("1", "0"):
        monkeypatch.setenv("OLC_TRD_DET", det)
        for g in (1, 3, 8):
            monkeypatch.setenv("OLC_TRD_CLUSTER", str(g))
            got = ctx.scf_iteration(sysm.pot_coeffs, n, precision=api.PREC_MIXED)
            assert np.abs(got - want).max() <= 1e-6, f"n={n} G={g} det={det}"
    ctx.close()


@pytest.mark.gpu
def test_largest_order(gpu_lib):
    f = gpu_lib._ZN3olc11hetrd_max_nEv
    f.restype = C.c_int
    assert f() == 8908
