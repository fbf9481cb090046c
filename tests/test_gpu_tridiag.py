"""The panel kernel of the blocked tridiagonalisation (gpu): eigenvalues of the
mixed solver against the FP64 path for sizes and cluster sizes at the edges
of its ownership (rows in blocks of 32, columns in strips of 16, panels of 32
reflectors, two rows a lane).

n = 104 and 117 (odd) run the small-block variant, 208 and 312 the large one;
one to 16 CTAs per matrix, some of which own no row of the last blocks.  Bar:
the mixed path's 1e-6 Ha; a rerun is bit-identical.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S


def _si(rx):
    rng = np.random.default_rng(6)
    a = 5.431 * S.ANGSTROM
    frac = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0],
                     [.25, .25, .25], [.25, .75, .75], [.75, .25, .75], [.75, .75, .25]])
    pos = np.concatenate([frac + [i, 0, 0] for i in range(rx)]) * a + rng.normal(0, 0.04, (8 * rx, 3))
    t = S.silicon_type(rng)
    n = len(pos)
    return S.System(name="si", real_vectors=a * np.diag([float(rx), 1, 1]), types=[t], site_type=np.zeros(n, np.int32),
                    site_pos=pos, pots=[S.silicon_pot()], pot_site_type=np.zeros(n, np.int32), pot_site_pos=pos,
                    kpoints_abc=S.mp_mesh((1, 1, 2), (0.5, 0.5, 0.5)),
                    pot_coeffs=0.1 * np.random.default_rng(60).standard_normal(16))


SYSTEMS = {104: lambda: _si(1), 117: lambda: S.quartz(reps=1), 208: lambda: _si(2), 312: lambda: _si(3)}


@pytest.mark.gpu
@pytest.mark.parametrize("n", sorted(SYSTEMS))
def test_cluster_sizes(gpu_lib, monkeypatch, n):
    from olcao_gb300 import api
    sysm = SYSTEMS[n]()
    ctx = api.Context(sysm)
    assert ctx.vale_dim == n
    ctx.scf_prepare(api.PREC_FP64, api.FORM_STORED)
    want = ctx.scf_iteration(sysm.pot_coeffs, n, precision=api.PREC_FP64)
    for det in ("1", "0"):
        monkeypatch.setenv("OLC_TRD_DET", det)
        for g in (1, 2, 3, 7, 8, 16):
            monkeypatch.setenv("OLC_TRD_CLUSTER", str(g))
            got = ctx.scf_iteration(sysm.pot_coeffs, n, precision=api.PREC_MIXED)
            assert np.abs(got - want).max() <= 1e-6, f"n={n} G={g} det={det}"
            if det == "1":
                again = ctx.scf_iteration(sysm.pot_coeffs, n, precision=api.PREC_MIXED)
                assert (got == again).all(), f"n={n} G={g}"
    ctx.close()
