"""The mixed-precision image sums (gpu) where two atom types of one element have
exponents far apart: the screen's centre then lies far from the pair's own, about which
the suppression that lets an image be summed in FP32 is meant.  Bar: 1e-10 of the
FP64 sum, an FP32 rounding (6e-8) of terms below exp(-22) = 3e-10 and their polynomials.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("ratio", [5.0, 30.0, 200.0])
def test_far_images(gpu_lib, ratio):
    from olcao_gb300 import api
    rng = np.random.default_rng(9)
    types = [S.make_type(rng, 1, 8, 0.4, 2.0e3, (8, 8, 5, 0), (0, 1, 2), (0,)),
             S.make_type(rng, 1, 8, 0.4 * ratio, 2.0e4, (8, 8, 5, 0), (0, 1, 2), (0,))]
    pos = np.array([[0.1, 0.2, 0.3], [1.9, 1.6, 1.4]])
    sysm = S.System(name="far", real_vectors=np.diag([6.5, 7.0, 6.0]), types=types, site_type=np.array([0, 1], np.int32),
                    site_pos=pos, pots=[S.PotSpec(1, 6.0, 20.0, S.even_tempered(4, 0.3, 1e3))],
                    pot_site_type=np.zeros(2, np.int32), pot_site_pos=pos, kpoints_abc=S.mp_mesh((2, 1, 1), (0.5, 0.5, 0.5)),
                    pot_coeffs=0.1 * rng.standard_normal(4))
    ctx = api.Context(sysm)
    want, got = ([b.cpu().numpy() for b in ctx.gauss_overlap(api.OP_HAMILTONIAN, 0, sysm.pot_coeffs * 1e6, precision=p)]
                 for p in (api.PREC_FP64, api.PREC_MIXED))
    ctx.close()
    for w, g in zip(want, got):
        assert np.abs(w - g).max() <= 1e-10 * np.abs(w).max()
