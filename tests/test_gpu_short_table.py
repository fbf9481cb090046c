"""Two atom types of one element where the second has more exponents than the first
(gpu).  The screens go by the element's table, that of its first type, and past its
end a radius is infinite.  The pairs of an exponent of the first atom end at the first one
out of reach, so that none past the table's end follows one that is out of reach; the
images of a pair past the table's end are those within its radius of the second atom; a
pair of two exponents past the end has no screen and gives no number.
"""

import numpy as np
import pytest

import oracle as orc
from olcao_gb300 import system as S


def _type(alphas, coeff):
    return S.TypeSpec(element=1, alphas=np.array(alphas), num_orb_alphas=(len(alphas), 0, 0, 0), vale_l=[0], core_l=[],
                      vale_coeff=np.array([coeff], float), core_coeff=np.zeros((0, len(alphas))))


def _system(types, site, pos, cpos, thresh):
    return S.System(name="s", real_vectors=60.0 * np.eye(3), types=types, site_type=np.array(site, np.int32),
                    site_pos=np.array(pos, float), pots=[S.PotSpec(2, 1.0, 3.0, np.array([3.0]))],
                    pot_site_type=np.zeros(1, np.int32), pot_site_pos=np.array([cpos], float),
                    kpoints_abc=np.zeros((1, 3)), pot_coeffs=np.ones(1), thresh=thresh)


S_NORM = 0.2820947917738782 ** 2


def _prim(kind, p):
    return orc.primitive(kind, p, [1, 1])[0, 0]


@pytest.mark.gpu
def test_pairs_end_at_the_first_out_of_reach(gpu_lib):
    from olcao_gb300 import api
    table, more = [0.3, 1.0], [0.3, 1.0, 4.0, 9.0]
    T = -np.log(1e-2)
    # 0.3 reaches 0.3 but not 1.0 at this distance: 4.0 and 9.0 are not reached either
    d = np.sqrt(T * 0.5 * ((1 / 0.3 + 1 / 0.3) + (1 / 0.3 + 1 / 1.0)))
    pos = [[0.0, 0.0, 0.0], [d, 0.0, 0.0]]
    sysm = _system([_type(table, [1, 1]), _type(more, [1, 1, 1, 1])], [0, 1], pos, [1.0, 2.0, 3.0], 1e-2)
    ctx = api.Context(sysm)
    got = ctx.gauss_overlap(api.OP_OVERLAP)[0].cpu().numpy()[0, 1, 0].real / S_NORM
    ctx.close()
    want = _prim(1, [0.3, 0.3, 0, *pos[0], *pos[1], 0, 0, 0])
    assert abs(got - want) <= 1e-12 * abs(want)


@pytest.mark.gpu
def test_images_about_the_second_atom(gpu_lib):
    from olcao_gb300 import api
    pos, cpos = [[0.0, 0.0, 0.0], [8.0, 0.0, 0.0]], [16.0, 0.0, 0.0]
    sysm = _system([_type([0.3], [1]), _type([0.5, 0.8], [0, 1])], [1, 0], pos, cpos, 1e-16)
    ctx = api.Context(sysm)
    for op, kind, sign in ((api.OP_ELECPOT, 4, 1.0), (api.OP_NUCLEAR, 3, -1.0)):
        vv = ctx.gauss_overlap(op)[0].cpu().numpy()[0].real
        want = sign * _prim(kind, [0.8, 0.3, 3.0, *pos[0], *pos[1], *cpos])
        assert want != 0.0 and abs(vv[1, 0] / S_NORM - want) <= 1e-9 * abs(want)
        assert np.isnan(vv[0, 0]) and np.isfinite(vv[1, 1])       # 0.8 with 0.8; 0.3 with 0.3
    ctx.close()
