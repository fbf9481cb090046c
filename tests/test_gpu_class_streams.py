"""Third-centre classes on side streams (gpu): while stages are timed the
classes run one after the other on the context's stream, otherwise beside each
other; the blocks are the same numbers, call after call, and so with
accumulation (the sum of all operators in one pass)."""

import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["c2", "sif"])
def test_streams_do_not_change_blocks(gpu_lib, kind):
    from olcao_gb300 import api
    sysm = S.small_test_system(kind, nk=(2, 1, 1))
    ctx = api.Context(sysm)

    def passes():
        out = []
        for args in ((3,), (4, 0), (4, 3), (6, 0, sysm.pot_coeffs), (6, 0, sysm.pot_coeffs, api.PREC_MIXED)):
            out += [x.cpu().numpy().copy() for x in ctx.gauss_overlap(*args) if x is not None]
        return out

    together = passes()
    ctx.profile(True)
    alone = passes()
    ctx.profile(False)
    again = passes()
    ctx.close()
    for a, b, c in zip(together, alone, again):
        assert (a == b).all() and (a == c).all()
