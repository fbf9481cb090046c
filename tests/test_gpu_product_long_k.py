"""FP64-accurate product over a long contraction (gpu): past k = 1018035 the
accumulator's unit lies 32 and more bits above the lowest digit group's.  Operands of
small integers, whose low-order digits are all zero and whose product every digit
group holds exactly: the result is exact.  Sizes on both sides of that length and of
the next bit's."""

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("k", [509000, 1018000, 1018100, 2036100])
def test_long_contraction(gpu_lib, k):
    import torch
    from olcao_gb300 import api
    rng = np.random.default_rng(k)
    a, b = rng.integers(-100, 101, (2, 2, k)), rng.integers(-100, 101, (2, k, 2))
    ctx = api.Context(S.small_test_system("c2", nk=(1, 1, 1)))
    c = ctx.split_zgemm(torch.from_numpy(a[0] + 1j * a[1]).cuda(), torch.from_numpy(b[0] + 1j * b[1]).cuda()).cpu().numpy()
    ctx.close()
    assert (c.real == a[0] @ b[0] - a[1] @ b[1]).all() and (c.imag == a[0] @ b[1] + a[1] @ b[0]).all()
