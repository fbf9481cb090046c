"""FP32-accurate product (gpu): its rounding errors have no preferred sign and do not
grow as K gets short.  Like-signed operands of one binade, the case where cut-off bits
add up.  The leading piece pair's products have 16 bits and their sum over a drain of 256
of K' is below 2^10 of the smallest one, an exact number, so that what is left is one
rounding per drain and group of the register sum (half of 2^-23, unbiased), the dropped
pairs (3 2^-24) and the five lower pairs' sum, 2^-7 of the result, cut off 80 times per
drain at 2^-23 of itself: mean within 2^-24 of the result, single elements within (4 + drains)
2^-24.
"""

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 8, 33, 64, 100, 128, 129, 320, 1000])
def test_like_signed(gpu_lib, k):
    import torch
    from olcao_gb300 import api
    rng = np.random.default_rng(k)
    ctx = api.Context(S.small_test_system("c2", nk=(1, 1, 1)))
    a, b = ((rng.random(s).astype(np.float32) + 1).astype(np.complex64) for s in ((200, k), (k, 170)))
    c = ctx.split_cgemm32(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
    ctx.close()
    ref = a.real.astype(float) @ b.real.astype(float)
    rel = (c.real.astype(float) - ref) / ref
    drains = (2 * ((k + 31) // 32 * 32) + 255) // 256
    assert not c.imag.any()
    assert abs(rel.mean()) <= 2.0 ** -24
    assert np.abs(rel).max() <= (4 + drains) * 2.0 ** -24
