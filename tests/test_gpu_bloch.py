"""Bloch sums with one, two and four k-points a thread (gpu): the blocks at a
k-point do not depend on how many others the context holds.  With 36 pairs of
18 x 18 elements a mesh of 27 k-points takes two a thread and 61 take four
(the last group one); contexts of three k-points take one.  The sums run over
the same tasks in the same order, so the bar is rounding of the last
operations: 4 eps of the largest element."""

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
@pytest.mark.parametrize("nk", [27, 30, 54, 61])
def test_blocks_independent_of_mesh(gpu_lib, nk):
    from olcao_gb300 import api
    rng = np.random.default_rng(nk)
    kp = rng.uniform(-0.5, 0.5, (nk, 3))
    kp[0] = 0.0
    pick = [0, nk // 2, nk - 1]

    def blocks(points):
        sysm = S.silicon_supercell(1, mesh=(1, 1, 1))
        sysm.kpoints_abc = points
        ctx = api.Context(sysm)
        out = [[x.cpu().numpy() for x in ctx.gauss_overlap(1)], [x.cpu().numpy() for x in ctx.gauss_overlap(4, 3)]]
        ctx.close()
        return out

    for many, few in zip(blocks(kp), blocks(kp[pick])):
        for a, b in zip(many, few):
            assert np.abs(a[pick] - b).max() <= 4 * np.finfo(float).eps * np.abs(b).max()
