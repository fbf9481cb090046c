"""Contexts of different sizes used by several threads at once (gpu): a launch's
shared-memory limit does not depend on what another thread launched last, and every
result is the one the context gives by itself."""

import threading

import numpy as np
import pytest

from olcao_gb300 import system as S


@pytest.mark.gpu
def test_threads(gpu_lib):
    import torch
    from olcao_gb300 import api
    systems = [S.small_test_system("c2", nk=(1, 1, 1)), S.small_test_system("sif", nk=(1, 1, 1)),
               S.silicon_supercell(1, mesh=(1, 1, 2)), S.quartz(reps=1)]
    ctxs = [api.Context(s) for s in systems]
    for c in ctxs:
        c.scf_prepare(api.PREC_FP64, api.FORM_STORED)
    rng = np.random.default_rng(2)
    a, b = (torch.from_numpy(rng.standard_normal((70, 70)) + 1j * rng.standard_normal((70, 70))).cuda() for _ in "ab")

    def step(q):
        ctx, sysm = ctxs[q], systems[q]
        out = [x.cpu().numpy() for x in ctx.gauss_overlap(api.OP_KINETIC) if x is not None]
        out.append(ctx.split_zgemm(a, b).cpu().numpy())
        out.append(ctx.scf_iteration(sysm.pot_coeffs, ctx.vale_dim, precision=api.PREC_MIXED))
        return out

    alone = [step(q) for q in range(len(ctxs))]
    faults = []

    def work(q):
        try:
            for _ in range(40):
                for x, y in zip(step(q), alone[q]):
                    assert np.array_equal(x, y), f"context {q}"
        except BaseException as e:  # noqa: BLE001
            faults.append(repr(e))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(ctxs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not faults, faults
