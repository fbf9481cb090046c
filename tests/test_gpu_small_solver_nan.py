"""A pencil that holds NaN or Inf in a batch of the in-shared-memory solver (gpu):
its eigenvalues are not numbers (or, where NaN leaves some alone, numbers of the
matrix: their order is a permutation of the slots that hold them), and the pencils
beside it come out the same to the last bit as in a batch without it."""

import ctypes as C

import numpy as np
import pytest


def _solve(lib, H):
    import torch
    nk, n = H.shape[:2]
    iu = np.tril_indices(n)
    pack = lambda M: np.stack([M.transpose(0, 2, 1)[:, iu[0], iu[1]].real,  # noqa: E731
                               M.transpose(0, 2, 1)[:, iu[0], iu[1]].imag], -1)
    dh = torch.from_numpy(np.ascontiguousarray(pack(H))).cuda()
    ds = torch.from_numpy(np.ascontiguousarray(pack(np.broadcast_to(np.eye(n, dtype=complex), H.shape)))).cuda()
    eig = torch.zeros(nk, n, dtype=torch.float64, device="cuda")
    vec = torch.zeros(nk, n, n, dtype=torch.complex128, device="cuda")
    info = torch.zeros(nk, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.olc_solve_zhegv_noalloc(n, nk, p(dh), p(ds), n, p(eig), p(vec), p(info), None) == 0
    torch.cuda.synchronize()
    return eig.cpu().numpy(), vec.cpu().numpy(), info.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [2, 17, 33, 64])
def test_not_a_number(gpu_lib, n, bad):
    rng = np.random.default_rng(n)
    H = rng.standard_normal((3, n, n)) + 1j * rng.standard_normal((3, n, n))
    H = H + H.conj().transpose(0, 2, 1)
    clean = _solve(gpu_lib, H)
    H[1] = bad                                # every element
    full = _solve(gpu_lib, H)
    assert not np.isfinite(full[0][1]).any()
    H[1] = np.diag(np.arange(n, 0, -1.0))     # one element of a diagonal matrix
    H[1, n // 2, n // 2] = bad
    one = _solve(gpu_lib, H)
    w = one[0][1]
    assert not np.isfinite(w).all() and set(w[np.isfinite(w)]) <= set(np.arange(n, 0, -1.0))
    for eig, vec, info in (full, one):
        assert (info == 0).all()
        for q in (0, 2):
            assert (eig[q] == clean[0][q]).all() and (vec[q] == clean[1][q]).all()
