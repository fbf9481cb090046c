"""The batched in-shared-memory solver on pencils where its FP32 start and its
FP64 refinement can go wrong (gpu), against LAPACK.

Sizes at the edges of its thread counts and column blocks, spectra that are
generic, exactly degenerate, degenerate to 1e-9, graded over 14 decades and
diagonal, and overlaps of condition 1, 1e3 and 1e6; scales far outside
FP32's range.  Bars from backward stability: eigenvalues, residuals and
S-orthonormality within 60 n eps of the norms that enter them (LAPACK's own
bounds have the form c n eps with c of this order).
"""

import ctypes as C

import numpy as np
import pytest

EPS = 2.2e-16
SIZES = [1, 2, 3, 10, 16, 17, 24, 25, 31, 32, 33, 48, 63, 64]
KINDS = ["generic", "degenerate", "near", "graded", "diagonal"]


def _unitary(rng, n):
    return np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]


def _pencil(rng, n, kind, cond, scale):
    lam = np.sort(rng.uniform(-2.0, 3.0, n))
    if kind == "degenerate":
        lam = np.repeat(lam[::4], 4)[:n]
    elif kind == "near":
        lam = np.repeat(lam[::3], 3)[:n] + 1e-9 * np.arange(n)
    elif kind == "graded":
        lam = np.logspace(-8, 6, n)
    Q = np.eye(n) if kind == "diagonal" else _unitary(rng, n)
    A = (Q * lam) @ Q.conj().T
    P = _unitary(rng, n)
    S = (P * np.logspace(-np.log10(cond), 0.0, n)) @ P.conj().T if cond > 1 else np.eye(n, dtype=complex)
    w, U = np.linalg.eigh(S)
    R = (U * np.sqrt(w)) @ U.conj().T
    H = R @ A @ R * scale
    return 0.5 * (H + H.conj().T), 0.5 * (S + S.conj().T)


def _pack(M):
    n = M.shape[-1]
    out = np.empty((M.shape[0], n * (n + 1) // 2, 2))
    c = 0
    for i in range(n):
        out[:, c:c + i + 1, 0] = M[:, :i + 1, i].real
        out[:, c:c + i + 1, 1] = M[:, :i + 1, i].imag
        c += i + 1
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES)
def test_small_solver_pencils(gpu_lib, n):
    import scipy.linalg as sl
    import torch
    rng = np.random.default_rng(100 + n)
    cases = [(k, c, s) for k in KINDS for c, s in ((1.0, 1.0), (1e3, 1.0), (1e6, 1.0))]
    cases += [("generic", 1e3, 1e60), ("generic", 1e3, 1e-60)]
    HS = [_pencil(rng, n, *c) for c in cases]
    H, S = np.stack([h for h, _ in HS]), np.stack([s for _, s in HS])
    nk = len(cases)
    dh, ds = torch.from_numpy(_pack(H)).cuda(), torch.from_numpy(_pack(S)).cuda()
    eig = torch.zeros(nk, n, dtype=torch.float64, device="cuda")
    vec = torch.zeros(nk, n, n, dtype=torch.complex128, device="cuda")
    info = torch.zeros(nk, dtype=torch.int32, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    assert gpu_lib.olc_solve_zhegv_noalloc(n, nk, p(dh), p(ds), n, p(eig), p(vec), p(info), None) == 0
    torch.cuda.synchronize()
    assert (info.cpu().numpy() == 0).all()
    for q, (kind, cond, scale) in enumerate(cases):
        w, X = eig[q].cpu().numpy(), vec[q].cpu().numpy().T
        ref = sl.eigh(H[q], S[q], eigvals_only=True, driver="gv")
        hn, sn, si = np.linalg.norm(H[q], 2), np.linalg.norm(S[q], 2), 1.0 / np.linalg.eigvalsh(S[q])[0]
        what = f"n={n} {kind} cond {cond:g} scale {scale:g}"
        tol = 60 * n * EPS
        assert (np.diff(w) >= 0).all(), what
        assert np.abs(w - ref).max() <= tol * si * (hn + np.abs(ref).max() * sn), what
        assert np.abs(X.conj().T @ S[q] @ X - np.eye(n)).max() <= tol * si * sn, what
        res = H[q] @ X - S[q] @ X * w
        assert np.abs(res).max() <= tol * (hn + np.abs(w).max() * sn) * np.linalg.norm(X, 2) * np.sqrt(si * sn), what
