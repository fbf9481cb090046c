"""The two tensor-core products at the edges of their tiles, K-blocks, digits
and pieces (gpu), against extended-precision products.

FP64-accurate product: operands keep 56 bits below their row's (column's)
largest magnitude, so an element's error is at most 2 k terms of each of two
truncations, 2^-56 of the scale product each, plus one rounding of the
result.  FP32-accurate product: the dropped piece pairs (3 of 2^-24), 24
accumulator additions per K-block and one register addition per K-block,
each 2^-24 of sum |a||b|.
"""

import numpy as np
import pytest

SHAPES = [(1, 1, 1), (2, 3, 31), (31, 33, 32), (127, 63, 33), (128, 64, 64), (129, 65, 65), (130, 200, 257),
          (257, 129, 96), (70, 300, 700)]


@pytest.fixture(scope="module")
def ctx(gpu_lib):
    from olcao_gb300 import api
    from olcao_gb300 import system as S
    c = api.Context(S.small_test_system("c2", nk=(1, 1, 1)))
    yield c
    c.close()


def _operands(kind, m, n, k, rng):
    a = rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))
    b = rng.standard_normal((k, n)) + 1j * rng.standard_normal((k, n))
    if kind == "graded":                       # 30 decades inside rows and columns
        a *= 10.0 ** rng.uniform(-15, 15, (m, k))
        b *= 10.0 ** rng.uniform(-15, 15, (k, n))
    elif kind == "ones":                       # every mantissa bit set, one sign: the largest digit sums
        full = np.nextafter(1.0, 0.0)
        a = np.full((m, k), full * (1 + 1j))
        b = np.full((k, n), full * (1 - 1j))
        a[::2] *= -1.0
    elif kind == "zeros":
        a[rng.random((m, k)) < 0.7] = 0.0
        b[:, ::2] = 0.0
    return a, b


def _exact(a, b):
    L = np.longdouble
    ar, ai, br, bi = (x.astype(L) for x in (a.real, a.imag, b.real, b.imag))
    return ar @ br - ai @ bi, ar @ bi + ai @ br


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["normal", "graded", "ones", "zeros"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_split_zgemm_edges(ctx, kind, m, n, k):
    import torch
    a, b = _operands(kind, m, n, k, np.random.default_rng(m * 1000 + k))
    c = ctx.split_zgemm(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
    re, im = _exact(a, b)
    ra = np.maximum(np.abs(a.real), np.abs(a.imag)).max(1)[:, None] * 2
    cb = np.maximum(np.abs(b.real), np.abs(b.imag)).max(0)[None, :] * 2
    bound = 4 * k * 2.0 ** -56 * ra * cb
    for got, ref in ((c.real, re), (c.imag, im)):
        assert (np.abs(got - ref) <= bound + 2.0 ** -52 * np.abs(ref)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("kind", ["normal", "ones", "zeros"])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_split_cgemm32_edges(ctx, kind, m, n, k, conj):
    import torch
    a, b = (x.astype(np.complex64) for x in _operands(kind, m, n, k, np.random.default_rng(m * 1000 + k + 1)))
    at = torch.from_numpy(np.ascontiguousarray(a.conj().T) if conj else a).cuda()
    c = ctx.split_cgemm32(at, torch.from_numpy(b).cuda(), conj_a=conj).cpu().numpy()
    re, im = _exact(a.astype(np.complex128), b.astype(np.complex128))
    aa, ab = np.abs(a.real) + np.abs(a.imag), np.abs(b.real) + np.abs(b.imag)
    bound = (28 + 25 * ((2 * k + 63) // 64)) * 2.0 ** -24 * (aa.astype(float) @ ab.astype(float)) + 1e-37
    for got, ref in ((c.real, re), (c.imag, im)):
        assert (np.abs(got - ref) <= bound).all()
