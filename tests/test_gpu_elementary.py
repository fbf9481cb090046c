"""The elementary functions written out in olc_elementary.cuh (gpu) against
extended precision: exp_neg and quotient, through a small kernel of each compiled here.

exp_neg: one rounding of the table entry and one of the result, 2^-53 of the value
each at most (the entries lie in [1/2, 1]), the remainder of the quintic (4e-17) and the
roundings of its product with |r| <= ln 2 / 128 (below 0.02 2^-53): within 2.4 2^-53 of the
value.  quotient: the last step rounds q + r (a - b q) with an exact residual and a
reciprocal good to 2^-23: half an ulp and 2^-21 of one.
"""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "olc_elementary.cuh"
__global__ void exp_kernel(const double* t, int n, double* out) {
  __shared__ double tab[64];
  if (threadIdx.x < 64) tab[threadIdx.x] = olc::kExp2Neg[threadIdx.x];
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = olc::exp_neg(t[i], tab);
}
__global__ void quotient_kernel(const float* a, const float* b, int n, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = olc::quotient(a[i], b[i]);
}
extern "C" int run_exp(const double* t, int n, double* out) {
  exp_kernel<<<(n + 127) / 128, 128>>>(t, n, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_quotient(const float* a, const float* b, int n, float* out) {
  quotient_kernel<<<(n + 127) / 128, 128>>>(a, b, n, out);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def kernels(gpu_lib, tmp_path_factory):
    from olcao_gb300 import build
    d = tmp_path_factory.mktemp("elementary")
    src, so = d / "kernels.cu", d / "kernels.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-I", build.CSRC, "-shared",
                    "-o", str(so), str(src)], check=True)
    return C.CDLL(str(so))


def _run(f, dtype, *args):
    import torch
    x = [torch.from_numpy(np.ascontiguousarray(a, dtype)).cuda() for a in args]
    out = torch.empty_like(x[0])
    p = [C.c_void_p(t.data_ptr()) for t in x]
    torch.cuda.synchronize()
    assert f(*p, C.c_int(x[0].numel()), C.c_void_p(out.data_ptr())) == 0
    return out.cpu().numpy()


@pytest.mark.gpu
def test_exp_neg(kernels):
    rng = np.random.default_rng(1)
    step = np.log(2.0) / 64
    t = np.concatenate([[0.0, 5e-324, 1e-300, 1e-17, 706.9, 707.0], rng.uniform(0, 706.9, 400000),
                        10.0 ** rng.uniform(-18, 2, 100000),
                        np.repeat(step * np.arange(1, 65000), 3) * (1 + np.tile([-1e-15, 0, 1e-15], 64999))])   # table edges
    got = _run(kernels.run_exp, np.float64, t).astype(np.longdouble)
    ref = np.exp(-t.astype(np.longdouble))
    assert (np.abs(got - ref) <= 2.4 * np.longdouble(2.0) ** -53 * ref).all()
    # 0 from there on, whatever the low bits of 64 t / ln 2 are
    wrap = 46516320.0 * np.arange(1, 200)[:, None] + np.linspace(0, 1600, 3001)[None, :]
    far = np.concatenate([[707.9, 708.0, 709.0, 800.0, 1e6, 1e9, 1e18, 1e100, 1e300, 1.7e308, np.inf], wrap.ravel(),
                          10.0 ** rng.uniform(2.86, 308, 100000)])
    assert not _run(kernels.run_exp, np.float64, far).any()


@pytest.mark.gpu
def test_quotient(kernels):
    rng = np.random.default_rng(2)
    n = 1000000
    b = (2.0 ** rng.uniform(-99, 99, n)).astype(np.float32) * rng.choice([-1, 1], n).astype(np.float32)
    q = 2.0 ** rng.uniform(-40, 40, n)
    with np.errstate(over="ignore"):
        a = (q * np.abs(b)).astype(np.float32)
    ok = (a < 2.0 ** 120) & (a > 2.0 ** -90)
    a, b = a[ok], b[ok]
    near = rng.integers(1 << 23, 1 << 24, 200000).astype(np.float32)       # quotients close to 1 and to ties
    a = np.concatenate([a, near, np.ones(200000, np.float32)])
    b = np.concatenate([b, near + rng.integers(-3, 4, 200000).astype(np.float32), near])
    got = _run(kernels.run_quotient, np.float32, a, b).astype(np.float64)
    ref = a.astype(np.longdouble) / b.astype(np.longdouble)
    ulp = np.spacing(np.abs(ref).astype(np.float32)).astype(np.float64)
    assert (np.abs(got - ref) <= (0.5 + 2.0 ** -21) * ulp).all()
