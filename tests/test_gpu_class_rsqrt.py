"""The class kernels' reciprocal square root (csrc/eri_common.cuh) on the device, against 64-bit-mantissa
values and against CUDA's rsqrt()."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chronusq_public_b200", "csrc")
SOURCE = """
#include "eri_common.cuh"
__global__ void k(const double *x, double *a, double *b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = class_rsqrt(x[i]), b[i] = rsqrt(x[i]);
}
extern "C" int run(const double *x, double *a, double *b, int n) {
  k<<<(n + 255) / 256, 256>>>(x, a, b, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("rsqrt")
    (d / "r.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-I", CSRC, "-o", str(d / "r.so"), str(d / "r.cu")], check=True)
    return ctypes.CDLL(str(d / "r.so")).run


# s = p + q of two primitive pairs, and m R^2 = p q R^2 of far ones: exponents from 1e-3 to 1e7,
# distances to 1e3
@pytest.mark.parametrize("lo,hi", [(1e-3, 1e8), (1e-2, 1e20), (1.0, 4.0)])
def test_class_rsqrt(run, lo, hi):
    n = 1 << 20
    rng = np.random.default_rng(3)
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    x[:64] = 2.0 ** np.arange(64) if hi > 2.0**64 else x[:64]
    t = torch.tensor(x, device="cuda")
    a, b = torch.empty_like(t), torch.empty_like(t)
    p = lambda v: ctypes.c_void_p(v.data_ptr())
    assert run(p(t), p(a), p(b), n) == 0
    ref = 1.0 / np.sqrt(x.astype(np.longdouble))
    rel = lambda v: np.abs(v.cpu().numpy().astype(np.longdouble) / ref - 1.0).astype(np.float64).max()
    # start y0 within 2^-20 of the value: e = 1 - x y0^2 < 2^-18.9, so the third-order step leaves
    # 5 e^3 / 16 < 2^-58; e carries one rounding of x y0 (2^-53, halved by the step), the terms of the
    # step roundings of 2^-53 |e|, and the last fma one of 2^-53
    assert rel(a) <= 2.0**-53 * 1.51 + 2.0**-58
    # rsqrt() is documented to 1 ulp (2^-52 relative): the two differ by no more than both errors
    diff = ((a - b).abs() / b).max().item()
    assert diff <= 2.0**-53 * 1.51 + 2.0**-58 + 2.0**-52
