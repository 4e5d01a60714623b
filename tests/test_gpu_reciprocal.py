"""The reciprocal of the FP64 pair terms (csrc/mf_device.cuh: rcp64) by itself, over the range it is
used in, against the quotient: within 0.5001 units in the last place.

That bound, from its derivation: half a unit for its last rounding; the approximation is within 2^-23 of
1 / x and the argument's rounding to float within 2^-24, so the series' truncated part is below
(1.8e-7)^3 = 6e-21, and a unit is at least 2^-53 of the value: 5e-5 units; the residual's rounding is less.
The error is measured exactly, as 1 - x r with the product in two doubles."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "mf_device.cuh"
__global__ void k_reciprocal(int n, const double *x, double *r) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = mf::rcp64(x[i]);
}
extern "C" int reciprocal(int n, const double *x, double *r) {
  double *dx = nullptr, *dr = nullptr;
  const size_t bytes = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&dx, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&dr, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) k_reciprocal<<<(n + 255) / 256, 256>>>(n, dx, dr);
  if (e == cudaSuccess) e = cudaMemcpy(r, dr, bytes, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dr);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def reciprocal(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("reciprocal")
    (d / "r.cu").write_text(SOURCE)
    r = subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler",
                        "-fPIC", "-I", str(ROOT / "include"), "-I", str(ROOT / "mfree_iwf-ul_cut_gpu_b200" / "csrc"),
                        "-o", str(d / "r.so"), str(d / "r.cu"), "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(d / "r.so"))


def residual(a, b):
    """1 - a b of numbers near 1 whose product is near 1 (Dekker's product: the halves' products are exact)."""
    def halves(v):
        t = v * 134217729.0  # 2^27 + 1
        hi = t - (t - v)
        return hi, v - hi
    (ah, al), (bh, bl) = halves(a), halves(b)
    p = a * b
    low = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    return (1.0 - p) - low


@pytest.mark.parametrize("kind", ["range", "one_octave", "near_ends"])
def test_against_the_quotient(reciprocal, kind):
    rng = np.random.default_rng(8)
    n = 1 << 20
    if kind == "range":  # every magnitude
        x = 10.0 ** rng.uniform(-37, 37, n)
    elif kind == "one_octave":  # mantissas of the reference cut's densities, and their ends
        x = np.concatenate([rng.uniform(1.0, 2.0, n - 64), 1 + np.arange(32) * 2.0**-52, 2 - np.arange(1, 33) * 2.0**-52])
    else:
        x = np.concatenate([1e-37 * rng.uniform(1, 10, n // 2), 1e37 * rng.uniform(0.1, 1, n // 2)])
    x *= rng.choice([-1.0, 1.0], n)
    r = np.empty(n)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert reciprocal.reciprocal(n, p(x), p(r)) == 0
    # x and r scaled to [1/2, 1) and (1, 2]: 1 - x r without rounding, relative to 1 / x
    mx, e = np.frexp(np.abs(x))
    mr = np.ldexp(np.abs(r), e)
    assert (np.sign(r) == np.sign(x)).all()
    err = np.abs(residual(mx, mr)) / mx
    unit = np.spacing(mr)
    assert (err <= 0.5001 * unit).all(), float((err / unit).max())
