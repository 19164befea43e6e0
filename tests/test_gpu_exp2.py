"""The FP64 integrands' 2^x against exact values: within 0.85 units in the last
place (half a unit of the final sum, the rest of the small term's rounding and
of exponents near a power of two), and the library's results where |x| is large
or not finite."""
import ctypes
import math
import os
import shutil
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sfsim_gb300", "csrc")
SOURCE = """
#include "exp2_table.cuh"
__global__ void evaluate(const double* x, double* y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = sfsim::exp2_table(x[i]);
}
extern "C" int run(const double* x, double* y, int n) {
  double* d = nullptr;
  if (cudaMalloc(&d, 2 * n * sizeof(double))) return 1;
  cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
  evaluate<<<(n + 255) / 256, 256>>>(d, d + n, n);
  const cudaError_t e = cudaMemcpy(y, d + n, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def exp2(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    d = tmp_path_factory.mktemp("exp2")
    (d / "exp2.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, "-o", str(d / "exp2.so"), str(d / "exp2.cu")], check=True)
    lib = ctypes.CDLL(str(d / "exp2.so"))

    def call(x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.empty_like(x)
        p = ctypes.POINTER(ctypes.c_double)
        assert lib.run(x.ctypes.data_as(p), y.ctypes.data_as(p), x.size) == 0
        return y
    return call


@pytest.mark.parametrize("lo,hi", [(-1.0, 0.0), (-200.0, 0.0), (-999.0, 999.0), (-1e-6, 1e-6)])
def test_within_a_unit(exp2, lo, hi):
    getcontext().prec = 50
    ln2 = Decimal(2).ln()
    x = np.concatenate([np.random.default_rng(1).uniform(lo, hi, 1500), np.linspace(lo, hi, 513)])
    for a, y in zip(x, exp2(x)):
        exact = (Decimal(float(a)) * ln2).exp()
        ulp = Decimal(2) ** (math.frexp(float(exact))[1] - 53)
        assert abs(Decimal(float(y)) - exact) <= Decimal("0.85") * ulp, (a, y)


def test_large_and_not_finite(exp2):
    y = exp2(np.array([1000.0, -1000.0, 1023.5, -1030.0, -1080.0, 1e9, -1e9, math.inf, -math.inf, math.nan, 0.0, -0.0]))
    np.testing.assert_allclose(y[:4], np.exp2([1000.0, -1000.0, 1023.5, -1030.0]), rtol=1e-12)
    assert list(y[4:9]) == [0.0, math.inf, 0.0, math.inf, 0.0] and math.isnan(y[9]) and list(y[10:]) == [1.0, 1.0]
