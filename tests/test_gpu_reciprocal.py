"""The pivots' reciprocal (newton_rcp, common.cuh) against 1 / d over the whole range of
FP64, both signs, with zeros, infinities and NaN: within 2^-52 relative (the first step
leaves about 2^-40 of the approximation's error, the second one its own rounding), and
equal to the division where the result is not a normal number."""
import ctypes
import subprocess

import numpy as np
import pytest

from macaw_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"
__global__ void rcp_kernel(const double* d, double* r, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = newton_rcp(d[i]);
}
extern "C" int rcp(const double* d, double* r, int n) {
  double *x, *y;
  if (cudaMalloc(&x, 8 * n) || cudaMalloc(&y, 8 * n)) return 1;
  cudaMemcpy(x, d, 8 * n, cudaMemcpyHostToDevice);
  rcp_kernel<<<(n + 255) / 256, 256>>>(x, y, n);
  const int e = cudaMemcpy(r, y, 8 * n, cudaMemcpyDeviceToHost);
  cudaFree(x);
  cudaFree(y);
  return e;
}
"""


def test_reciprocal(tmp_path):
    src, lib = tmp_path / "rcp.cu", tmp_path / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-Xcompiler", "-fPIC", "-shared",
                    str(src), "-o", str(lib)], check=True)
    rng = np.random.default_rng(5)
    d = np.ldexp(rng.uniform(1.0, 2.0, 1 << 20), rng.integers(-1074, 1024, 1 << 20)) * rng.choice([-1.0, 1.0], 1 << 20)
    ends = np.ldexp(1.0, np.array([-1074, -1073, -1023, -1022, -1021, -1020, 1019, 1020, 1021, 1022, 1023]))
    d = np.concatenate([d, ends, -ends, 1.5 * ends, [0.0, -0.0, np.inf, -np.inf, np.nan, np.finfo(float).max]])
    out = np.empty_like(d)
    p = ctypes.POINTER(ctypes.c_double)
    assert ctypes.CDLL(str(lib)).rcp(d.ctypes.data_as(p), out.ctypes.data_as(p), ctypes.c_int(d.size)) == 0
    with np.errstate(all="ignore"):
        ref = 1.0 / d
    normal = np.isfinite(ref) & (np.abs(ref) >= np.finfo(float).tiny)
    assert (np.abs(out[normal] - ref[normal]) <= 2.0 ** -52 * np.abs(ref[normal])).all()
    assert np.array_equal(out[~normal], ref[~normal], equal_nan=True)
