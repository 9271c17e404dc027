"""The device's refined reciprocal and reciprocal square root (rcp_pos, rsqrt_pos) themselves, compiled
from the kernels' header, over the exponents whose reciprocals are normal: within 1.5 units in the last
place (relative 1.5 * 2^-52), the bound that the series leaves on a start of 20 correct bits.  The
residuals are formed in 80-bit arithmetic, whose own roundings are 2^-64."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, requires_gpu

pytestmark = [pytest.mark.gpu, requires_gpu]

SOURCE = """
#include "common.cuh"
__global__ void reciprocals(const double* x, double* r, double* s, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  r[i] = sb200::rcp_pos(x[i]);
  s[i] = sb200::rsqrt_pos(x[i]);
}
extern "C" int run(const double* x, double* r, double* s, int n) {
  double* d = nullptr;
  const size_t b = (size_t)n * 8;
  if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 1;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  reciprocals<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
  cudaMemcpy(r, d + n, b, cudaMemcpyDeviceToHost);
  cudaMemcpy(s, d + 2 * n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)cudaGetLastError();
}
"""


def test_reciprocals_are_within_one_and_a_half_ulp(tmp_path):
    (tmp_path / "r.cu").write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "--expt-relaxed-constexpr", "-shared", "-cudart", "static", "-I",
                    str(ROOT / "streams-2_b200" / "csrc" / "cuda"), "-I", str(ROOT / "include"),
                    "-o", str(tmp_path / "r.so"), str(tmp_path / "r.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "r.so"))
    rng = np.random.default_rng(5)
    e = np.arange(-1020, 1021)
    m = np.concatenate([rng.uniform(1.0, 2.0, 200), [1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0)]])
    x = np.ldexp(m[:, None], e[None, :]).ravel()
    x = np.ascontiguousarray(np.concatenate([x, np.nextafter(x[-2 * e.size:], 0.0)]))
    r, s = np.empty_like(x), np.empty_like(x)
    p = ctypes.POINTER(ctypes.c_double)
    assert lib.run(*(a.ctypes.data_as(p) for a in (x, r, s)), ctypes.c_int(x.size)) == 0
    xl, rl, sl = (a.astype(np.longdouble) for a in (x, r, s))
    assert np.finfo(np.longdouble).nmant >= 63
    assert float(np.abs(rl * xl - 1).max()) <= 1.5 * 2.0 ** -52
    assert float(np.abs((sl * xl) * sl - 1).max()) <= 2 * 1.5 * 2.0 ** -52  # (1 + d)^2
