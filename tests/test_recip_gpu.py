"""The column solve's reciprocal (csrc/recip.cuh) against FP64 division: within
one unit in the last place for every exponent, and the division's own result
for zero, infinite, NaN and subnormal arguments and where the quotient is
subnormal.  The bound: Newton-Raphson's second step starts from a relative
error of 2^-40 or less, so only its last rounding is left."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = """
#include "recip.cuh"
__global__ void k(const double* x, double* y, double* z, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { y[i] = olamgpu::recip(x[i]); z[i] = 1.0 / x[i]; }
}
extern "C" int run(const double* x, double* y, double* z, int n) {
  k<<<(n + 255) / 256, 256>>>(x, y, z, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_reciprocal_against_division(tmp_path):
    import torch
    src, lib = tmp_path / "recip.cu", tmp_path / "recip.so"
    src.write_text(SOURCE)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-O3", "-std=c++17", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(ROOT, "olam_b200", "csrc"), "-o", str(lib), str(src)], check=True)
    rng = np.random.default_rng(1)
    e = np.repeat(np.arange(-1074, 1024), 500)
    x = np.ldexp(rng.uniform(1.0, 2.0, e.size), e) * rng.choice([-1.0, 1.0], e.size)
    # 1 + d and 1 - d (the eliminated diagonals), powers of two and their neighbours, the specials
    d = 10.0 ** rng.uniform(-17, 0, 20000)
    p = np.ldexp(1.0, np.arange(-1074, 1024))
    x = np.concatenate([x, 1.0 + d, 1.0 - d[d < 1], p, np.nextafter(p, 0.0), np.nextafter(p, np.inf),
                        [0.0, -0.0, np.inf, -np.inf, np.nan]])
    t = torch.from_numpy(x).cuda()
    y, z = torch.zeros_like(t), torch.zeros_like(t)
    f = ctypes.CDLL(str(lib)).run
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]
    assert f(t.data_ptr(), y.data_ptr(), z.data_ptr(), x.size) == 0
    y, z = y.cpu().numpy(), z.cpu().numpy()
    with np.errstate(all="ignore"):
        ref = 1.0 / x
    assert np.array_equal(z, ref, equal_nan=True)       # the device divides as IEEE does
    tiny = np.finfo(np.float64).tiny                    # the smallest normal number
    plain = (np.abs(ref) >= tiny) & np.isfinite(ref) & (np.abs(x) >= tiny)
    ulp = np.abs(y[plain].view(np.int64) - ref[plain].view(np.int64))
    assert ulp.max() <= 1, ulp.max()
    assert np.array_equal(y[~plain], ref[~plain], equal_nan=True)
    assert np.array_equal(np.signbit(y[~plain & ~np.isnan(ref)]), np.signbit(ref[~plain & ~np.isnan(ref)]))
