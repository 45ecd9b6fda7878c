"""The reciprocal of the FP64 update's divisor (recip, r2d3c_kernels.cuh) against
the division, in a small library of its own built from the header.

Tolerance: half a unit in the last place and what the iteration leaves, 2^-66
of the value, which is at most 2^-13 of a unit.  (The difference of two nearest
values at a tie is one unit: such cases are measured exactly.)
"""
import ctypes
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from rot2d3c_gb300 import build as B

pytestmark = pytest.mark.gpu

SOURCE = """
#include "r2d3c_pass64.cuh"
__global__ void k(const double* d, double* r, double* q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    r[i] = r2d3c::recip(d[i]);
    q[i] = 1.0 / d[i];
  }
}
extern "C" int run(const double* d, double* r, double* q, int n) {
  k<<<(n + 255) / 256, 256>>>(d, r, q, n);
  return (int)cudaDeviceSynchronize();
}
"""


def values():
    rng = np.random.default_rng(3)
    mant = [rng.uniform(1, 2, 1 << 20)]
    edge = np.concatenate([1 + np.arange(4096) * 2.0 ** -52, 2 - np.arange(1, 4097) * 2.0 ** -52,
                           1 + 2.0 ** -np.arange(1, 53), 2 - 2.0 ** -np.arange(1, 53)])
    # just above and below the FP32 values that the estimate is taken of
    f = rng.uniform(1, 2, 1 << 16).astype(np.float32).astype(np.float64)
    mant += [f, np.nextafter(f, 2), np.nextafter(f, 1)]
    mant = np.clip(np.concatenate(mant), 1, np.nextafter(2, 1))
    out = [np.ldexp(mant, rng.integers(-100, 100, mant.size)), 1 + rng.uniform(0, 1e-3, 1 << 18)]
    out += [np.ldexp(edge, e) for e in (-101, -100, -99, -1, 0, 1, 99, 100, 101)]
    # the division's range, and what is not a positive normal number
    out += [np.ldexp(rng.uniform(1, 2, 4096), rng.integers(-1022, 1023, 4096)), -rng.uniform(0.5, 2, 64),
            np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7e308])]
    return np.concatenate(out)


def test_reciprocal_is_the_nearest(gpu, tmp_path):
    import torch
    src, lib = tmp_path / "recip.cu", tmp_path / "recip.so"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", B.CSRC, "-I",
                    B.INCLUDE, str(src), "-o", str(lib)], check=True, capture_output=True)
    d = values()
    t = torch.from_numpy(d).cuda()
    r, q = torch.empty_like(t), torch.empty_like(t)
    torch.cuda.synchronize()
    ptr = [ctypes.c_void_p(x.data_ptr()) for x in (t, r, q)]
    assert ctypes.CDLL(str(lib)).run(*ptr, ctypes.c_int(d.size)) == 0
    r, q = r.cpu().numpy(), q.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(r), np.isnan(q))
    off = np.flatnonzero((r != q) & ~np.isnan(q))
    assert off.size < 1e-3 * d.size  # 2^-12 of them are that near to a tie
    for i in off:
        exact = 1 / Fraction(float(d[i]))
        assert abs(Fraction(float(r[i])) - exact) <= Fraction(float(np.spacing(q[i]))) * (Fraction(1, 2) + Fraction(1, 2 ** 13))
