"""The arithmetic of csrc/gc_math.cuh against CUDA's, through a kernel compiled here.

Reciprocal: the last operation rounds z = y + y (r + r^2) and leaves an error below 2^-62 of the
quotient beside that rounding, so the result is the rounded quotient or a neighbour of it.
Rotation: c and s carry a few roundings each (c three, s one more), so c^2 + s^2 is 1 to 8 units of
2^-53; the FP32 tangent has an error of at most 2^-20 of itself (truncated operands, product, sum, root,
sum and quotient: eight roundings of 2^-23), and an error of t by delta t leaves 2 delta h at most."""
import ctypes
import subprocess
from fractions import Fraction as F

import numpy as np
import pytest
import torch

from gammcor_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = """
#include "gc_math.cuh"
__global__ void rec(int n, const double *x, double *y, double *ref) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) { y[i] = gc::reciprocal(x[i]); ref[i] = 1.0 / x[i]; }
}
__global__ void rot(int n, const double *h, const double *d, double *c, double *s) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) gc::jacobi_rotation(h[i], d[i], c + i, s + i);
}
extern "C" int run_rec(int n, const double *x, double *y, double *ref) {
  rec<<<(n + 255) / 256, 256>>>(n, x, y, ref);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_rot(int n, const double *h, const double *d, double *c, double *s) {
  rot<<<(n + 255) / 256, 256>>>(n, h, d, c, s);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    (d / "m.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I",
                    str(build.CSRC), str(d / "m.cu"), "-o", str(d / "m.so")], check=True)
    return ctypes.CDLL(str(d / "m.so"))


def call(fn, *inputs):
    dev = [torch.as_tensor(x, device="cuda") for x in inputs]
    out = [torch.zeros_like(dev[0]) for _ in range(2)]
    torch.cuda.synchronize()
    assert fn(len(inputs[0]), *(ctypes.c_void_p(t.data_ptr()) for t in dev + out)) == 0
    return [t.cpu().numpy() for t in out]


def test_reciprocal_is_the_quotient_or_its_neighbour(lib):
    rng = np.random.default_rng(0)
    one = np.float64(1.0)
    m = np.concatenate([[one, np.nextafter(one, 2), 1.5, np.nextafter(2 * one, 1), 2 - 2.0 ** -24],
                        1.0 + np.arange(64) * 2.0 ** -23, 2.0 - np.arange(1, 65) * 2.0 ** -23,
                        rng.uniform(1.0, 2.0, 2000)])
    e = np.r_[0, 1, -1, 52, -52, 999, 1000, 1001, 1022, 1023, -999, -1000, -1001, -1021, -1022,
              rng.integers(-1000, 1001, 40)]
    x = np.concatenate([np.ldexp(m, k) for k in e] + [[5e-324, 2.0 ** -1040, 1e-310, np.inf]])
    y, ref = call(lib.run_rec, x)
    inside = np.abs(np.frexp(x)[1] - 1) <= 1000
    assert np.array_equal(y[~inside], ref[~inside])                     # CUDA's own division there
    assert np.abs(y.view(np.int64) - ref.view(np.int64)).max() <= 1


def test_rotation_is_orthogonal_and_shrinks_its_element(lib):
    rng = np.random.default_rng(1)
    n = 4000
    h = rng.standard_normal(n) * 2.0 ** rng.integers(-60, 60, n)
    d = h * rng.standard_normal(n) * 2.0 ** rng.integers(-70, 70, n)
    d[::17] = 0.0
    h[1::19] *= 2.0 ** -900
    d[1::19] *= 2.0 ** -900
    c, s = call(lib.run_rot, h, d)
    for i in range(n):
        hh, dd, cc, ss = F(float(h[i])), F(float(d[i])), F(float(c[i])), F(float(s[i]))
        assert abs(cc * cc + ss * ss - 1) <= F(8, 2 ** 53), (h[i], d[i])
        # a_pp = 0, a_qq = d: the rotated off-diagonal element
        assert abs(hh * (cc * cc - ss * ss) - cc * ss * dd) <= abs(hh) / 2 ** 19, (h[i], d[i])
        assert c[i] > 0 and abs(s[i]) <= c[i] * (1 + 2.0 ** -20), (h[i], d[i])
