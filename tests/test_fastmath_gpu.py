"""The binary64 reciprocal and roots of pmhd/fastmath.hpp against correctly rounded
values, over random mantissas and exponents of their stated domain, and their
special arguments.

Limits: a seed error of at most 2^-19 leaves its cube, 2^-57, before the last
rounding: 0.5 + 2^-4 < 0.6 ulp; fast_rsqrt adds half the rounding of x y, 2^-54 of
the result, at most half an ulp: 1.1."""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <vector>
#include "pmhd/fastmath.hpp"
__global__ void k(const double* x, double* o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[4 * i] = pmhd::fast_rcp(x[i]);
  o[4 * i + 1] = pmhd::fast_rsqrt(x[i]);
  o[4 * i + 2] = pmhd::fast_sqrt(x[i]);
  o[4 * i + 3] = pmhd::fast_sqrt_pos(x[i]);
}
int main(int argc, char** argv) {
  std::vector<double> x;
  double v;
  FILE* f = fopen(argv[1], "rb");
  while (f && fread(&v, 8, 1, f) == 1) x.push_back(v);
  if (f) fclose(f);
  const int n = (int)x.size();
  std::vector<double> o(4 * (size_t)n);
  double *dx, *dout;
  if (cudaMalloc(&dx, 8 * (size_t)n) != cudaSuccess || cudaMalloc(&dout, 32 * (size_t)n) != cudaSuccess) return 2;
  cudaMemcpy(dx, x.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(dx, dout, n);
  if (cudaMemcpy(o.data(), dout, 32 * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
  f = fopen(argv[2], "wb");
  return f && fwrite(o.data(), 8, o.size(), f) == o.size() && fclose(f) == 0 ? 0 : 4;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("fastmath")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "include"), str(d / "t.cu"), "-o", str(d / "t")], check=True)

    def run(x):
        np.ascontiguousarray(x, np.float64).tofile(d / "x")
        subprocess.run([str(d / "t"), str(d / "x"), str(d / "o")], check=True, timeout=120)
        return np.fromfile(d / "o").reshape(-1, 4)

    return run


def _ulps(got, want):
    """Distance in units of the last place of the (extended precision) value."""
    return np.abs(got.astype(np.longdouble) - want) / np.spacing(np.abs(want).astype(np.float64)).astype(np.longdouble)


def test_errors_over_the_stated_domain(program):
    assert np.finfo(np.longdouble).nmant >= 63
    rng = np.random.default_rng(2)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-950, 1000, n))
    # Mantissas at the ends of a binade and around the powers of two as well.
    x[:4096] = np.ldexp(1.0 + np.arange(4096) * 2.0 ** -52, rng.integers(-900, 900, 4096))
    x[4096:8192] = np.ldexp(2.0 - (1 + np.arange(4096)) * 2.0 ** -52, rng.integers(-900, 900, 4096))
    o, X = program(x), x.astype(np.longdouble)
    worst = [float(_ulps(o[:, k], want).max())
             for k, want in enumerate((1 / X, 1 / np.sqrt(X), np.sqrt(X), np.sqrt(X)))]
    assert worst[0] < 0.6 and worst[1] < 1.1 and worst[2] < 0.6 and worst[3] < 0.6, worst
    np.testing.assert_array_equal(program(-x[:1000])[:, 0], -o[:1000, 0])


def test_special_arguments_of_the_square_root(program):
    o = program(np.array([0.0, np.inf, -1.0, -1e-300, 4.0, 2.0 ** -1021]))[:, 2]
    assert o[0] == 0.0 and o[1] == np.inf and np.isnan(o[2]) and np.isnan(o[3]) and o[4] == 2.0
    assert abs(o[5] / np.sqrt(2.0 ** -1021) - 1) < 2.0 ** -51
