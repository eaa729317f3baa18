"""The phase step's logarithm of a quotient and reciprocal square root over their whole range.

The header's device functions, compiled into a small library of their own, against 80-bit arithmetic.
log_ratio: its last operation rounds once (half an ulp of the result), the atanh part s(2 + ...) is
off by at most an ulp of a summand no larger than one and a half times the result: two ulps.
rsqrt_fast: the product x y is off by half an ulp, which the step halves, and the result is rounded
once: 3/4 of 2^-52, asserted at 2^-52.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from mhit36_mixedp_b200 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "phase_math.cuh"
__global__ void k(int n, int what, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = what == 0 ? mhit::log_ratio<false>(a[i], b[i])
                     : (what == 1 ? mhit::log_ratio<true>(a[i], b[i]) : mhit::rsqrt_fast(a[i]));
}
extern "C" int run(int n, int what, const double* a, const double* b, double* out) {
  double* d;
  if (cudaMalloc(&d, 3 * sizeof(double) * n)) return 1;
  cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(n, what, d, d + n, d + 2 * n);
  const int rc = cudaMemcpy(out, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return rc;
}
"""


@pytest.fixture(scope="module")
def run(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    (d / "m.cu").write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I", build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                    str(d / "m.cu"), "-o", str(d / "m.so")], check=True, capture_output=True)
    lib = ctypes.CDLL(str(d / "m.so"))

    def call(what, a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        out = np.empty_like(a)
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, out)]
        assert lib.run(a.size, what, *p) == 0
        return out
    return call


def operands(phi):
    """k_phase's, multi/main.f90:527-528."""
    val = np.minimum(phi, 1.0)
    return val + 1e-16, 1.0 - val + 1e-16


def exact_log(a, b):
    a, b = a.astype(np.longdouble), b.astype(np.longdouble)
    return np.where(np.abs(a - b) < 0.25 * b, np.log1p((a - b) / b), np.log(a / b))


def test_log_ratio_is_within_two_ulps(run):
    rng = np.random.default_rng(0)
    n = 1 << 20
    near = np.concatenate([0.5 + np.arange(-64, 65) * s for s in (2.0**-54, 2.0**-53, 2.0**-50, 2.0**-40, 1e-6)])
    phi = np.concatenate([rng.random(n), 10 ** rng.uniform(-18, 0, n), 1 - 10 ** rng.uniform(-17, 0, n), near,
                          np.linspace(0, 1, n), [0.0, 5e-324, 1e-300, 1e-17, 1.0 - 2.0**-53, 1.0, -5e-17, 1.0 + 2.0**-52]])
    a, b = operands(phi)
    ref = exact_log(a, b)
    ulp = np.spacing(np.abs(ref.astype(np.float64)))
    for what in (0, 1):
        got = run(what, a, b)
        assert (got[a == b] == 0).all()
        assert np.max(np.abs(got.astype(np.longdouble) - ref) / ulp) <= 2.0


def test_log_ratio_outside_its_domain(run):
    phi = np.array([-1e-16, -1.5e-16, -1e-15, -0.5, -1e300, -np.inf, np.nan, np.inf, 2.0])
    a, b = operands(phi)
    assert a[0] == 0.0
    got = run(0, a, b)
    assert got[0] == -np.inf
    assert np.isnan(got[1:7]).all()
    top = float(exact_log(*operands(np.array([1.0])))[0])
    assert np.max(np.abs(got[7:] - top)) <= 2 * np.spacing(top)


def test_rsqrt_fast_is_within_2_to_the_minus_52(run):
    rng = np.random.default_rng(1)
    x = np.concatenate([10 ** rng.uniform(-307, 308, 1 << 20), 10 ** rng.uniform(-70, 4, 1 << 20), 1 + rng.random(1 << 20),
                        1 + 3 * rng.random(1 << 20), 2.0 ** np.arange(-1022, 1024),
                        [np.finfo(float).tiny, np.finfo(float).max]])
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    got = run(2, x, x)
    assert np.max(np.abs(got.astype(np.longdouble) / ref - 1)) <= 2.0**-52
    assert np.isnan(run(2, np.array([np.nan]), np.array([0.0])))[0]
