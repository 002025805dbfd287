"""The reciprocals and inverse square roots of csrc/dcg_recip.cuh, element by element against 1/x and
1/sqrt(x) in extended precision: over the exponent range, both signs, at powers of two and their
neighbours, at the guards' edges and at the special values.

Bounds, in units in the last place of the result (ulp): fast_rcp and safe_rcp 1 (half for the last
rounding, the series' rest and the roundings of its terms below 2^-55 of the result), fast_rsqrt 1.5
(the rounding of x y adds up to half an ulp through e / 2).  h_recip 2^-46 (1 + 2^-20) relative from
two FP32 roundings squared, and 2^-52 for the FP64 ones."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cuda_runtime.h>
#include <stdint.h>
#include "dcg_recip.cuh"
__global__ void apply(int which, int n, const double *x, double *y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    y[i] = which == 0 ? dcg::fast_rcp(v) : which == 1 ? dcg::safe_rcp(v) : which == 2 ? dcg::fast_rsqrt(v) : dcg::h_recip(v);
}
extern "C" int run(int which, int n, const double *x, double *y) {
    double *dx, *dy;
    if (cudaMalloc(&dx, 8 * (size_t)n) || cudaMalloc(&dy, 8 * (size_t)n)) return 1;
    cudaMemcpy(dx, x, 8 * (size_t)n, cudaMemcpyHostToDevice);
    apply<<<(n + 255) / 256, 256>>>(which, n, dx, dy);
    cudaMemcpy(y, dy, 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def fn(gpu_lib, tmp_path_factory):
    from dirac_caspt2_gb300 import build
    d = tmp_path_factory.mktemp("recip")
    (d / "recip.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    str(d / "recip.cu"), "-o", str(d / "librecip.so")], check=True)
    lib = ctypes.CDLL(str(d / "librecip.so"))

    def call(which, x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.empty_like(x)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        assert lib.run(which, len(x), p(x), p(y)) == 0
        return y

    return call


def _values(lo, hi, signs=True):
    """Doubles with exponents lo..hi - 1: random significands, powers of two and their neighbours."""
    rng = np.random.default_rng(lo + 5000)
    e = np.arange(lo, hi)
    x = np.ldexp(rng.uniform(1.0, 2.0, size=(len(e), 200)), e[:, None]).ravel()
    p = np.ldexp(1.0, e)
    x = np.concatenate([x, p, np.nextafter(p[1:], 0.0), np.nextafter(p, np.inf)])
    return np.concatenate([x, -x]) if signs else x


def _ulps(y, ref):
    return np.abs((y.astype(np.longdouble) - ref) / np.spacing(np.abs(ref.astype(np.float64)))).max()


@pytest.mark.parametrize("which,lo,hi", [(0, -959, 960), (1, -1022, 1022)])
def test_reciprocal(fn, which, lo, hi):
    x = _values(lo, hi)
    assert _ulps(fn(which, x), 1 / x.astype(np.longdouble)) <= 1.0


def test_reciprocal_of_special_values(fn):
    x = np.array([0.0, -0.0, np.inf, -np.inf, 5e-324, -5e-324, 2.0 ** 1023, -2.0 ** 1023])
    with np.errstate(divide="ignore", over="ignore"):
        assert np.array_equal(fn(1, x), 1.0 / x)
        assert np.array_equal(fn(3, x), 1.0 / x)
    assert np.isnan(fn(1, np.array([np.nan]))).all() and np.isnan(fn(3, np.array([np.nan]))).all()


def test_inverse_root(fn):
    x = _values(-1022, 1024, signs=False)
    x = x[np.isfinite(x)]
    assert _ulps(fn(2, x), 1 / np.sqrt(x.astype(np.longdouble))) <= 1.5


def test_reciprocal_by_an_fp32_one(fn):
    x = _values(-1022, 1022)   # FP32 range inside, division outside
    ref = 1 / x.astype(np.longdouble)
    err = np.abs((fn(3, x).astype(np.longdouble) - ref) / ref).max()
    assert err <= 2.0 ** -46 * (1 + 2.0 ** -20) + 2.0 ** -52
