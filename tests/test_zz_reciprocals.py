"""rcp_ and rsqrt_ of the flux kernels (hardware approximation and one
third-order step) against extended precision over the exponent range, and
against the plain operations outside the range that takes the step.

Bounds.  rcp_: the residual 1 - x r is exact to 2^-53 of itself, the remainder
of the step is the cube of the approximation's error (2^-20), so the final
rounding is all but 2^-6 of an ulp: 0.52 ulp.  rsqrt_: the square of the
approximation y (21 bits) is exact, so 1 - x y^2 rounds once as well, and the same
bound holds."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "eg_internal.h"
#include "eg_kernels.cuh"
#include "eg_physics.cuh"
__global__ void k(const double* x, double* out, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    out[i] = eg::rcp_(x[i]);
    out[n + i] = eg::rsqrt_(x[i]);
    out[2 * n + i] = 1.0 / x[i];
    out[3 * n + i] = ::rsqrt(x[i]);
  }
}
extern "C" int run(const double* x, double* out, int n) {
  double *dx = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&dx, 8 * (size_t)n);
  if (e == cudaSuccess) e = cudaMalloc(&dout, 4 * 8 * (size_t)n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, 8 * (size_t)n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k<<<256, 256>>>(dx, dout, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, 4 * 8 * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dout);
  return (int)e;
}
"""


@pytest.fixture(scope="module")
def reciprocals(tmp_path_factory):
    """x -> rcp_(x), rsqrt_(x), 1 / x, rsqrt(x) on the device"""
    from pdesolver_gb300 import build
    d = tmp_path_factory.mktemp("rcp")
    src, lib = os.path.join(d, "rcp.cu"), os.path.join(d, "librcp.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    r = subprocess.run([build._nvcc(), *build.ARCH, *build.NVFLAGS, "-shared", "-o", lib, src, "-lcudart"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    fn = C.CDLL(lib).run

    def run(x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.zeros((4, x.size))
        assert fn(x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), x.size) == 0
        return out
    return run


def _ulps(got, exact):
    return np.abs((got.astype(np.longdouble) - exact) / np.spacing(np.abs(got))).max()


def _mid_range():
    rng = np.random.default_rng(1)
    m = np.concatenate([rng.uniform(1.0, 2.0, size=1 << 20), 1.0 + np.ldexp(1.0, -np.arange(1, 53)),
                        2.0 - np.ldexp(1.0, -np.arange(0, 53))])
    return np.concatenate([np.ldexp(m, rng.integers(-898, 898, size=m.size)), m, np.ldexp(m, 1)])


def test_accuracy(reciprocals):
    x = _mid_range()
    rcp, rsq, _, _ = reciprocals(x)
    X = x.astype(np.longdouble)
    assert _ulps(rcp, 1 / X) <= 0.52
    assert _ulps(rsq, 1 / np.sqrt(X)) <= 0.52
    assert np.array_equal(reciprocals(-x)[0], -rcp)


def test_range_edges_and_special_values(reciprocals):
    tiny, big = np.ldexp(1.0, -900), np.ldexp(1.0, 900)
    near = np.array([np.nextafter(tiny, 0), tiny, np.nextafter(tiny, 1), np.nextafter(big, 0), big,
                     np.nextafter(big, np.inf)] + [np.ldexp(1.5, e) for e in (-902, -901, -900, 899, 900, 901)])
    for x in (near, -near):
        rcp, rsq, plain, plain_rsq = reciprocals(x)
        assert _ulps(rcp, 1 / x.astype(np.longdouble)) <= 0.52
        if x[0] > 0:
            assert _ulps(rsq, 1 / np.sqrt(x.astype(np.longdouble))) <= 0.52
        else:
            assert np.all(np.isnan(rsq))
    odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-310, 2.2250738585072014e-308,
                    1.7976931348623157e308, -1.7976931348623157e308, 1e-290, -1e-290, 1e290])
    rcp, rsq, plain, plain_rsq = reciprocals(odd)
    assert np.array_equal(rcp, plain, equal_nan=True) and np.array_equal(np.signbit(rcp), np.signbit(plain))
    assert np.array_equal(rsq, plain_rsq, equal_nan=True)
