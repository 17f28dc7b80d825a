"""The FP64 kernels' reciprocal and roots against 80-bit host arithmetic: their bounds over random
normal arguments of the whole exponent range, and their values at its edges. The bounds follow from
the forms: with u = 2^-53, a correction adds less than 2^-59 relative to the roundings, which are u for
the reciprocal (the last operation), u + u/2 for the root and the reciprocal root (the product with the
argument enters the correction by half), and one u more for a factor (2 % of slack each)."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mhd_gpu_solver_b200 import _capi

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(_capi.LIB_PATH), "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
SOURCE = r"""
#include "physics.cuh"
__global__ void apply(const double* a, const double* x, double* out, int n, int op)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const double v = x[i];
        out[i] = op == 0 ? mhdb::fast_rcp(v) : op == 1 ? mhdb::sqrt_or_zero(v)
               : op == 2 ? mhdb::scaled_rsqrt(1.0, v) : op == 3 ? mhdb::scaled_rsqrt(a[i], v)
               : op == 4 ? mhdb::rcp_any(v) : mhdb::sqrt_any(v);
    }
}
extern "C" int run(const double* a, const double* x, double* out, int n, int op)
{
    double *da = nullptr, *dx = nullptr, *dout = nullptr;
    const size_t bytes = n * sizeof(double);
    if (cudaMalloc(&da, bytes) || cudaMalloc(&dx, bytes) || cudaMalloc(&dout, bytes)) return 1;
    cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(dx, x, bytes, cudaMemcpyHostToDevice);
    apply<<<(n + 255) / 256, 256>>>(da, dx, dout, n, op);
    const cudaError_t e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(dx);
    cudaFree(dout);
    return e == cudaSuccess ? 0 : 2;
}
"""
RCP, SQRT, RSQRT, SCALED, RCP_ANY, SQRT_ANY = range(6)


@pytest.fixture(scope="module")
def apply(tmp_path_factory):
    path = tmp_path_factory.mktemp("primitives")
    src, lib = str(path / "primitives.cu"), str(path / "primitives.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, src, "-o", lib], check=True)
    run = C.CDLL(lib).run

    def call(op, x, a=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        a = np.ones_like(x) if a is None else np.ascontiguousarray(a, dtype=np.float64)
        out = np.empty_like(x)
        p = [v.ctypes.data_as(C.c_void_p) for v in (a, x, out)]
        assert run(*p, x.size, op) == 0
        return out

    return call


def _arguments(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1021, 1021, n))


@pytest.mark.parametrize("op,bound", [(RCP, 1.02), (SQRT, 1.52), (RSQRT, 1.52), (SCALED, 2.52)])
def test_error_bounds(apply, op, bound):
    x = _arguments(1_000_000, op)
    a = np.random.Generator(np.random.PCG64(99)).uniform(0.5, 2.0, x.size)
    xl, al = x.astype(np.longdouble), a.astype(np.longdouble)
    want = {RCP: 1 / xl, SQRT: np.sqrt(xl), RSQRT: 1 / np.sqrt(xl), SCALED: al / np.sqrt(xl)}[op]
    err = np.abs(apply(op, x, a).astype(np.longdouble) - want) / want * 2.0 ** 53
    assert err.max() <= bound, float(err.max())


def test_edges(apply):
    tiny, inf, nan = 5e-324, np.inf, np.nan
    x = np.array([0.0, -0.0, inf, -inf, nan, 1.0, -4.0, 2.0 ** -1022, 2.0 ** 1021, 1e-310, 1e308])
    got = apply(RCP_ANY, x)
    want = np.array([inf, -inf, 0.0, -0.0, nan, 1.0, -0.25, 2.0 ** 1022, 2.0 ** -1021, inf, 0.0])
    assert np.array_equal(got, want, equal_nan=True), got
    assert np.array_equal(np.signbit(got[:4]), np.signbit(want[:4]))
    x = np.array([0.0, inf, nan, 1.0, 4.0, 2.0 ** -1022, 2.0 ** 1022, tiny])
    want = np.array([0.0, inf, nan, 1.0, 2.0, 2.0 ** -511, 2.0 ** 511, 0.0])
    assert np.array_equal(apply(SQRT_ANY, x), want, equal_nan=True)
    assert not apply(SQRT, np.array([0.0, -0.0, -1.0, -inf, tiny, -1e-310])).any()
