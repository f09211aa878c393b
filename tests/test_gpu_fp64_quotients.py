"""FP64 reciprocal, quotient and square root of the transport against IEEE.

The last fused operation of each rounds a value whose error before the rounding
is far below an ulp, so ordinary operands give IEEE's bits and only operands at
a midpoint (mantissas of ones, powers of two) may differ, by one ulp.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from tam_gb300 import build

SOURCE = """
#include "transport_common.cuh"
namespace {
__global__ void ops(const double *a, const double *b, double *o, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = tam::rcp64(b[i]);
    o[n + i] = tam::div64(a[i], b[i]);
    o[2 * n + i] = tam::sqrt64(fabs(a[i]));
}
}
extern "C" int run_ops(const double *a, const double *b, double *o, int n)
{
    double *d = nullptr;
    if (cudaMalloc(&d, 5 * sizeof(double) * n) != cudaSuccess) return 1;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
    ops<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
    const int rc = cudaMemcpy(o, d + 2 * n, 3 * sizeof(double) * n, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    p = tmp_path_factory.mktemp("quotients")
    (p / "ops.cu").write_text(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(p / "ops.so"), str(p / "ops.cu")], check=True)
    return ctypes.CDLL(str(p / "ops.so"))


def operands(kind):
    r = np.random.default_rng(5)
    if kind == "hard":
        m = np.array([1.0, np.nextafter(1, 2), np.nextafter(1, 0), np.nextafter(2, 0), 1.5, np.nextafter(1.5, 2)])
        v = np.ldexp(m[:, None], np.arange(-400, 401, 25)).ravel()
        a, b = (x.ravel() for x in np.meshgrid(np.concatenate([v, -v, [0.0]]), np.concatenate([v, -v])))
        return a, b
    n = 1 << 20
    e = {"walk": 2.0, "wide": 120.0}[kind]
    return tuple(r.choice([-1.0, 1.0], n) * 10.0 ** r.uniform(-e, e, n) for _ in range(2))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,ulps", [("walk", 0), ("wide", 0), ("hard", 1)])
def test_bits_of_ieee(lib, kind, ulps):
    a, b = (np.ascontiguousarray(x) for x in operands(kind))
    o = np.empty((3, a.size))
    ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, o)]
    assert lib.run_ops(*ptr, ctypes.c_int(a.size)) == 0
    for got, want in zip(o, (1.0 / b, a / b, np.sqrt(np.abs(a)))):
        assert np.abs(got.view(np.int64) - want.view(np.int64))[want != 0].max() <= ulps
        assert (got[want == 0] == 0).all()
