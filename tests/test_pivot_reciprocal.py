"""The reciprocal that the latency and throughput kernels take of their pivots (seed and two Newton steps in FP64) against
the division: each Newton step squares the seed's error of 2^-20, so what is left is the rounding of the last one, within
a unit in the last place of the correctly rounded quotient."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "symboltz.jl_gb300", "csrc")
SOURCE = r'''
#include "sbz_pt_lat.cuh"
__global__ void run64(int n, const double* x, double* y) { const int i = blockIdx.x * 256 + threadIdx.x; if (i < n) y[i] = sbz::ptk::lat_rcp<double>(x[i]); }
__global__ void run32(int n, const float* x, float* y) { const int i = blockIdx.x * 256 + threadIdx.x; if (i < n) y[i] = sbz::ptk::lat_rcp<float>(x[i]); }
extern "C" int rcp64(int n, const double* x, double* y) { run64<<<(n + 255) / 256, 256>>>(n, x, y); return (int)cudaDeviceSynchronize(); }
extern "C" int rcp32(int n, const float* x, float* y) { run32<<<(n + 255) / 256, 256>>>(n, x, y); return (int)cudaDeviceSynchronize(); }
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    torch = pytest.importorskip("torch")
    nvcc = os.environ.get("NVCC", "nvcc")
    if not torch.cuda.is_available() or not shutil.which(nvcc):
        pytest.skip("no GPU or no nvcc")
    d = tmp_path_factory.mktemp("rcp")
    src, so = d / "rcp.cu", d / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "-I", CSRC, "-shared", "-Xcompiler", "-fPIC",
                    "-o", str(so), str(src)], check=True, capture_output=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("lo,hi", [(-6, 24), (-150, 150)])  # what pivots are, and far beyond
def test_fp64(lib, lo, hi):
    import torch
    rng = np.random.default_rng(hi)
    n = 1 << 22
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo * 10 // 3, hi * 10 // 3, n)) * rng.choice([-1.0, 1.0], n)
    x[:64] = np.ldexp(1.0, np.arange(64) - 32)
    x[64:128] = np.nextafter(np.ldexp(1.0, np.arange(64) - 32), 0)
    t = torch.tensor(x, device="cuda")
    y = torch.empty_like(t)
    assert lib.rcp64(n, C.c_void_p(t.data_ptr()), C.c_void_p(y.data_ptr())) == 0
    ulps = np.abs(y.cpu().numpy().view(np.int64) - (1.0 / x).view(np.int64))
    assert ulps.max() <= 1
    assert np.count_nonzero(ulps) <= n // 1000  # correctly rounded but for near ties


def test_fp32(lib):
    """The hardware approximation: 1 ulp (2^-23) of the exact reciprocal."""
    import torch
    rng = np.random.default_rng(2)
    n = 1 << 20
    x = (np.ldexp(rng.uniform(1, 2, n), rng.integers(-100, 100, n)) * rng.choice([-1.0, 1.0], n)).astype(np.float32)
    t = torch.tensor(x, device="cuda")
    y = torch.empty_like(t)
    assert lib.rcp32(n, C.c_void_p(t.data_ptr()), C.c_void_p(y.data_ptr())) == 0
    np.testing.assert_allclose(y.cpu().numpy().astype(np.float64), 1.0 / x.astype(np.float64), rtol=2.0 ** -23)
