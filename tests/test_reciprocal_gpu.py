"""wrcp (aeo_common.cuh) against 1/x: every exponent whose number and reciprocal are normal, both signs, random
mantissas and those beside powers of two.  Bounds: rcp.approx's 1 ulp in FP32; in FP64 the last rounding (half an ulp)
and the series' remainder (2^-57 of the result, 2^-4 ulp at the most), 0.57 ulp."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeolus.jl_b200", "csrc")

SOURCE = r"""
#include "aeo_common.cuh"
template <typename R> __global__ void each(const R* x, R* y, long long n) {
    const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (q < n) y[q] = wrcp(x[q]);
}
template <typename R> int run(const R* x, R* y, long long n) {
    R *dx = nullptr, *dy = nullptr;
    if (cudaMalloc(&dx, n * sizeof(R)) || cudaMalloc(&dy, n * sizeof(R))) return 1;
    int e = cudaMemcpy(dx, x, n * sizeof(R), cudaMemcpyHostToDevice);
    if (!e) each<R><<<(unsigned)((n + 255) / 256), 256>>>(dx, dy, n);
    if (!e) e = cudaGetLastError();
    if (!e) e = cudaMemcpy(y, dy, n * sizeof(R), cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    return e;
}
extern "C" int run_f32(const float* x, float* y, long long n) { return run(x, y, n); }
extern "C" int run_f64(const double* x, double* y, long long n) { return run(x, y, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("wrcp")
    (d / "wrcp.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-shared", "-Xcompiler", "-fPIC", "-I", CSRC, "-o", str(d / "wrcp.so"), str(d / "wrcp.cu")], check=True)
    return ctypes.CDLL(str(d / "wrcp.so"))


@pytest.mark.parametrize("name,dtype,lo,hi,bits,bound", [("run_f32", np.float32, -126, 125, 23, 1.0),
                                                        ("run_f64", np.float64, -1022, 1021, 52, 0.57)])
def test_reciprocal_of_every_exponent(lib, name, dtype, lo, hi, bits, bound):
    rng = np.random.default_rng(7)
    u = 2.0 ** -bits
    near = np.concatenate([1 + u * np.arange(64), 2 - 2 * u * np.arange(1, 65), 1 + 2.0 ** -np.arange(1, bits + 1)])
    m = np.concatenate([near, 1 + u * rng.integers(0, 1 << bits, 4096)]).astype(dtype)
    e = np.arange(lo, hi + 1)
    x = np.ldexp(m[None, :], e[:, None]).astype(dtype).ravel()
    x = np.ascontiguousarray(np.concatenate([x, -x]))
    with np.errstate(all="ignore"):
        want = 1 / x.astype(np.longdouble)
    x = x[np.abs(want) >= np.finfo(dtype).tiny]
    want = want[np.abs(want) >= np.finfo(dtype).tiny]
    y = np.empty_like(x)
    f = getattr(lib, name)
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong]
    assert f(x.ctypes.data, y.ctypes.data, x.size) == 0
    assert np.isfinite(y).all() and (np.sign(y) == np.sign(x)).all()
    ulp = np.ldexp(np.longdouble(1), (np.frexp(want)[1] - 1 - bits).astype(np.int64).astype(np.int32))
    worst = float((np.abs(y.astype(np.longdouble) - want) / ulp).max())
    print(name, "largest error", worst, "ulp")
    assert worst <= bound
