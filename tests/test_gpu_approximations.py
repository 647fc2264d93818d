"""The straight-line reciprocal and roots of mhd_physics.cuh against extended precision, over random mantissas and
exponents: in ulps of the result.

1/a and sqrt(a) round the corrected value once: half an ulp, and what the correction itself is off, 0.51 and 0.52 as
stated there. 1/sqrt(a) forms its residual from a rounded product (2^-53 of 1, half of which reaches the result: up to
half an ulp) before that rounding: 1.01. sqrt(X/r) = X * (1/sqrt(X r)) adds the rounding of X r, halved, and of the last
product: 3.01 in all.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
SOURCE = r"""
#include "mhd_physics.cuh"
template <int F>
__global__ void apply(const double* a, const double* b, double* o, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = F == 0 ? mhd::rcp_nr(a[i]) : F == 1 ? mhd::sqrt_nr(a[i]) : F == 2 ? mhd::rsqrt_nr(a[i]) : mhd::sqrt_quotient(a[i], b[i]);
}
extern "C" int run(int f, const double* a, const double* b, double* o, long long n) {
    const unsigned g = (unsigned)((n + 255) / 256);
    if (f == 0) apply<0><<<g, 256>>>(a, b, o, n);
    else if (f == 1) apply<1><<<g, 256>>>(a, b, o, n);
    else if (f == 2) apply<2><<<g, 256>>>(a, b, o, n);
    else apply<3><<<g, 256>>>(a, b, o, n);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("approx")
    src, so = str(d / "approx.cu"), str(d / "approx.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    csrc = os.path.join(ROOT, "magnetohydrodynamics_simulator_b200", "csrc")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", csrc, "-shared", "-Xcompiler", "-fPIC", "-o", so, src], check=True)
    lib = ctypes.CDLL(so)
    lib.run.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_longlong]
    return lib


@pytest.mark.parametrize("f,bound", [(0, 0.51), (1, 0.52), (2, 1.01), (3, 3.01)])
def test_error_in_ulps(lib, f, bound):
    import torch

    rng = np.random.default_rng(f)
    worst = 0.0
    for n, lo, hi in ((1 << 23, -300, 300), (1 << 23, -4, 4)):
        a = np.ldexp(1 + rng.random(n), rng.integers(lo, hi, n))
        b = np.ldexp(1 + rng.random(n), rng.integers(lo, hi, n))
        da, db = torch.tensor(a, device="cuda"), torch.tensor(b, device="cuda")
        o = torch.empty_like(da)
        torch.cuda.synchronize()
        assert lib.run(f, da.data_ptr(), db.data_ptr(), o.data_ptr(), n) == 0
        got = o.cpu().numpy()
        A, B = a.astype(np.longdouble), b.astype(np.longdouble)
        want = 1 / A if f == 0 else np.sqrt(A) if f == 1 else 1 / np.sqrt(A) if f == 2 else np.sqrt(A / B)
        err = np.abs((got.astype(np.longdouble) - want).astype(float)) / np.spacing(want.astype(float))
        worst = max(worst, float(err.max()))
    print(f"form {f}: {worst:.4f} ulp")
    assert worst <= bound
