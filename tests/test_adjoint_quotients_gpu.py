"""Quotients of the FP64 reverse sweeps (csrc/zj_adjoint.cuh) are IEEE divisions,
correctly rounded, not products with a reciprocal (two or three roundings).

The transposed viscous flux is evaluated where each quotient stands alone: at
rest with rho = 1, gamma = 2 and dv/dy-free shear du/dy = 1, T = p = rho E exactly,
so with the adjoint 1 on tau_xy

    the returned Fvb . Fv          is mu            = T^0.7 / Re
    the adjoint of rho E           is (0.7 mu) / T  (the viscosity law's slope)

with every other term an exact zero.  Both are compared bit for bit with the same
two operations in numpy, T^0.7 taken from the device routine.  A small harness is
compiled here with nvcc for sm_100a."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "ns_kernels.cuh"
#include "zj_adjoint.cuh"
__global__ void k(const double* T, double Re, double* pw, double* mu, double* eb, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s[4] = {1.0, 0.0, 0.0, T[i]}, dx[4] = {0.0, 0.0, 0.0, 0.0}, dy[4] = {0.0, 1.0, 0.0, 0.0};
    const double Fb[4] = {0.0, 0.0, 1.0, 0.0}, Gb[4] = {0.0, 0.0, 0.0, 0.0};
    double sb[4] = {0.0, 0.0, 0.0, 0.0}, xb[4] = {0.0, 0.0, 0.0, 0.0}, yb[4] = {0.0, 0.0, 0.0, 0.0};
    mu[i] = zj::adj::viscous_vjp(s, dx, dy, 2.0, Re, 2.0 / 0.72, Fb, Gb, sb, xb, yb);
    eb[i] = sb[3];
    pw[i] = zj::zj_pow07(T[i]);
}
extern "C" int run(const double* T, double Re, double* out, int n) {
    double *dT = nullptr, *d = nullptr;
    if (cudaMalloc(&dT, n * 8) != cudaSuccess || cudaMalloc(&d, 3 * n * 8) != cudaSuccess) return 1;
    cudaMemcpy(dT, T, n * 8, cudaMemcpyHostToDevice);
    k<<<(n + 127) / 128, 128>>>(dT, Re, d, d + n, d + 2 * n, n);
    const cudaError_t e = cudaMemcpy(out, d, 3 * n * 8, cudaMemcpyDeviceToHost);
    cudaFree(dT); cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
'''


@pytest.mark.parametrize("Re", [50.0, 5000.0, 3.0e6])
def test_viscosity_quotients_are_correctly_rounded(tmp_path, Re):
    (tmp_path / "m.cu").write_text(SRC)
    so = tmp_path / "m.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "zhijian_b200", "csrc"), str(tmp_path / "m.cu"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.run.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_int]
    n = 1 << 16
    T = 10.0 ** np.random.default_rng(3).uniform(-3.0, 6.0, n)
    out = np.empty((3, n))
    assert lib.run(T.ctypes.data, Re, out.ctypes.data, n) == 0
    pw, mu, eb = out
    assert np.array_equal(mu, pw / Re)
    assert np.array_equal(eb, 0.7 * mu / T)
