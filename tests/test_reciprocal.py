"""The reciprocal of the elimination's pivots (lsms_b200/csrc/cplx.cuh), and diagonal blocks of any scale."""

import ctypes
import subprocess

import numpy as np
import pytest

from lsms_b200 import build as B

SRC = r'''
#include "cplx.cuh"
using namespace b200::cx;
// ours, and the same by CUDA's division
__global__ void recip(const double2 *d, double2 *ours, double2 *div, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ours[i] = reciprocal(d[i]);
  int e;
  frexp(fmax(fabs(d[i].x), fabs(d[i].y)), &e);
  const double x = ldexp(d[i].x, -e), y = ldexp(d[i].y, -e), r = 1.0 / (x * x + y * y);
  div[i] = make_double2(ldexp(x * r, -e), ldexp(-y * r, -e));
}
extern "C" int run(const double *d, double *ours, double *div, int n) {
  double2 *p;
  if (cudaMalloc(&p, 3 * n * sizeof(double2)) != cudaSuccess) return 1;
  cudaMemcpy(p, d, n * sizeof(double2), cudaMemcpyHostToDevice);
  recip<<<(n + 255) / 256, 256>>>(p, p + n, p + 2 * n, n);
  cudaMemcpy(ours, p + n, n * sizeof(double2), cudaMemcpyDeviceToHost);
  cudaMemcpy(div, p + 2 * n, n * sizeof(double2), cudaMemcpyDeviceToHost);
  cudaFree(p);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
'''


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("recip")
    (d / "recip.cu").write_text(SRC)
    so = str(d / "recip.so")
    subprocess.run([B.nvcc(), "-shared", "-Xcompiler", "-fPIC", "-O3", "-std=c++17", *B.ARCH, "-I", B.CSRC,
                    str(d / "recip.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def call(d):
        out = [np.empty_like(d), np.empty_like(d)]
        assert lib.run(*(ctypes.c_void_p(a.ctypes.data) for a in (d, *out)), ctypes.c_int(d.size)) == 0
        return out

    return call


@pytest.mark.gpu
def test_reciprocal_over_its_range(run):
    """Squares between 2^-1020 and 2^1020."""
    rng = np.random.default_rng(0)
    n = 200000
    e = rng.integers(-510, 509, size=n)
    x, y = rng.uniform(1.0, 2.0, size=(2, n)) * rng.choice([-1.0, 1.0], size=(2, n))
    other = np.where(rng.random(n) < 0.8, rng.integers(0, 4, size=n), rng.integers(0, 1000, size=n))
    a, b = np.ldexp(x, e), np.ldexp(y, np.maximum(e - other, -1074))
    swap = rng.random(n) < 0.5
    d = np.where(swap, b, a) + 1j * np.where(swap, a, b)
    ours, div = run(d)
    xl, yl = d.real.astype(np.longdouble), d.imag.astype(np.longdouble)
    q = xl * xl + yl * yl
    size = 1 / np.sqrt(q)
    # the sum of squares is off by at most 2 u, its reciprocal by 1.5 u more, each product by u (u = 2^-53)
    for got, bound in ((ours.real - xl / q, 5), (ours.imag + yl / q, 5), (ours - div, 5)):
        assert np.all(np.abs(got) <= bound * 2.0 ** -53 * size)


@pytest.mark.gpu
def test_reciprocal_of_special_values(run):
    d = np.array([0.0, -0.0, complex(np.inf, 1.0), complex(1.0, -np.inf), complex(np.nan, 1.0)])
    got = run(d)[0]
    assert np.all(got[:2] == 0)
    assert np.all(np.isnan(got[2:].real) & np.isnan(got[2:].imag))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-300, 1e-170, 1e-154, 1.2e-154, 1e-100, 1e10, 1e20, 7e153, 1e200])
def test_matrices_of_any_scale(solver_factory, scale):
    """Pivots whose squares leave the range are neither lost nor reported as singular."""
    from lsms_b200 import tau as T
    rng = np.random.default_rng(5)
    n = 96
    m = scale * (np.eye(n) + 0.04 * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))))
    t0 = scale * (rng.normal(size=(16, 16)) + 1j * rng.normal(size=(16, 16)))
    rhs = np.zeros((n, 16), np.complex128)
    rhs[:16] = t0
    want = np.linalg.solve(m / scale, rhs / scale)[:16]
    got = solver_factory(3, 1, 1).solve_tau00_dense(m, t0, T.PREC_FP64)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-10)])
@pytest.mark.parametrize("scale", [1e-12, 1e6, 1e12])
@pytest.mark.parametrize("b", [9, 32])
def test_central_block_of_any_scale(solver_factory, b, scale, prec, tol):
    """The central site's rows and t0 scaled together leave tau00 as it is: the solve with the b x b Schur
    complement keeps its digits."""
    rng = np.random.default_rng(b)
    n = b + 150
    m = np.eye(n) + 0.03 * (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)))
    t0 = rng.normal(size=(b, b)) + 1j * rng.normal(size=(b, b))
    rhs = np.zeros((n, b), np.complex128)
    rhs[:b] = t0
    want = np.linalg.solve(m, rhs)[:b]
    m[:b] *= scale
    got = solver_factory(3, 1, 1).solve_tau00_dense(m, t0 * scale, prec)
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
