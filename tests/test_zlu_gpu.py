"""zlu_solve (csrc/lu_fp64.cu) by itself: systems that no small deck has -- random ones whose pivots move
rows over the whole height, clusters of 1 to 16 blocks, batches, right-hand sides around the 8 and 16
columns of its kernels, zero pivots, and entries near the ends of the exponents' range."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_series import CSRC

pytestmark = pytest.mark.gpu

SHIM = r"""
#include "lu_fp64.h"
extern "C" int supported(int n) { return zlu_supported(n); }
// batch systems a (n x n) and x (n x nrhs), column by column, one after another; x is replaced by the solution
extern "C" int solve(int batch, int n, int nrhs, const double* a, double* x, int* info) {
  if (zlu_supported(n)) return 100;
  cublasHandle_t blas;
  cudaStream_t st;
  double2 *A = nullptr, *X = nullptr;
  int *work = nullptr, *dinfo = nullptr, rc = 101;
  const size_t sa = (size_t)n * n, sx = (size_t)n * nrhs;
  long long la = 0, lb = 0;
  if (cublasCreate(&blas) || cudaStreamCreate(&st)) return 102;
  cublasSetStream(blas, st);
  if (!cudaMalloc(&A, batch * sa * 16) && !cudaMalloc(&X, batch * sx * 16) &&
      !cudaMalloc(&work, zlu_work_ints(batch) * 4) && !cudaMalloc(&dinfo, 4) &&
      !cudaMemcpy(A, a, batch * sa * 16, cudaMemcpyHostToDevice) &&
      !cudaMemcpy(X, x, batch * sx * 16, cudaMemcpyHostToDevice)) {
    rc = zlu_solve(st, blas, batch, n, nrhs, A, sa, X, sx, dinfo, work, nullptr, &la, &lb);
    if (cudaStreamSynchronize(st) || cudaMemcpy(x, X, batch * sx * 16, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(info, dinfo, 4, cudaMemcpyDeviceToHost))
      rc = 103;
  }
  cudaFree(A);
  cudaFree(X);
  cudaFree(work);
  cudaFree(dinfo);
  cudaStreamDestroy(st);
  cublasDestroy(blas);
  return rc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("zlu")
    (d / "shim.cu").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o", so, str(d / "shim.cu"),
                    os.path.join(CSRC, "lu_fp64.cu"), "-L/usr/local/cuda/lib64", "-lcublas", "-lcudart", "-Xlinker",
                    "-rpath,/usr/local/cuda/lib64"], check=True)
    return ctypes.CDLL(so)


def _solve(lib, a, b):
    """a (batch, n, n), b (batch, n, nrhs) -> the solutions and the info word."""
    at = np.ascontiguousarray(a.transpose(0, 2, 1))
    xt = np.ascontiguousarray(b.transpose(0, 2, 1)).copy()
    info, P = ctypes.c_int(-1), ctypes.POINTER(ctypes.c_double)
    rc = lib.solve(a.shape[0], a.shape[1], b.shape[2], at.ctypes.data_as(P), xt.ctypes.data_as(P), ctypes.byref(info))
    assert rc == 0, rc
    return xt.transpose(0, 2, 1), info.value


def _random(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("n,nrhs,batch", [
    (1, 1, 3), (2, 8, 1), (15, 9, 2), (16, 16, 1), (17, 17, 3), (64, 7, 5), (65, 1, 2), (130, 33, 4),
    (513, 9, 2), (1025, 17, 1), (2049, 9, 1), (4097, 17, 1), (8192, 8, 1)])
def test_random_systems(lib, n, nrhs, batch):
    """Partial pivoting on random matrices: a growth of n^(2/3) and so a backward error of n^(5/3) units."""
    rng = np.random.default_rng(n)
    a, b = _random(rng, batch, n, n), _random(rng, batch, n, nrhs)
    x, info = _solve(lib, a, b)
    assert info == 0
    for k in range(batch):
        back = np.linalg.norm(a[k] @ x[k] - b[k]) / (np.linalg.norm(a[k]) * np.linalg.norm(x[k]))
        assert back < n ** (5.0 / 3.0) * 2.0 ** -53, (k, back)


@pytest.mark.parametrize("n,zero", [(1, 0), (40, 39), (65, 0), (65, 17), (65, 63), (65, 64), (700, 513), (2100, 2099)])
def test_zero_pivot(lib, n, zero):
    """A column of zeros is left with a zero pivot, its number from one; of two such the first."""
    rng = np.random.default_rng(n + zero)
    a, b = _random(rng, 1, n, n), _random(rng, 1, n, 3)
    a[0, :, zero] = 0.0
    assert _solve(lib, a, b)[1] == zero + 1
    a[0, :, n - 1] = 0.0
    assert _solve(lib, a, b)[1] == zero + 1


def test_zero_pivot_of_a_batch(lib):
    rng = np.random.default_rng(1)
    a, b = _random(rng, 4, 100, 100), _random(rng, 4, 100, 2)
    assert _solve(lib, a, b)[1] == 0
    a[2, :, 70] = 0.0
    assert _solve(lib, a, b)[1] == 71


@pytest.mark.parametrize("power", [-960, -400, 400, 960])
def test_scaled_system_has_the_same_bits(lib, power):
    """Every entry of the matrix times a power of two: the same pivots, and the solution divided by it."""
    rng = np.random.default_rng(3)
    a, b = _random(rng, 1, 150, 150), _random(rng, 1, 150, 5)
    want, _ = _solve(lib, a, b)
    got, info = _solve(lib, a * 2.0 ** power, b)
    assert info == 0
    assert np.array_equal(got * 2.0 ** power, want)


def test_supported_orders(lib):
    assert [lib.supported(n) for n in (0, 1, 512, 8192, 8193)] == [1, 0, 0, 0, 1]
