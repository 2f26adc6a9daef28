"""csrc/epsilon.h as the GPU runs it: its branch-free reciprocal against the correctly rounded one, and
the row-ordered table on the sequences of test_series.py (ties, equal neighbours, converged and empty
tails), which meshes hardly ever produce."""
import ctypes
import subprocess

import numpy as np
import pytest

import test_series

pytestmark = pytest.mark.gpu

SHIM = r"""
#include <cuda_runtime.h>
#include "epsilon.h"
using namespace hams;
__global__ void k_rcp(int n, const double* d, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  out[t] = eps_rcp(d[t]);
  out[n + t] = __drcp_rn(d[t]);
}
// one sequence per thread: partial sums s[off[t]] .. s[off[t + 1] - 1]
__global__ void k_table(int n, const int* off, const double* s, double* e, unsigned* m, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double* q = s + off[t];
  const int rows = off[t + 1] - off[t], r0 = (rows - 1) % kEpsRows + 1, pad = kEpsRows - r0;
  EpsBest b;
  double x[kEpsRows];
#pragma unroll
  for (int j = 0; j < kEpsRows; ++j) x[j] = j >= pad ? q[j - pad] : 0.0;
  eps_block(x, 0, pad, e + t, m + t, n, r0 < rows, b);
  for (int k = r0; k < rows; k += kEpsRows) {
#pragma unroll
    for (int j = 0; j < kEpsRows; ++j) x[j] = q[k + j];
    eps_block(x, k, 0, e + t, m + t, n, k + kEpsRows < rows, b);
  }
  out[t] = eps_result(b, q[rows - 1]);
  out[n + t] = b.redo;
}
template <class T> static T* put(const T* h, size_t n) {
  T* p = nullptr;
  if (cudaMalloc(&p, n * sizeof(T)) == cudaSuccess && h) cudaMemcpy(p, h, n * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}
extern "C" int rcp(int n, const double* d, double* out) {
  double *x = put(d, n), *y = put<double>(nullptr, 2 * (size_t)n);
  k_rcp<<<(n + 255) / 256, 256>>>(n, x, y);
  const int rc = cudaGetLastError() ? 1 : cudaMemcpy(out, y, 2 * (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(x);
  cudaFree(y);
  return rc;
}
extern "C" int table(int n, const int* off, const double* s, int most, double* out) {
  int* o = put(off, n + 1);
  double *x = put(s, off[n]), *y = put<double>(nullptr, 2 * (size_t)n),
         *e = put<double>(nullptr, (size_t)eps_columns(most) * n);
  unsigned* m = put<unsigned>(nullptr, (size_t)eps_pairs(most) * n);
  k_table<<<(n + 63) / 64, 64>>>(n, o, x, e, m, y);
  const int rc = cudaGetLastError() ? 1 : cudaMemcpy(out, y, 2 * (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess;
  cudaFree(o);
  cudaFree(x);
  cudaFree(y);
  cudaFree(e);
  cudaFree(m);
  return rc;
}
"""
P = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("epsgpu")
    (d / "shim.cu").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "--fmad=false", "-Xcompiler", "-fPIC", "-shared", "-I", test_series.CSRC, "-o", so,
                    str(d / "shim.cu")], check=True)
    return ctypes.CDLL(so)


def _rcp(lib, bits):
    d = np.ascontiguousarray(bits.astype(np.uint64)).view(np.float64)
    out = np.zeros(2 * d.size)
    assert lib.rcp(d.size, d.ctypes.data_as(P), out.ctypes.data_as(P)) == 0
    return d, out[:d.size], out[d.size:]


def test_reciprocal_is_correctly_rounded(lib):
    """Every exponent of the range, both signs: significands near one, near all ones, of a single run of
    ones or zeros, and random ones; then random ones in numbers."""
    rng = np.random.default_rng(5)
    full = (1 << 52) - 1
    sig = list(range(40)) + [full - k for k in range(40)]
    for b in range(52):
        sig += [1 << b, (1 << b) - 1, full ^ ((1 << b) - 1), full ^ (1 << b)]
    sig = np.array(sig, dtype=np.uint64)
    exps = np.arange(-1020, 1021, dtype=np.int64)
    e = ((exps + 1023).astype(np.uint64) << np.uint64(52))[:, None]
    some = rng.integers(0, 1 << 52, (exps.size, 300), dtype=np.uint64)
    bits = np.concatenate([(e | sig).ravel(), (e | some).ravel()])
    bits = np.concatenate([bits, bits | np.uint64(1 << 63)])
    many = rng.integers(0, 1 << 52, 20_000_000, dtype=np.uint64) | (rng.integers(993, 1054, 20_000_000).astype(np.uint64)
                                                                    << np.uint64(52))
    for part in (bits, many):
        d, got, want = _rcp(lib, part)
        bad = got.view(np.uint64) != want.view(np.uint64)
        assert not bad.any(), (int(bad.sum()), [(float(x).hex(), float(y).hex()) for x, y in zip(d[bad][:4], got[bad][:4])])


def test_reciprocal_of_special_operands(lib):
    """Zero and subnormal operands give NaN (the table's sign of equal neighbours); operands of 2^1021 and
    more nothing of the size that the table acts on."""
    zero = np.array([0, 1 << 63, 1, (1 << 63) | 1, (1 << 52) - 1, 1 << 51], dtype=np.uint64)
    assert np.isnan(_rcp(lib, zero)[1]).all()
    huge = np.array([2044 << 52, (2045 << 52) | 5, (2046 << 52) | ((1 << 52) - 1), (1 << 63) | (2046 << 52)], dtype=np.uint64)
    assert (np.abs(_rcp(lib, huge)[1]) < 2.0 ** -1020).all()


@pytest.mark.parametrize("kind", ["noise", "geometric", "waves", "gaps", "steps", "settled", "zero", "last bits"])
def test_table_gives_the_column_order_bits(lib, both, kind):
    rng = np.random.default_rng(11)
    seqs = [np.concatenate([[0.0], np.cumsum(test_series._terms(kind, n, rng))]) if n else np.zeros(1)
            for n in range(99) for _ in range(40)]
    off = np.concatenate([[0], np.cumsum([s.size for s in seqs])]).astype(np.int32)
    s = np.ascontiguousarray(np.concatenate(seqs))
    out = np.zeros((2, len(seqs)))
    assert lib.table(len(seqs), off.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), s.ctypes.data_as(P),
                     max(q.size for q in seqs), out.ctypes.data_as(P)) == 0
    host = np.array([both(q) for q in seqs])
    got, again, want = out[0], out[1] != 0.0, host[:, 0]
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    assert (again | same).all(), (kind, np.nonzero(~(again | same))[0][:5])
    assert (again == (host[:, 2] != 0.0)).all()


both = test_series.both
