"""The epsilon series: the row-ordered table (csrc/epsilon.h) against the reference's column order,
and the assembled system over meshes with many and with few equal pair distances."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import hams_b200
import meshgen
import oracle_lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hams-mrel_b200", "csrc")

SHIM = r"""
#include <cmath>
#include <vector>
#include "epsilon.h"
using namespace hams;
// Limes, FinGrnExtSubs.f90:370-470, column by column
static double columns(int n, std::vector<double> s) {
  std::vector<double> a(n + 2, 0.0);
  double amax = 0.0, rl = s[n];
  for (int k = 1; n - 2 * k + 1 >= 0; ++k) {
    for (int i = 0; i <= n - 2 * k + 1; ++i) a[i] = s[i + 1] != s[i] ? a[i + 1] + 1.0 / (s[i + 1] - s[i]) : a[i + 1];
    for (int i = 0; i <= n - 2 * k; ++i) {
      s[i] = a[i + 1] != a[i] ? s[i + 1] + 1.0 / (a[i + 1] - a[i]) : s[i + 1];
      if (std::fabs(a[i]) > amax) {
        amax = std::fabs(a[i]);
        rl = s[i];
        if (s[i + 1] == s[i]) return rl;
      }
    }
  }
  return rl;
}
extern "C" void both(int n, const double* s, double* out) {
  const int rows = n + 1, r0 = n % kEpsRows + 1, pad = kEpsRows - r0;
  std::vector<double> e(eps_columns(rows), NAN);
  std::vector<uint32_t> m(eps_pairs(rows), 0xdeadbeefu);
  EpsBest b;
  double x[kEpsRows];
  for (int j = 0; j < kEpsRows; ++j) x[j] = j >= pad ? s[j - pad] : 0.0;
  eps_block(x, 0, pad, e.data(), m.data(), 1, r0 < rows, b);
  for (int q = r0; q < rows; q += kEpsRows) {
    for (int j = 0; j < kEpsRows; ++j) x[j] = s[q + j];
    eps_block(x, q, 0, e.data(), m.data(), 1, q + kEpsRows < rows, b);
  }
  out[0] = columns(n, std::vector<double>(s, s + n + 1));
  out[1] = eps_result(b, s[n]);
  out[2] = b.redo;
}
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    d = tmp_path_factory.mktemp("eps")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["/usr/bin/g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                    "-I", CSRC, "-o", so, str(d / "shim.cpp")], check=True)
    lib = ctypes.CDLL(so)

    def run(s):
        s = np.ascontiguousarray(s, dtype=np.float64)
        out = np.zeros(3)
        lib.both(len(s) - 1, s.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                 out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
        return out

    return run


def _terms(kind, n, rng):
    i, r, x = np.arange(n), np.exp(-rng.uniform(0.02, 2.0)), rng.uniform(-1.0, 1.0, n)
    return {"noise": x, "geometric": r ** i * x[:1].repeat(n), "waves": r ** i * np.cos(0.3 * i + x[:1]),
            "gaps": np.where(rng.uniform(size=n) < 0.3, 0.0, x), "steps": 0.25 * rng.integers(-1, 2, n),
            "settled": np.where(i > n // 2, 0.0, r ** i), "zero": np.zeros(n),
            "last bits": r ** i * (1.0 + 2.0 ** -52 * rng.integers(0, 4, n))}[kind]


@pytest.mark.parametrize("kind", ["noise", "geometric", "waves", "gaps", "steps", "settled", "zero", "last bits"])
def test_row_order_gives_the_column_order_bits(both, kind):
    """Every series length (0 to 98 terms), with ties, zero differences, converged and empty tails."""
    rng = np.random.default_rng(7)
    redo = total = 0
    for n in range(99):
        for _ in range(12):
            ref, got, again = both(np.concatenate([[0.0], np.cumsum(_terms(kind, n, rng))]) if n else np.zeros(1))
            total += 1
            redo += again != 0.0
            # a table that asks for the column order is repeated there by the kernel
            assert again or ref == got or (np.isnan(ref) and np.isnan(got)), (kind, n, ref, got)
    if kind in ("noise", "waves"):
        assert redo < 0.2 * total


def _rough(bodies, size, seed):
    """Every node moved by up to `size`, so that hardly two pair distances are equal."""
    rng, out = np.random.default_rng(seed), []
    for xyz, ncn, ncon in bodies:
        p = xyz + rng.uniform(-size, size, xyz.shape)
        p[:, 2] = np.minimum(np.where(xyz[:, 2] == 0.0, 0.0, p[:, 2]), 0.0)
        out.append((p, ncn, ncon))
    return out


# meshes: equal distances (numbered rows); none, below and above the size at which the tables of the
# EIGENE distances go a chunk of pairs at a time; depths that reach
# all branches and nearly one
MESHES = {
    "equal": ([meshgen.cylinder(4.0, 6.0, 12, 3, 2), meshgen.box(9.1, 5.0, 4.0, 5, 3, 2, 17.3, 1.0)], 30.0),
    "shallow": ([meshgen.cylinder(4.0, 6.0, 12, 3, 2), meshgen.cylinder(4.0, 6.0, 12, 3, 2, 12.0, 0.0)], 6.03),
    "deep": ([meshgen.cylinder(4.0, 6.0, 12, 3, 2)], 180.0),
    "rough": (_rough([meshgen.cylinder(4.0, 6.0, 12, 3, 2), meshgen.cylinder(4.0, 6.0, 12, 3, 2, 12.0, 0.0)], 0.02, 1), 30.0),
    "rough large": (_rough([meshgen.cylinder(4.0, 6.0, 40, 10, 6), meshgen.cylinder(4.0, 6.0, 30, 9, 4, 12.0, 0.0)], 0.02, 2),
                    45.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", list(MESHES))
def test_assembly_over_distance_patterns(mesh):
    bodies, h = MESHES[mesh]
    xyz, ncn, ncon, cnt = meshgen.combine(bodies)
    xr = np.zeros((len(bodies), 3))
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, xr)
    ctx = hams_b200.Context(geom, h, rho=1025.0, g=9.81)
    oc = oracle_lib.Case(xyz, ncn, ncon, cnt, xr, h, rho=1025.0, g=9.81)
    betas = np.array([0.4])
    stride = 1 if ncn.size < 300 else 37
    for omega in (0.5, 1.6):
        a, b, d = ctx.assemble(ctx.wave(omega), betas)
        oa, ob, od = oc.assemble_rows(oc.wave(omega), betas, stride)
        # the assembly's bound in test_gpu_parity
        for got, ref in ((a[::stride], oa[:, :, 0]), (b[::stride], ob[:, :, 0]), (d[::stride], od[:, 0, :])):
            assert np.linalg.norm(got - ref) < 1e-10 * np.linalg.norm(ref)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 31, 33, 97, 4096])
@pytest.mark.parametrize("lo,hi", [(1e-4, 2.0), (0.0005, 0.05), (0.05, 0.5)])
def test_points_by_branch_equal_points_one_by_one(n, lo, hi):
    """hams_eval_green files its points by branch and series length; hams_eval_green_static takes them
    a thread each, as they come.  The EIGENE and PIDCOCK sums have the same bits either way, and so has
    LINTON's quadrature by lanes: the results are equal."""
    lib = hams_b200.load_library()
    lib.hams_eval_green_static.argtypes = lib.hams_eval_green.argtypes
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(4.0, 4.0, 8, 2, 2)])
    ctx = hams_b200.Context(hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3))), 31.0, g=9.81)
    rng = np.random.default_rng(n)
    r, th = 31.0 * np.exp(rng.uniform(np.log(lo), np.log(hi), n)), rng.uniform(0.0, 6.28, n)
    pts = np.zeros((n, 6), order="F")
    pts[:, 3], pts[:, 4] = r * np.cos(th), r * np.sin(th)
    pts[:, 2], pts[:, 5] = rng.uniform(-12.0, -0.3, n), rng.uniform(-12.0, -0.3, n)
    flag = (rng.uniform(size=n) < 0.5).astype(np.int32)
    wave = ctx.wave(1.3)
    got, ref = ctx.eval_green(wave, pts, flag), np.zeros((n, 4), dtype=np.complex128, order="F")
    assert lib.hams_eval_green_static(ctx._h, ctypes.byref(wave), n, pts.ctypes.data_as(hams_b200.P_dbl),
                                      flag.ctypes.data_as(hams_b200.P_int),
                                      ref.ctypes.data_as(hams_b200.P_dbl)) == 0
    assert np.array_equal(got, ref)
    ctx.close()
