"""hams_eval_green: tables of one branch only, whatever their number."""
import ctypes

import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 130, 4096])
@pytest.mark.parametrize("odd", [None, 0.2, np.nan])
def test_one_branch(n, odd):
    """All at R/h >= 0.5, or one of them nearer or no number: the bits of the points taken one by one."""
    lib = hams_b200.load_library()
    lib.hams_eval_green_static.argtypes = lib.hams_eval_green.argtypes
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(4.0, 4.0, 8, 2, 2)])
    ctx = hams_b200.Context(hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3))), 31.0, g=9.81)
    rng = np.random.default_rng(n)
    r, th = 31.0 * rng.uniform(0.5, 3.0, n), rng.uniform(0.0, 6.28, n)
    if odd is not None:
        r[n // 2] = 31.0 * odd
    pts = np.zeros((n, 6), order="F")
    pts[:, 3], pts[:, 4] = r * np.cos(th), r * np.sin(th)
    pts[:, 2], pts[:, 5] = rng.uniform(-12.0, -0.3, n), rng.uniform(-12.0, -0.3, n)
    flag = (rng.uniform(size=n) < 0.5).astype(np.int32)
    wave, ref = ctx.wave(1.3), np.zeros((n, 4), dtype=np.complex128, order="F")
    rc = lib.hams_eval_green_static(ctx._h, ctypes.byref(wave), n, pts.ctypes.data_as(hams_b200.P_dbl),
                                    flag.ctypes.data_as(hams_b200.P_int), ref.ctypes.data_as(hams_b200.P_dbl))
    if rc:  # the quadrature of a point that is no number may give up: then both do
        with pytest.raises(hams_b200.HamsError):
            ctx.eval_green(wave, pts, flag)
    else:
        assert np.array_equal(ctx.eval_green(wave, pts, flag), ref, equal_nan=True)
    ctx.close()


def test_large_tables_agree_with_their_parts():
    """9,000 points of the branch (listed first) and the same in two parts (looked at by the host)."""
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(4.0, 4.0, 8, 2, 2)])
    ctx = hams_b200.Context(hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3))), 31.0, g=9.81)
    rng, n = np.random.default_rng(1), 9000
    pts = np.zeros((n, 6))
    pts[:, 3] = 31.0 * rng.uniform(0.5, 3.0, n)
    pts[:, 2], pts[:, 5] = rng.uniform(-12.0, -0.3, n), rng.uniform(-12.0, -0.3, n)
    flag, wave = np.zeros(n, dtype=np.int32), ctx.wave(0.7)
    whole = ctx.eval_green(wave, pts, flag)
    parts = np.concatenate([ctx.eval_green(wave, pts[k:k + 4500], flag[k:k + 4500]) for k in (0, 4500)])
    assert np.array_equal(whole, parts)
    ctx.close()


def test_many_linton_points_agree_with_few():
    """5,500 points at R/h < 0.0005 (a thread each) and the same in parts of 500 (a warp each): the lanes of a
    warp take the quadrature's nodes in the thread's order, so the bits are equal."""
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(4.0, 4.0, 8, 2, 2)])
    ctx = hams_b200.Context(hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3))), 31.0, g=9.81)
    rng, n = np.random.default_rng(1), 5500
    pts = np.zeros((n, 6))
    pts[:, 3] = 31.0 * rng.uniform(0.0, 4.9e-4, n)
    pts[:, 2], pts[:, 5] = rng.uniform(-12.0, -0.3, n), rng.uniform(-12.0, -0.3, n)
    flag, wave = np.zeros(n, dtype=np.int32), ctx.wave(1.3)
    whole = ctx.eval_green(wave, pts, flag)
    parts = np.concatenate([ctx.eval_green(wave, pts[k:k + 500], flag[k:k + 500]) for k in range(0, n, 500)])
    assert np.array_equal(whole, parts)
    ctx.close()
