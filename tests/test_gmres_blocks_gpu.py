"""GMRES's body-block preconditioner (inverses by the complex128 LU, runs of equal bodies together)
against the direct solve: bodies in runs of one, two and three sizes, around the panels' 16 and the
blocks' 64 columns, and more than one 512-row block."""
import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


def _count(s):
    nl, nb, nz = s
    return nl * nb + 2 * nz * (nl + nb)


@pytest.mark.parametrize("shapes", [
    [(2, 2, 1), (2, 2, 1)],
    [(3, 7, 2), (3, 5, 3), (3, 5, 3)],
    [(5, 5, 2), (2, 15, 1), (5, 5, 2), (5, 9, 3), (5, 9, 3)],
    [(16, 24, 2), (2, 2, 1), (16, 24, 2)],
])
def test_blocks_match_direct_solve(shapes):
    """Tolerance 1e-11 on the preconditioned residual, systems of condition below 1e3: 1e-8."""
    centres = np.array([(25.0 * i, 0.0, 0.0) for i in range(len(shapes))])
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.box(8.0, 6.0, 4.0, *s, x0=25.0 * i)
                                           for i, s in enumerate(shapes)])
    assert list(cnt) == [_count(s) for s in shapes]
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, centres)
    kw = dict(rho=1025.0, g=9.81)
    direct = hams_b200.Context(geom, 40.0, **kw)
    ctx = hams_b200.Context(geom, 40.0, solver=hams_b200.SOLVER_GMRES, gmres_restart=40, gmres_maxit=400,
                            gmres_tol=1e-11, gmres_dense=1, **kw)
    wave, betas = hams_b200.wave_properties(0.9, 40.0, 9.81), [0.3, 1.0]
    want = direct.solve_frequency(wave, betas)
    got = ctx.solve_frequency(wave, betas)
    assert ctx.note() == "", ctx.note()
    for p, q in zip(got, want):
        assert np.linalg.norm(p - q) < 1e-8 * np.linalg.norm(q)
    again = ctx.solve_frequency(wave, betas)
    assert all(np.array_equal(p, q) for p, q in zip(got, again))
    direct.close()
    ctx.close()
