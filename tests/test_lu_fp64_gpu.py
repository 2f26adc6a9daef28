"""The plain form's complex128 LU and solve (16-column panels in a cluster of 512-row blocks, 64-column
blocks) against LAPACK's solution of the assembled system."""
import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


def _amas(geom, x, rho):
    """Added mass of a single body from the radiation potentials (RFORCE)."""
    return rho * (np.asarray(geom["dxyz"]) * np.asarray(geom["ds"])[:, None]).T @ x.real


# 12, 16, 20, 31, 48, 61, 63, 64, 65, 80, 127, 128, 129, 511, 512, 513, 1024, 1025 panels:
# around the panels' 16 and the blocks' 64 columns, and around the 512 and 1,024 rows at which the
# panel's cluster grows
SIZES = [(2, 2, 1), (2, 3, 1), (2, 2, 2), (3, 5, 1), (2, 11, 1), (3, 7, 2), (3, 5, 3), (2, 15, 1), (5, 5, 2),
         (2, 4, 6), (3, 5, 7), (2, 9, 5), (5, 9, 3), (13, 27, 2), (4, 29, 6), (19, 19, 2), (16, 24, 8), (19, 23, 7)]


@pytest.mark.parametrize("nl,nb,nz", SIZES)
def test_solution(nl, nb, nz):
    """A backward-stable solve of systems whose condition is below 1e3: 1e-11 of LAPACK's."""
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.box(12.0, 7.0, 4.0, nl, nb, nz)])
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3)))
    ctx = hams_b200.Context(geom, -1.0, rho=1025.0, g=9.81)
    wave, betas = ctx.wave(0.8), [0.3, 1.0, 2.0]
    a, b, _ = ctx.assemble(wave, betas)
    amas, bdmp, exfc = ctx.solve_frequency(wave, betas)
    ref = _amas(geom, np.linalg.solve(a, b), 1025.0)
    assert np.linalg.norm(amas - ref) < 1e-11 * np.linalg.norm(ref)
    assert np.isfinite(bdmp).all() and np.isfinite(exfc).all()
    again = ctx.solve_frequency(wave, betas)
    assert all(np.array_equal(p, q) for p, q in zip((amas, bdmp, exfc), again))
    ctx.close()
