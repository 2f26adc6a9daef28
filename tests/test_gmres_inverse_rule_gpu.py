"""Which bodies GMRES inverts: blocks of up to 5,000 rows by the complex128 LU, above that the library's
factors, as before there were inverses.  Both sides of the line against the direct solve."""
import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,rows,inverse", [(70, (50, 20), True), (72, (50, 20), False)])
def test_line_between_inverses_and_factors(nt, rows, inverse):
    """Two bodies of 4,900 and of 5,040 panels.  Tolerance 1e-11 on the preconditioned residual, systems of
    condition below 1e3: 1e-8."""
    centres = np.array([(25.0 * k, 0.0, 0.0) for k in range(2)])
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(6.0, 9.0, nt, *rows, c[0], 0.0) for c in centres])
    assert list(cnt) == [nt * 70] * 2
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, centres)
    kw = dict(rho=1025.0, g=9.81)
    wave, betas = hams_b200.wave_properties(0.9, -1.0, 9.81), [0.3]
    direct = hams_b200.Context(geom, -1.0, **kw)
    want = direct.solve_frequency(wave, betas)
    direct.close()
    ctx = hams_b200.Context(geom, -1.0, solver=hams_b200.SOLVER_GMRES, gmres_restart=40, gmres_maxit=400,
                            gmres_tol=1e-11, gmres_dense=1, **kw)
    own = ctx.launch_count()
    got = ctx.solve_frequency(wave, betas)
    own = ctx.launch_count() - own
    assert ctx.note() == "", ctx.note()
    # the own LU launches several kernels for each of its 77 blocks of columns
    assert (own > 77 * 6) == inverse, own
    for p, q in zip(got, want):
        assert np.linalg.norm(p - q) < 1e-8 * np.linalg.norm(q)
    ctx.close()
    hams_b200.release_cached()
