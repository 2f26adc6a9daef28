"""The three kernels of the LINTON rows: a block of four warps per row up to 3 rows per SM, a warp per row
below 64, a thread per row above."""
import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("omega", [0.3, 1.2, 2.5])
def test_many_rows_as_few(omega):
    """Field points straight below the bottom panels, each at its own depth, so each with LINTON rows of its
    own: 20,000 of them at once (a thread per row), in parts of 4,000 (a warp per row) and 2,000 of them in
    parts of 200 (a block per row).  A row is sums and quadratures of some tens of terms in double
    precision, taken in another order by the kernels,
    and the quadrature's acceptance test may then differ where the estimate meets its bound of 1e-6: the
    potentials agree to 1e-9 of the largest."""
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(5.0, 6.0, 12, 3, 2)])
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((1, 3)))
    ctx = hams_b200.Context(geom, 40.0, rho=1025.0, g=9.81)
    centres = np.asarray(geom["xyz_p"])
    centres = centres[np.abs(centres[:, 2] + 6.0) < 1e-9]
    rng, n = np.random.default_rng(2), 20000
    at = rng.integers(0, len(centres), n)
    points = np.column_stack([centres[at, 0], centres[at, 1], -rng.uniform(6.5, 39.5, n)])
    wave, betas = ctx.wave(omega), [0.4]

    def potentials(p):
        ctx.set_field_points(p)
        ctx.solve_frequency(wave, betas)
        return ctx.field_potentials(1)

    whole = potentials(points)
    parts = np.concatenate([potentials(points[k:k + 4000]) for k in range(0, n, 4000)])
    assert whole.shape == parts.shape and np.isfinite(whole).all()
    assert np.abs(whole - parts).max() < 1e-9 * np.abs(whole).max()
    few = np.concatenate([potentials(points[k:k + 200]) for k in range(0, 2000, 200)])
    assert np.abs(whole[:2000] - few).max() < 1e-9 * np.abs(whole).max()
    ctx.close()
