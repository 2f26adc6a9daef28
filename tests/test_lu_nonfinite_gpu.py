"""A system that is not finite is refused by the mixed form, not answered."""
import numpy as np
import pytest

import hams_b200
import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("panel", [0, 63, 64, 100, 250, 358])
def test_mixed_form_refuses_a_column_that_is_not_finite(panel, value):
    """A panel's area that is no number makes its column of the system so: the block LU finds no pivot
    there, the library's LU neither, and the call fails (the panels at the ends of the 64-column blocks, in
    the first, a middle and the last block of 360 columns)."""
    xyz, ncn, ncon, cnt = meshgen.combine([meshgen.cylinder(5.0, 8.0, 18, 7, 3, 30.0 * k, 0.0) for k in range(2)])
    assert sum(cnt) == 360
    geom = hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, np.zeros((2, 3)))
    good = np.array(geom["ds"])
    geom["ds"] = good.copy()
    geom["ds"][panel] = value
    ctx = hams_b200.Context(geom, -1.0, rho=1025.0, g=9.81, precision=hams_b200.PREC_MIXED)
    with pytest.raises(hams_b200.HamsError, match="singular pivot"):
        ctx.solve_frequency(ctx.wave(0.9), [0.3])
    ctx.close()
    geom["ds"] = good
    ctx = hams_b200.Context(geom, -1.0, rho=1025.0, g=9.81, precision=hams_b200.PREC_MIXED)
    assert all(np.isfinite(x).all() for x in ctx.solve_frequency(ctx.wave(0.9), [0.3]))
    ctx.close()
