"""The right-hand sides' chunked sums over source panels: chunk lengths that do not divide the bodies,
headings around the eight of one pass."""
import numpy as np
import pytest

import hams_b200
import meshgen
import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbeta", [0, 1, 7, 8, 9, 17])
@pytest.mark.parametrize("boxes", [[(3, 7, 2)], [(2, 3, 1), (5, 5, 2)], [(11, 9, 4), (3, 5, 3)]], ids=str)
def test_right_hand_sides(boxes, nbeta):
    """Bodies of 61, 16 + 65 and 259 + 63 panels against the oracle; sums of at most 322 terms in another
    order, and the assembly's bound of 1e-10."""
    bodies = [meshgen.box(9.0, 6.0, 4.0, *b, 25.0 * k, 0.0) for k, b in enumerate(boxes)]
    xyz, ncn, ncon, cnt = meshgen.combine(bodies)
    xr = np.array([[25.0 * k, 0.0, 0.0] for k in range(len(boxes))])
    ctx = hams_b200.Context(hams_b200.prepare_geometry(xyz, ncn, ncon, cnt, xr), -1.0, rho=1025.0, g=9.81)
    oc = oracle_lib.Case(xyz, ncn, ncon, cnt, xr, -1.0, rho=1025.0, g=9.81)
    betas = np.linspace(0.0, 3.0, nbeta)
    _, b, d = ctx.assemble(ctx.wave(0.9), betas)
    _, ob, od = oc.assemble(oc.wave(0.9), betas)
    assert np.linalg.norm(b - ob[:, :, 0]) < 1e-10 * np.linalg.norm(ob)
    if nbeta:
        assert np.linalg.norm(d - od[:, 0, :]) < 1e-10 * np.linalg.norm(od)
    ctx.close()
