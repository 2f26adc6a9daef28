"""Irregular meshes: the pairs of a branch with too many distances for one table are worked off in the order
of their distances, a chunk's table at a time."""
import numpy as np
import pytest

import hams_b200
import meshgen
import test_series
import train_surrogate

pytestmark = pytest.mark.gpu


def _geom():
    # 1,440 panels, about a million distances: several chunks of every branch in 15 m of water
    bodies = test_series._rough([meshgen.cylinder(4.0, 6.0, 40, 12, 6, x, 0.0) for x in (0.0, 14.0)], 0.02, 3)
    return hams_b200.prepare_geometry(*meshgen.combine(bodies), np.array([[0.0, 0.0, 0.0], [14.0, 0.0, 0.0]]))


def test_far_pairs_of_a_surrogate_context():
    """A surrogate context at a frequency outside the network's domain: its far pairs' series run from lists of
    their own, and the system has the bits of a context without the network."""
    geom, betas = _geom(), [0.3]
    plain = hams_b200.Context(geom, 15.0, rho=1025.0, g=9.81)
    wave = plain.wave(1.1)
    want = plain.assemble(wave, betas)
    plain.close()
    ctx = hams_b200.Context(geom, 15.0, rho=1025.0, g=9.81)
    ctx.set_surrogate(train_surrogate.load(), 3.0, (39.0, 40.0))
    assert all(np.array_equal(a, b) for a, b in zip(ctx.assemble(wave, betas), want))
    ctx.set_surrogate(None)
    assert all(np.array_equal(a, b) for a, b in zip(ctx.assemble(wave, betas), want))
    ctx.close()


def test_batch_has_the_bits_of_single_frequencies():
    geom, betas = _geom(), [0.3, 2.0]
    ctx = hams_b200.Context(geom, 15.0, rho=1025.0, g=9.81, batch_lanes=3)
    waves = [ctx.wave(v) for v in (0.4, 0.8, 1.2, 1.6)]
    single = [ctx.solve_frequency(w, betas) for w in waves]
    batch = ctx.solve_batch(waves, betas)
    for k, one in enumerate(single):
        assert all(np.array_equal(a, b[k]) for a, b in zip(one, batch))
    ctx.close()


def test_field_points_at_distances_of_their_own():
    """2,000 points, every distance to a panel another one: together and in parts that number the few
    distances of a branch in one table.  The influences have the same bits, the products sum 360 terms."""
    geom = hams_b200.prepare_geometry(*meshgen.combine([meshgen.cylinder(4.0, 6.0, 24, 10, 5)]), np.zeros((1, 3)))
    ctx = hams_b200.Context(geom, 25.0, rho=1025.0, g=9.81)
    rng, n = np.random.default_rng(4), 2000
    points = np.column_stack([rng.uniform(-25.0, 25.0, n), rng.uniform(-25.0, 25.0, n), -rng.uniform(7.0, 24.0, n)])
    wave = ctx.wave(1.0)

    def potentials(p):
        ctx.set_field_points(p)
        ctx.solve_frequency(wave, [0.4])
        return ctx.field_potentials(1)

    whole = potentials(points)
    parts = np.concatenate([potentials(points[k:k + 100]) for k in range(0, n, 100)])
    assert np.isfinite(whole).all() and np.abs(whole - parts).max() < 1e-12 * np.abs(whole).max()
    ctx.close()
