"""Large sun grids around a body that covers little of them take two groups of rays a grab: same sums."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("grid", [1537, 2048])   # 7.1 and 12.6 M rays, a ragged and a whole number of tiles
def test_a_grab_of_two_groups_changes_nothing(ctx, grid):
    q = scenes.random_quaternions(3, 4)
    sun = np.array([0.3, 0.5, 0.8])
    scene = ctx.scene(scenes.spacecraft())
    force, torque, facets = scene.srp(sun, q, grid, num_bounces=1, facet_power=True)
    for k in range(3):   # an attitude alone: too few rays for more than a group a grab
        f, t, p = scene.srp(sun, q[k:k + 1], grid, num_bounces=1, facet_power=True)
        assert np.array_equal(f[0], force[k]) and np.array_equal(t[0], torque[k])
        assert np.allclose(p[0], facets[k], rtol=1e-9, atol=0.0)   # sums of up to millions of rays, any order
    assert np.abs(force).max() > 0
