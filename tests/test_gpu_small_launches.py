"""Traces of few rays: warps then take fewer than 32 rays at a time, which must not show in the results."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu

WARPS = 152 * 8 * 4   # resident trace warps: the group size changes at multiples of it


@pytest.fixture(scope="module")
def world():
    ctx = lib.Context(0)
    scene = ctx.scene([scenes.EntitySpec("a", scenes.asteroid(2000, seed=0), smooth=False)])
    rng = np.random.default_rng(5)
    n = 20 * WARPS
    o = rng.normal(size=(n, 3))
    o *= 3000.0 / np.linalg.norm(o, axis=1)[:, None]
    d = rng.normal(size=(n, 3)) * 500.0 - o
    d /= np.linalg.norm(d, axis=1)[:, None]
    rays = lib.make_rays(o.astype(np.float32), d.astype(np.float32))
    yield scene, rays, scene.trace_closest(rays), scene.trace_any(rays)
    ctx.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, WARPS - 1, 2 * WARPS + 1, 4 * WARPS, 8 * WARPS - 1, 8 * WARPS,
                               16 * WARPS - 1, 16 * WARPS])
def test_results_do_not_depend_on_the_launch_size(world, n):
    scene, rays, hits, occluded = world
    assert (hits["prim"] != lib.CRT_MISS).any() and (hits["prim"] == lib.CRT_MISS).any()
    assert np.array_equal(scene.trace_closest(rays[:n]), hits[:n])
    assert np.array_equal(scene.trace_any(rays[:n]), occluded[:n])
