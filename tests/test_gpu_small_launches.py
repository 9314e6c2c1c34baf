"""Traces of few rays take eight lanes per ray and fewer rays per warp, which must not show in the results."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[2_000, 40_000])   # the second: deep enough for the larger limit
def world(request):
    ctx = lib.Context(0)
    scene = ctx.scene([scenes.EntitySpec("a", scenes.asteroid(request.param, seed=0), smooth=False)])
    rng = np.random.default_rng(5)
    n = 100_000
    o = rng.normal(size=(n, 3))
    o *= 3000.0 / np.linalg.norm(o, axis=1)[:, None]
    d = rng.normal(size=(n, 3)) * 500.0 - o
    d /= np.linalg.norm(d, axis=1)[:, None]
    rays = lib.make_rays(o.astype(np.float32), d.astype(np.float32))
    yield scene, rays, scene.trace_closest(rays), scene.trace_any(rays)
    ctx.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 33, 255, 3_647, 3_649, 7_297, 14_593, 39_999, 40_000, 40_001, 80_000,
                               80_001])
def test_results_do_not_depend_on_the_launch_size(world, n):
    scene, rays, hits, occluded = world
    assert (hits["prim"] != lib.CRT_MISS).any() and (hits["prim"] == lib.CRT_MISS).any()
    assert np.array_equal(scene.trace_closest(rays[:n]), hits[:n])
    assert np.array_equal(scene.trace_any(rays[:n]), occluded[:n])


@pytest.mark.parametrize("n", [3, 500, 40_000])
def test_ranges_and_skips_of_few_rays(world, n):
    """t ranges cut short, or beginning past the hit: the same answers as in a large launch."""
    scene, rays, hits, _ = world
    cut = rays.copy()
    cut["tmax"] = np.where(hits["prim"] != lib.CRT_MISS, hits["t"] * np.where(np.arange(len(rays)) % 2, 0.999, 1.0), 1.0)
    late = rays.copy()
    late["tmin"] = np.where(hits["prim"] != lib.CRT_MISS, np.nextafter(hits["t"], np.float32(np.inf)), 0.0)
    for r in (cut, late):
        assert np.array_equal(scene.trace_closest(r[:n]), scene.trace_closest(r)[:n])
        assert np.array_equal(scene.trace_any(r[:n]), scene.trace_any(r)[:n])
