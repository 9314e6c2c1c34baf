"""Incoherent rays have their triangles dealt to the warp, which must not show in the results."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu

N = 100_003   # past the launches of eight lanes per ray, and not a multiple of a warp


@pytest.fixture(scope="module", params=["asteroid", "doubled", "fan"])
def world(request):
    ctx = lib.Context(0)
    spec = scenes.EntitySpec("a", scenes.asteroid(3_000, seed=0), smooth=False)
    if request.param == "asteroid":
        specs = [spec]
    elif request.param == "doubled":   # every triangle twice: of equal distances the same one has to win
        specs = [spec, scenes.EntitySpec("b", scenes.asteroid(3_000, seed=0), smooth=False)]
    else:   # many overlapping large triangles: leaves that every ray meets
        class Fan:
            def soup(self):
                rng = np.random.default_rng(3)
                return rng.normal(size=(1_200, 9)) * 1500.0
        specs = [scenes.EntitySpec("f", Fan())]
    yield ctx.scene(specs)
    ctx.close()


def make(order):
    rng = np.random.default_rng(9)
    o = rng.normal(size=(N, 3))
    o *= 3000.0 / np.linalg.norm(o, axis=1)[:, None]
    d = rng.normal(size=(N, 3)) * 500.0 - o
    if order == "camera":
        o[:] = (4000.0, 300.0, 200.0)
        i = np.arange(N)
        d = np.stack([np.full(N, -4000.0), (i % 320) * 8.0 - 1280.0, (i // 320) * 8.0 - 1280.0], 1)
    elif order == "mixed":   # warps of one kind beside warps of the other, and warps of both
        near = (np.arange(N) // 48) % 2 == 0
        o[near], d[near] = (0.0, 2500.0, 2500.0), (0.0, -1.0, -1.0) + 0.2 * rng.normal(size=(near.sum(), 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    return lib.make_rays(o.astype(np.float32), d.astype(np.float32))


@pytest.mark.parametrize("order", ["random", "camera", "mixed"])
@pytest.mark.parametrize("cut", [False, True])
def test_as_in_launches_of_few_rays(world, order, cut):
    rays = make(order)
    parts = [slice(k, k + 25_000) for k in range(0, N, 25_000)]   # eight lanes per ray: one ray at a time
    if cut:   # ranges that end at or before the hit, begin past it, or are empty
        h = world.trace_closest(rays)
        some = h["prim"] != lib.CRT_MISS
        t = np.where(some, h["t"], np.float32(1000.0))
        k = np.arange(N) % 4
        rays["tmax"] = np.where(k == 0, t, np.where(k == 1, np.nextafter(t, np.float32(0)), rays["tmax"]))
        rays["tmin"] = np.where(k == 2, np.nextafter(t, np.float32(np.inf)), np.where((k == 0) & ~some, np.float32(2e3), rays["tmin"]))
    hits, occluded = world.trace_closest(rays), world.trace_any(rays)
    assert (hits["prim"] != lib.CRT_MISS).any()
    assert np.array_equal(hits, np.concatenate([world.trace_closest(rays[p]) for p in parts]))
    assert np.array_equal(occluded, np.concatenate([world.trace_any(rays[p]) for p in parts]))
    assert np.array_equal(occluded != 0, hits["prim"] != lib.CRT_MISS)


@pytest.mark.parametrize("n", [28_000, 28_001, 28_033])   # from where on a scene of few triangles is traced so
def test_sizes_about_the_limit(world, n):
    rays = make("mixed")
    assert np.array_equal(world.trace_closest(rays[:n]), world.trace_closest(rays)[:n])
    assert np.array_equal(world.trace_any(rays[:n]), world.trace_any(rays)[:n])
