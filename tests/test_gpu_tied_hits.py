"""Hits at equal distances, at -0 beside +0 and at infinity: the triangle that is reported, and its distance
to the last bit, do not depend on a ray's neighbours or on the size of the launch."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


def vertices():
    """Rays that start at the vertices of a closed mesh, 32 of a kind at each.  Every triangle comes with each
    of its vertices first, so that a ray is at distance 0 from six triangles, -0 from those it leaves by the back."""
    m = scenes.asteroid(2_000, seed=0)
    f = np.concatenate([np.roll(m.faces, k, axis=1) for k in range(3)])
    rng = np.random.default_rng(2)
    at = np.repeat(np.arange(len(m.vertices)), 96)
    d = np.abs(rng.normal(size=(len(at), 3))) * np.repeat(rng.choice([-1.0, 1.0], (len(at) // 32, 3)), 32, axis=0)
    d /= np.linalg.norm(d, axis=1)[:, None]
    return scenes.Mesh(m.vertices, f), lib.make_rays(m.vertices[at].astype(np.float32), d.astype(np.float32))


def slivers():
    """Triangles in layers of z, each with an edge along (1, 1, 0) but for its last bits, and a ray in that
    direction through each: some meet a triangle whose n . d is exactly zero, at t = +inf."""
    n = 20_000
    rng = np.random.default_rng(0)
    d = np.tile(np.array([1, 1, 0], np.float32), (n, 1))
    p0 = np.concatenate([rng.uniform(1, 2, (n, 2)), 5e-5 * np.arange(n)[:, None]], 1).astype(np.float32)
    p1 = (p0 + rng.uniform(0.1, 0.5, (n, 1)) * d).astype(np.float32)
    p1[:, 0] += (rng.integers(-2, 3, n) * 1.2e-7).astype(np.float32)
    p2 = p0 + rng.normal(size=(n, 1)) * 0.3 * d
    p2[:, 0] += rng.normal(size=n) * 4e-5
    p2[:, 2] += rng.uniform(1e-5, 4e-5, n)
    p2 = p2.astype(np.float32)
    o = (p0 + rng.uniform(0, 0.9, (n, 1)) * (p2 - p0) - d * rng.uniform(1.5, 2.5, (n, 1))).astype(np.float32)
    o[:, 0] += (rng.integers(-2, 3, n) * 6e-8).astype(np.float32)
    rays = lib.make_rays(np.tile(o, (5, 1)), np.tile(d, (5, 1)))
    rays["tmax"] = np.inf
    v = np.stack([p0, p1, p2], 1).reshape(-1, 3)
    return scenes.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(-1, 3)), rays


@pytest.mark.parametrize("kind", [vertices, slivers])
def test_hits_do_not_depend_on_the_company(kind):
    mesh, rays = kind()
    n = len(rays)
    assert n > 80_000
    rng = np.random.default_rng(4)
    order = rng.permutation(n)
    back = np.argsort(order)
    strange = rays.copy()   # rays of all directions, one beside each
    d = rng.normal(size=(n, 3))
    strange["d"] = (d / np.linalg.norm(d, axis=1)[:, None]).astype(np.float32)
    beside = np.stack([rays, strange], 1).ravel()
    ctx = lib.Context(0)
    try:
        sc = ctx.scene([scenes.EntitySpec("m", mesh, smooth=False)])

        def closest(r):
            h = sc.trace_closest(r)
            return np.stack([h["prim"], h["t"].view(np.uint32), h["u"].view(np.uint32), h["v"].view(np.uint32)], 1)

        alike = closest(rays)
        t = alike[:, 1].copy().view(np.float32)
        hit = alike[:, 0] != lib.CRT_MISS
        if kind is vertices:
            assert (hit & (t == 0)).mean() > 0.9 and not np.signbit(t).any()
        else:
            assert (hit & np.isinf(t)).any()
        for what, got in (("shuffled", closest(rays[order])[back]), ("beside others", closest(beside)[::2]),
                          ("few", np.concatenate([closest(rays[k:k + 20_000]) for k in range(0, n, 20_000)]))):
            np.testing.assert_array_equal(got, alike, err_msg=what)
        occluded = sc.trace_any(rays)
        np.testing.assert_array_equal(occluded != 0, hit)
        np.testing.assert_array_equal(sc.trace_any(rays[order])[back], occluded)
        np.testing.assert_array_equal(sc.trace_any(beside)[::2], occluded)
        np.testing.assert_array_equal(np.concatenate([sc.trace_any(rays[k:k + 20_000]) for k in range(0, n, 20_000)]), occluded)
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [20_000, 96_000])   # eight lanes per ray; a lane per ray and dealt triangles
@pytest.mark.parametrize("alike", [True, False])
def test_ranges_that_end_at_minus_zero(n, alike):
    """[0, -0] and [-0, -0] hold t = 0 as [0, 0] does."""
    mesh, rays = vertices()
    rays = rays[:n] if alike else rays[np.random.default_rng(4).permutation(len(rays))[:n]]
    rays["tmax"] = 0.0
    ctx = lib.Context(0)
    try:
        sc = ctx.scene([scenes.EntitySpec("m", mesh, smooth=False)])
        hits, occluded = sc.trace_closest(rays), sc.trace_any(rays)
        assert (hits["prim"] != lib.CRT_MISS).mean() > 0.9
        for tmin in (0.0, -0.0):
            rays["tmin"], rays["tmax"] = tmin, -0.0
            np.testing.assert_array_equal(sc.trace_closest(rays), hits)
            np.testing.assert_array_equal(sc.trace_any(rays), occluded)
    finally:
        ctx.close()
