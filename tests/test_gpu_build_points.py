"""Bodies whose FP32 vertices coincide (a small body far from the origin): every area and every cost of the
8-wide collapse is zero, so its nodes keep two children and there are more of them than in any other tree."""
import numpy as np
import oracle
import pytest
from helpers import TriIndex, check_hits

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


def point(n, at=(5.0, 6.0, 7.0)):
    v = np.tile(np.asarray(at, np.float32), (3 * n, 1))
    return scenes.EntitySpec("p", scenes.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(-1, 3)))


# 32: 15 nodes of more than three triangles, 1000: 487 (a full tree has fewer than n / 3); 3000 and 100 000: with
# levels of tasks before the subtrees
@pytest.mark.parametrize("n", [9, 12, 32, 33, 1000, 3000, 100_000])
@pytest.mark.parametrize("sah", [True, False])
@pytest.mark.parametrize("beside", [False, True])
def test_scene_builds_and_answers(n, sah, beside):
    ents = [point(n)] + ([scenes.EntitySpec("a", scenes.asteroid(2_000, seed=3), smooth=False)] if beside else [])
    ctx = lib.Context(0)
    ctx.set_tuning(build_sah=sah)
    try:
        sc = ctx.scene(ents)
        st = sc.stats()
        total = n + (2_000 if beside else 0)
        assert st["n_tris"] == total and st["n_nodes"] <= total
        if n >= 32 and not beside:   # the case is there: more nodes than the first array has
            assert st["n_nodes"] > n // 3 + 2
        rng = np.random.default_rng(n)
        m = 40_000
        o = rng.normal(size=(m, 3))
        o *= 3000.0 / np.linalg.norm(o, axis=1)[:, None]
        d = rng.normal(size=(m, 3)) * 500.0 * beside + (5.0, 6.0, 7.0) - o
        d /= np.linalg.norm(d, axis=1)[:, None]
        r64 = np.zeros((m, 8))
        r64[:, 0:3], r64[:, 3:6] = o.astype(np.float32), d.astype(np.float32)
        r64[:, 7] = np.finfo(np.float64).max
        for k in (m, 5_000):   # a lane per ray, eight lanes per ray
            h = sc.trace_closest(lib.make_rays(r64[:k, 0:3].astype(np.float32), r64[:k, 3:6].astype(np.float32)))
            prim = np.where(h["prim"] == lib.CRT_MISS, -1, h["prim"].astype(np.int64))
            assert ((prim < 0) | (prim >= n)).all()   # a triangle without area is not hit
            if not beside:
                assert (prim < 0).all()
            elif k == 5_000:
                orc = oracle.Scene(ents[1:])   # the body beside it alone
                prim_o, t_o, _, _ = orc.trace_closest(r64[:k])
                check_hits(TriIndex(orc.tris()), r64[:k], np.where(prim < 0, -1, prim - n), h["t"], prim_o, t_o,
                           what=f"beside {n}")
        other = ctx.scene([scenes.EntitySpec("b", scenes.asteroid(500, seed=1), smooth=False)])   # the context goes on
        assert other.stats()["n_tris"] == 500
    finally:
        ctx.close()
