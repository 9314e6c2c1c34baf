"""Scene builds around the sizes where the build changes shape: one leaf, one node, a treelet's seven
leaves, a segment, the warp and block limits of its kernels; and geometry without a usable split."""
import numpy as np
import oracle
import pytest
from helpers import TriIndex, check_hits

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


def soup(kind, n):
    rng = np.random.default_rng(n)
    if kind == "random":
        p = rng.uniform(-10, 10, (n, 1, 3)) + rng.normal(size=(n, 3, 3))
    elif kind == "flat":      # one plane: no extent along an axis
        p = rng.uniform(-10, 10, (n, 1, 3)) + rng.normal(size=(n, 3, 3))
        p[:, :, 2] = 1.0
    else:                     # "line": centroids on one axis, sizes growing along it
        x = np.linspace(0, 1, n) ** 3
        p = np.array([[0, -1, -1], [0, 1, -1], [0, 0, 1]])[None] * (0.1 + x)[:, None, None]
        p[:, :, 0] += 20 * x[:, None]
    v = p.reshape(-1, 3).astype(np.float32)
    return scenes.Mesh(v, np.arange(3 * n, dtype=np.int32).reshape(-1, 3))


@pytest.mark.parametrize("kind,n", [("random", k) for k in (1, 2, 3, 4, 5, 6, 7, 8, 9, 33, 65, 1023, 1025, 2049, 5000)] +
                         [("flat", 700), ("flat", 3000), ("line", 600), ("line", 2500)])
@pytest.mark.parametrize("sah,treelets", [(True, 1), (False, 0)])
def test_hits_of_scenes_of_every_size(kind, n, sah, treelets):
    ents = [scenes.EntitySpec("s", soup(kind, n))]
    ctx = lib.Context(0)
    ctx.set_tuning(build_sah=sah, treelet_passes=treelets)
    try:
        sc = ctx.scene(ents)
        o = oracle.Scene(ents)
        rng = np.random.default_rng(7)
        m = 4000
        org = rng.normal(size=(m, 3))
        org *= 40.0 / np.linalg.norm(org, axis=1)[:, None]
        d = rng.uniform(-10, 10, (m, 3)) - org
        d /= np.linalg.norm(d, axis=1)[:, None]
        r64 = np.zeros((m, 8))
        r64[:, 0:3], r64[:, 3:6] = org.astype(np.float32), d.astype(np.float32)
        r64[:, 7] = np.finfo(np.float64).max
        h = sc.trace_closest(lib.make_rays(r64[:, 0:3].astype(np.float32), r64[:, 3:6].astype(np.float32)))
        prim = np.where(h["prim"] == lib.CRT_MISS, -1, h["prim"].astype(np.int64))
        prim_o, t_o, _, _ = o.trace_closest(r64)
        check_hits(TriIndex(o.tris()), r64, prim, h["t"], prim_o, t_o, what=f"{kind} {n}")
        assert sc.stats()["n_tris"] == n
    finally:
        ctx.close()
