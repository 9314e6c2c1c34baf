"""Batches over scenes either side of the sizes at which traces take other kernels: as the requests alone."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(0,), (0, 2), (1, 2), (2, 3), (0, 1, 2, 3)])
@pytest.mark.parametrize("wave_paths", [1 << 16, 1 << 23])   # several waves (graphs), one
def test_batch_as_alone(sizes, wave_paths):
    ctx = lib.Context(0)
    try:
        ents, ccam, clights = scenes.cornell()
        scs = [ctx.scene(ents)] + [ctx.scene([scenes.EntitySpec("a", scenes.asteroid(n, seed=0), (0.3, 0.2, 0.1), rho_s=0.4,
                                                                rho_d=0.2)]) for n in (1_022, 1_024, 40_000)]
        sun = [dict(type="point", intensity=1e18, position=[6e8, 8e8, 1e8])]
        reqs, alone = [], []
        for k in sizes:
            cam = dict(ccam, resolution=[150, 131]) if k == 0 else scenes.fov_camera(0.6, (150, 131), (0.0, 3000.0, 2500.0),
                                                                                     (0.0, 0.0, 0.0))
            li = clights if k == 0 else sun
            reqs.append(dict(kind="render", scene=scs[k], camera=cam, lights=li, min_samples=5, max_samples=5,
                             noise_threshold=0.0, num_bounces=3, seed=k, request=k, radiance=True))
            alone.append(scs[k].render(cam, li, 5, 5, 0.0, 3, seed=k, request=k))
            if k:
                q = dict(sun_dir=[0.3, 0.5, 0.8], quaternions=scenes.random_quaternions(2, seed=k), grid=200, num_bounces=2)
                reqs.append(dict(q, kind="srp", scene=scs[k]))
                alone.append(scs[k].srp(q["sun_dir"], q["quaternions"], 200, num_bounces=2)[:2])
        ctx.set_tuning(wave_paths=wave_paths)
        outs, _ = ctx.batch(reqs)
        for a, b in zip(outs, alone):
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x, y)
    finally:
        ctx.close()
