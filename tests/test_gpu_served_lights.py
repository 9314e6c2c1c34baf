"""Served renders whose number of lights grows from request to request: the lane's path buffers are laid out
anew, and no wave may run with the addresses of an earlier layout."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [3, 8])
def test_images_as_alone(most):
    srv = lib.Server(0, lanes=1, lane_budget_bytes=1 << 30, max_batch=8, wave_paths=1 << 16)
    try:
        sc = srv.scene([scenes.EntitySpec("a", scenes.asteroid(3_000, seed=0), (0.3, 0.2, 0.1), smooth=True)])
        cam = scenes.fov_camera(0.6, (70, 41), (0.0, 3000.0, 2500.0), (0.0, 0.0, 0.0))
        for rounds in range(2):
            for n in range(1, most + 1):
                lights = [dict(type="point", intensity=1e18, position=list(1e9 * scenes.unit_vector(k))) for k in range(n)]
                q = dict(kind="render", scene=sc, camera=cam, lights=lights, min_samples=2, max_samples=2,
                         noise_threshold=0.0, num_bounces=2, seed=n, request=0, radiance=True)
                res, (rgba, rad) = srv.wait(srv.submit(q), timeout=60.0)
                assert res["status"] == 0
                alone = sc.render(cam, lights, 2, 2, 0.0, 2, seed=n, request=0)
                np.testing.assert_array_equal(rad, alone[1], err_msg=f"{n} lights")
                np.testing.assert_array_equal(rgba, alone[0])
    finally:
        srv.close()
