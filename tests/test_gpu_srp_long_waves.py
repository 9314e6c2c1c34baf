"""Mixed batches with waves of more than 2^31 sun rays allowed (crt_tuning.wave_paths): the sums of crt_srp."""
import numpy as np
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


def test_more_items_than_a_wave_can_number():
    ctx = lib.Context(0)
    try:
        # 33,640,448 items an attitude, just above a power of two: the divisor's multiplier is largest there
        q = dict(sun_dir=[0.3, 0.5, 0.8], quaternions=scenes.random_quaternions(66, seed=4), grid=5800, num_bounces=0)
        sc = ctx.scene(scenes.spacecraft(bus_cell=0.25, panel_cell=0.2, dish_rings=16, dish_segments=16))
        f, t, _ = sc.srp(q["sun_dir"], q["quaternions"], q["grid"], num_bounces=0)
        assert (np.abs(f).max(axis=1) > 0).all()
        ctx.set_tuning(wave_paths=3_000_000_000)
        (out,), stats = ctx.batch([dict(q, kind="srp", scene=sc)])
        np.testing.assert_array_equal(out[0], f)
        np.testing.assert_array_equal(out[1], t)
    finally:
        ctx.close()
