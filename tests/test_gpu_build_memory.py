"""What a context holds between builds: the binned-SAH build keeps no more than the radix-tree build."""
import pytest

from crt_gb300 import lib, scenes

pytestmark = pytest.mark.gpu


def held(ents, sah):
    import torch
    ctx = lib.Context(0)
    try:
        ctx.set_tuning(build_sah=sah)
        free = torch.cuda.mem_get_info()[0]
        ctx.scene(ents).close()
        return free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()


def test_sah_builds_hold_no_temporaries():
    ents = [scenes.EntitySpec("a", scenes.asteroid(1_000_000, seed=0), smooth=False)]
    held(ents, True)   # the process's first build (kernels loaded)
    radix, sah = held(ents, False), held(ents, True)
    assert radix > 300 << 20   # about 320 bytes per triangle, and a quarter more
    assert sah <= radix + (4 << 20)   # (allocations come in 2 MB)
