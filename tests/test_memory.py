"""What the context does when the device has no room, on a fake CUDA runtime
(no GPU): optional tables and copies are done without, and nothing is read
that was not made."""
import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi, scene
from tests import fakegpu


@pytest.fixture(scope="module")
def fake():
    return fakegpu.load()


def plain(ctx, n=64, image=96):
    wl = scene.workload("plain", n=n, image=image)
    scene.prepare(ctx, wl)
    return lambda: ctx.render(wl.method, wl.cam, wl.light, wl.params, image, image)


def test_no_room_for_the_automatic_quad_copy(fake):
    """The plain array serves, the allocation is not tried again for the same
    volume, and bricks that gave their buffer up are made again."""
    ctx = fakegpu.Context(fake)
    try:
        frame = plain(ctx)
        abi.check(fake.cvr_set_brick_size(ctx.h, 8), ctx.h)
        frame()
        assert ctx.launches("k_brick") == 1
        abi.check(fake.cvr_set_brick_size(ctx.h, 0), ctx.h)
        ctx.resize(fake.fake_used() + (1 << 18))  # the quads take 1.2 MB
        for _ in range(3):
            frame()
        assert ctx.launches("k_quad_volume") == 0 and ctx.launches("k_march_plain") == 3
        assert fake.fake_refused() == 1
        ctx.resize(280 << 30)
        abi.check(fake.cvr_set_brick_size(ctx.h, 8), ctx.h)
        frame()
        assert ctx.launches("k_brick") == 1
        # another volume is tried again
        abi.check(fake.cvr_set_brick_size(ctx.h, 0), ctx.h)
        frame = plain(ctx)
        frame()
        assert ctx.launches("k_quad_volume") == 1
    finally:
        ctx.close()
