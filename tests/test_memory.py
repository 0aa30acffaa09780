"""What the context does when the device has no room, on a fake CUDA runtime
(no GPU): optional tables and copies are done without, and nothing is read
that was not made."""
import ctypes as C

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
        ctx.resize(280 << 30, 1 << 20)  # no 1.2 MB for the quads in one piece
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


def extinction(ctx, n=128, image=256, light=abi.LIGHT_DIRECTIONAL):
    wl = scene.workload("extinction", n=n, image=image)
    scene.prepare(ctx, wl)
    return lambda: ctx.render(wl.method, wl.cam, wl.light, wl.params, image, image)


def test_tables_and_lists_are_given_back(fake):
    """A volume that has no room beside the box tables and sample lists of the
    one before gets theirs; the next frame makes its own again."""
    ctx = fakegpu.Context(fake, 4 << 30)
    try:
        frame = extinction(ctx)
        frame()
        assert ctx.launches("k_box_tables") and ctx.launches("k_collect")
        held = fake.fake_used()
        assert held > 600 << 20
        ctx.resize(held + (200 << 20))
        ctx.set_volume(np.zeros((480, 1024, 1024), np.uint8))  # 480 MB
        assert fake.fake_used() < held
        ctx.resize(4 << 30)
        frame = extinction(ctx)
        frame()
        assert ctx.launches("k_box_tables") and ctx.launches("k_collect")
    finally:
        ctx.close()


def test_spare_buffers_leave_half(fake):
    """Lists and copies that would take more than half of what is free are not
    made: the direct marchers on the plain array."""
    ctx = fakegpu.Context(fake)
    try:
        wl = scene.workload("ground_truth", n=64, image=512)
        scene.prepare(ctx, wl)
        lists = 24 * 8192 * 256 * 31  # 8192 warps of 30 chunks of records, and the chunks' numbers
        ctx.resize(fake.fake_used() + 2 * lists - (200 << 20))
        ctx.render(wl.method, wl.cam, wl.light, wl.params, 512, 512)
        assert ctx.launches("k_collect") == 0 and ctx.launches("k_march_gt") == 1
        assert ctx.launches("k_quad_volume") == 1  # 1.2 MB
        assert fake.fake_refused() == 0
        ctx.resize(fake.fake_used() + 4 * lists)
        ctx.render(wl.method, wl.cam, wl.light, wl.params, 512, 512)
        assert ctx.launches("k_collect") == 1
    finally:
        ctx.close()


def test_failed_batch_keeps_the_current_volume(fake):
    ctx = fakegpu.Context(fake)
    try:
        vols = [scene.synth_blobs(24, 24, 24, abi.CVR_U8, 8, seed=7 + k) for k in range(2)]
        scene.prepare_batch_volumes(ctx, vols, pyramid=False)
        b = scene.batch_jobs(vols, n_views=1, lights=scene.BATCH_LIGHTS[:1], image=32, methods=(abi.EXTINCTION,),
                             out_ptrs=[1 << 20] * 2)
        bh = C.c_void_p()
        fake.fake_mute(1)
        try:
            assert fake.cvr_batch_create(ctx.h, (abi.Job * 2)(*b.jobs), 2, C.byref(bh)) == abi.CVR_ERR_CUDA
        finally:
            fake.fake_mute(0)
        assert fake.cvr_current_volume(ctx.h) == 0 and not bh
    finally:
        ctx.close()
