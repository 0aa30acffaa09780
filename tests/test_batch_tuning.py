"""A batch renders with the context's tuning at its creation: frames that other
volume layouts render afterwards leave the copies its jobs read alone."""
import ctypes as C

import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi, scene
from tests.devmem import DeviceMemory
from tests.test_batch import small_network

pytestmark = pytest.mark.gpu


# the second volume's bricks of 32 take more room than its quads
@pytest.mark.parametrize("shape,edges", [((64, 64, 64), (8,)), ((64, 64, 4), (8, 32))])
@pytest.mark.parametrize("layout", [abi.LAYOUT_PLAIN, abi.LAYOUT_QUADS])
def test_batch_keeps_its_copies(shape, edges, layout):
    ctx = scene.Context(0)
    mem = DeviceMemory()
    try:
        vols = [scene.synth_blobs(*shape, abi.CVR_U8, 12, seed=6100)]
        scene.prepare_batch_volumes(ctx, vols)
        small_network(ctx)
        abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, layout), ctx.h)
        W = H = 64
        outs = [mem.alloc(W * H * 16, fill=0) for _ in range(4)]
        b = scene.batch_jobs(vols, n_views=2, lights=scene.BATCH_LIGHTS[:1], image=W, out_ptrs=outs)
        bh = C.c_void_p()
        abi.check(ctx.lib.cvr_batch_create(ctx.h, (abi.Job * 4)(*b.jobs), 4, C.byref(bh)), ctx.h)

        def run():
            abi.check(ctx.lib.cvr_batch_run(bh), ctx.h)
            abi.check(ctx.lib.cvr_sync(ctx.h), ctx.h)
            return [mem.download(p, (H, W, 4)) for p in outs]

        try:
            first = run()
            abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, abi.LAYOUT_PLAIN), ctx.h)
            for edge in edges:
                abi.check(ctx.lib.cvr_set_brick_size(ctx.h, edge), ctx.h)
                j = b.jobs[0]
                ctx.render(j.method, j.camera, j.light, b.params[0], W, H)
                for k, img in enumerate(run()):
                    assert np.array_equal(img, first[k]), (edge, k)
        finally:
            ctx.lib.cvr_batch_destroy(bh)
    finally:
        mem.close()
        ctx.close()
