"""Box tables of volumes so deep that their builds exceed one launch: the frame
still reads them (on a fake CUDA runtime), and is the SAT marchers' frame (GPU)."""
import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi, scene
from tests import fakegpu

SIDE = 320  # pixels that repay 16 tables of 14.8 M cells


def deep_workload(depth):
    wl = scene.workload("extinction", n=8, image=8)
    rng = np.random.default_rng(8)
    wl.volume = rng.integers(0, 256, (depth, 4, 4), dtype=np.uint8)
    wl.spacing = (1.0, 1.0, 4.0 / depth)
    # 16 shells, of half a voxel and of one: 16 tables
    wl.params = scene.ext_params(0.05, wl.diagonal, ao_radii=(0.5,) * 8 + (1.0,) * 8, shadow_type=0)
    wl.params.apply_shadow = 0
    return wl


# the last: one table's planes alone exceed a launch, so the frame reads the SAT
@pytest.mark.parametrize("depth,shells,launches", [(60000, 16, 1), (70000, 16, 2), (550000, 2, 2), (1100000, 1, 0)])
def test_deep_volumes_build_their_tables(depth, shells, launches):
    lib = fakegpu.load()
    ctx = fakegpu.Context(lib)
    try:
        wl = deep_workload(depth)
        wl.params.ao_n_shells = shells
        scene.prepare(ctx, wl)
        ctx.render(wl.method, wl.cam, wl.light, wl.params, SIDE, SIDE)
        assert ctx.launches("k_box_tables") == launches
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [60000, 70000])
def test_deep_frames_equal_the_sat(ctx, depth):
    wl = deep_workload(depth)
    scene.prepare(ctx, wl)
    img = {}
    for refill in (1, 0):  # the refill marcher reads the SAT
        abi.check(ctx.lib.cvr_set_ray_refill(ctx.h, refill), ctx.h)
        img[refill], _ = ctx.render(wl.method, wl.cam, wl.light, wl.params, SIDE, SIDE)
    abi.check(ctx.lib.cvr_set_ray_refill(ctx.h, 0), ctx.h)
    assert np.isfinite(img[1]).all() and img[1][..., 3].max() > 0.0
    assert np.abs(img[0] - img[1]).max() <= 1e-5
