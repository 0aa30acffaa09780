"""Deferred frames over every storage, voxel type and tile size: collect and
resolve number a frame's samples each for themselves, so a step that they
rounded apart would give a ray another's light terms.  The ray-refill marcher
shades along each ray: the same samples, the same image but for the rounding of
the light terms' sums in another kernel."""
import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi, scene

pytestmark = pytest.mark.gpu

STORAGES = {  # brick edge, layout, sampling flags
    "plain": (0, abi.LAYOUT_PLAIN, 0),
    "quads": (0, abi.LAYOUT_QUADS, 0),
    "bricks": (8, abi.LAYOUT_PLAIN, 0),
    "texture": (0, abi.LAYOUT_PLAIN, abi.SAMPLING_TEX_VOLUME),
}
SHAPE = (31, 40, 37)


def forms_workload(name, dtype, image):
    wl = scene.workload(name, n=40, image=image[0])
    wl.volume = np.ascontiguousarray(scene.synth_blobs(40, 40, 40, dtype, 24, seed=3300, noise_max=20.0)
                                     [:SHAPE[0], :SHAPE[1], :SHAPE[2]])
    wl.width, wl.height = image
    if name == "ground_truth":
        wl.params = scene.gt_params(0.4, wl.diagonal, occ_distance=6.0, light_step=1.0, gap=1.0)
        wl.gt_spec = (2, 90.0, 1, 0.0, 1)
        wl.gt = scene.gt_vectors(*wl.gt_spec)
    elif name == "extinction":  # a point light: cones of their own for every sample
        wl.params = scene.ext_params(0.4, wl.diagonal, ao_radii=(1, 2.25), shadow_type=0)
        wl.light = scene.light(abi.LIGHT_POINT, position=(70.0, 50.0, 20.0))
    return wl


@pytest.mark.parametrize("storage", list(STORAGES))
@pytest.mark.parametrize("dtype", [abi.CVR_U8, abi.CVR_U16])
@pytest.mark.parametrize("name", ["ground_truth", "extinction", "cone"])
def test_deferred_forms(ctx, name, dtype, storage):
    brick, layout, sampling = STORAGES[storage]
    wl = forms_workload(name, dtype, (93, 61))
    scene.prepare(ctx, wl)
    ck = abi.check
    try:
        ck(ctx.lib.cvr_set_brick_size(ctx.h, brick), ctx.h)
        ck(ctx.lib.cvr_set_volume_layout(ctx.h, layout), ctx.h)
        ctx.set_sampling(sampling)
        ck(ctx.lib.cvr_set_ray_refill(ctx.h, 1), ctx.h)
        ref, sr = ctx.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height)
        ck(ctx.lib.cvr_set_ray_refill(ctx.h, 0), ctx.h)
        assert ref[..., 3].max() > 0.5
        for tile in ((8, 8), (16, 8), (32, 8)):  # CTAs of 64, 128 and 256 threads
            ck(ctx.lib.cvr_set_tuning(ctx.h, *tile, 0), ctx.h)
            img, st = ctx.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height)
            assert (st.samples, st.shaded_samples, st.aux_fetches) == (sr.samples, sr.shaded_samples, sr.aux_fetches), tile
            assert np.array_equal(img[..., 3], ref[..., 3]), tile  # opacities: the same bits
            assert np.abs(img - ref).max() <= 1e-5, tile
    finally:
        ck(ctx.lib.cvr_set_ray_refill(ctx.h, 0), ctx.h)
        ck(ctx.lib.cvr_set_tuning(ctx.h, 16, 8, 0), ctx.h)
        ck(ctx.lib.cvr_set_brick_size(ctx.h, 0), ctx.h)
        ck(ctx.lib.cvr_set_volume_layout(ctx.h, abi.LAYOUT_PLAIN), ctx.h)
        ctx.set_sampling(abi.SAMPLING_TEX_FEATURES)
