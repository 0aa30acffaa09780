"""Deferred shading (collect, light, resolve): the image and the counters of
the per-ray marchers, over ragged images, several bands of the record lists,
rays that shade nothing and transfer functions with transparent ranges."""
import numpy as np
import pytest

import oracle
from cpp_volume_rendering_gb300 import abi, scene
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu

GAPS = scene.TransferFunction(  # opaque shells between transparent ranges
    rgb=scene.BENCH_TF.rgb, alpha=[(0.0, 0), (0.0, 40), (0.6, 60), (0.0, 80), (0.0, 120), (0.9, 160), (0.9, 255)])


def gt_workload(shape, spacing, image, tf):
    wl = scene.workload("ground_truth", n=32, image=32)
    wl.volume = np.ascontiguousarray(scene.synth_blobs(32, 32, 32, abi.CVR_U8, 32, seed=3000, noise_max=20.0)
                                     [:shape[0], :shape[1], :shape[2]])
    wl.spacing, wl.tf = spacing, tf
    wl.width, wl.height = image
    wl.params = scene.gt_params(scene.default_step(spacing), wl.diagonal, occ_distance=4.0, light_step=1.0, gap=1.0)
    wl.gt_spec = (3, 90.0, 2, 1.0, 1)
    wl.gt = scene.gt_vectors(*wl.gt_spec)
    return wl


@pytest.mark.parametrize("shape,spacing,image,quads,tf", [
    ((32, 32, 32), (1.0, 1.0, 1.0), (41, 33), 0, scene.BENCH_TF),
    ((17, 32, 9), (1.0, 0.7, 1.6), (29, 50), 1, GAPS),
    ((3, 2, 1), (4.0, 5.0, 6.0), (16, 16), 1, scene.BENCH_TF),
    ((32, 5, 30), (1.0, 1.0, 1.0), (1, 1), 0, GAPS),
])
def test_deferred_frame_matches_oracle(ctx, shape, spacing, image, quads, tf):
    wl = gt_workload(shape, spacing, image, tf)
    scene.prepare(ctx, wl)
    abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, quads), ctx.h)
    try:
        img, st = ctx.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height)
        unseen, _ = ctx.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height, stats=False)
    finally:
        abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, 0), ctx.h)
    assert np.array_equal(img, unseen)
    orc = oracle.Oracle()
    oracle.prepare(orc, wl)
    ref, _, total = orc.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height, precision=64)
    compare(img, ref, f"ground truth {shape} {image}")
    assert abs(int(st.samples) - int(total)) <= max(2, total // 2000)


def test_bands_and_the_direct_marcher(ctx):
    """Steps of a hundredth of a voxel fill the lists before the image's last
    row (several bands); steps of 1e-4 voxels leave no room for one row, and a
    camera 200 diagonals away is not deferred: the persistent ray-refill
    marcher gives the same images (the same arithmetic in another kernel)."""
    wl = gt_workload((24, 24, 24), (1.0, 1.0, 1.0), (256, 96), scene.BENCH_TF)
    scene.prepare(ctx, wl)
    far = scene.camera(scene.orbit_eye(200.0 * wl.diagonal, 20.0, 30.0), fovy=0.4)
    for cam, step, size in ((wl.cam, 0.01, (256, 96)), (wl.cam, 1.0e-4, (24, 16)), (far, 0.5, (48, 40))):
        wl.params.step_size = step
        out = {}
        for refill in (0, 1):
            abi.check(ctx.lib.cvr_set_ray_refill(ctx.h, refill), ctx.h)
            out[refill], st = ctx.render(wl.method, cam, wl.light, wl.params, *size)
            out[refill, "n"] = (st.samples, st.shaded_samples, st.aux_fetches)
        abi.check(ctx.lib.cvr_set_ray_refill(ctx.h, 0), ctx.h)
        assert out[0, "n"] == out[1, "n"]
        assert np.abs(out[0] - out[1]).max() <= 1e-5
        assert out[0][..., 3].max() > 0.0
