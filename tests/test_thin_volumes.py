"""Ground truth of volumes one voxel thick: light rays that run inside the one
layer, at its middle (where both taps are the layer) and a hundredth of a voxel
off it."""
import numpy as np
import pytest

import oracle
from cpp_volume_rendering_gb300 import abi, scene
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu

N = 32
ALONG = {0: (0.0, 1.0, 0.0), 1: (1.0, 0.0, 0.0), 2: (1.0, 0.0, 0.0)}  # a direction in the layer


@pytest.mark.parametrize("layout", [abi.LAYOUT_PLAIN, abi.LAYOUT_QUADS])
@pytest.mark.parametrize("dtype", [abi.CVR_U8, abi.CVR_U16])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_one_voxel_thick(ctx, axis, dtype, layout):
    shape = [N, N, N]
    shape[2 - axis] = 1
    wl = scene.workload("ground_truth", n=N, image=33)
    wl.volume = np.ascontiguousarray(scene.synth_blobs(N, N, N, dtype, 24, seed=3100, noise_max=20.0)
                                     [:shape[0], :shape[1], :shape[2]])
    # an eye in the layer's plane (or just off it): the middle row or column of the image looks along it
    eye = 90.0 * np.array({0: (0.0, 0.0, 1.0), 1: (0.0, 0.0, 1.0), 2: (1.0, 0.0, 0.0)}[axis])
    fwd, up, right = scene.light_frame(ALONG[axis])
    wl.light = scene.light(abi.LIGHT_DIRECTIONAL, position=tuple(60.0 * np.array(fwd)), forward=fwd, up=up, right=right)
    wl.params = scene.gt_params(0.25, wl.diagonal, occ_distance=20.0, light_step=1.0, gap=1.0, shadow_type=2)
    wl.gt_spec = (1, 0.0, 1, 0.0, 1)  # one light ray straight along each cone's axis
    wl.gt = scene.gt_vectors(*wl.gt_spec)
    for off in (0.0, 0.01):
        at = eye.copy()
        at[axis] += off
        centre = np.zeros(3)
        centre[axis] = off
        wl.cam = scene.camera(tuple(at), center=tuple(centre), fovy=20.0)
        scene.prepare(ctx, wl)
        abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, layout), ctx.h)
        try:
            img, _ = ctx.render(wl.method, wl.cam, wl.light, wl.params, 33, 33)
        finally:
            abi.check(ctx.lib.cvr_set_volume_layout(ctx.h, abi.LAYOUT_PLAIN), ctx.h)
        orc = oracle.Oracle()
        oracle.prepare(orc, wl)
        ref, _, _ = orc.render(wl.method, wl.cam, wl.light, wl.params, 33, 33, precision=64)
        assert ref[..., 3].max() > 0.0
        compare(img, ref, f"axis {axis}, {off} off the layer's middle")
