"""Box tables (per-width box sums, one trilinear lookup per box): frames read
them once they pay for their build, so the first small frames of a view read
the SAT and later ones the tables; all of them are the same bits."""
import numpy as np
import pytest

import oracle
from cpp_volume_rendering_gb300 import abi, scene
from tests.test_gpu_parity import compare

pytestmark = pytest.mark.gpu

N = 44
SIDE = 12     # 144 pixels a frame
FRAMES = 24   # 3456 pixels in all, above 4e-4 of the at most 8 M cells of the tables below


@pytest.mark.parametrize("direction,radii,angle,interval,shape", [
    ((0.9, 0.3, 0.2), (2, 6, 16), None, 2.0, (N, N, N)),
    ((-0.2, 0.85, 0.3), (2, 6, 16), None, 2.0, (41, 44, 37)),
    ((0.25, -0.3, -0.9), (1, 3), None, 1.0, (44, 33, 40)),
    ((-0.8, -0.4, 0.3), (2.5, 7.5), 0.05, 3.0, (37, 41, 44)),
])
@pytest.mark.parametrize("compact,walk", [(1, 1), (1, 0), (0, 1)])
def test_box_tables_equal_the_sat(ctx, direction, radii, angle, interval, shape, compact, walk):
    wl = scene.workload("extinction", n=N, image=SIDE)
    wl.volume = np.ascontiguousarray(wl.volume[:shape[0], :shape[1], :shape[2]])
    wl.params = scene.ext_params(scene.default_step(wl.spacing), wl.diagonal, ao_radii=radii, shadow_type=1,
                                 interval=interval)
    if angle is not None:
        wl.params.sdw_cone_angle_rad = angle
    f, u, r = scene.light_frame(direction)
    wl.light = scene.light(abi.LIGHT_DIRECTIONAL, position=tuple(130.0 * np.array(f)), forward=f, up=u, right=r)
    scene.prepare(ctx, wl)
    abi.check(ctx.lib.cvr_set_compact_sat(ctx.h, compact), ctx.h)
    abi.check(ctx.lib.cvr_set_walk_tables(ctx.h, walk), ctx.h)
    try:
        first, st = ctx.render(wl.method, wl.cam, wl.light, wl.params, SIDE, SIDE)
        for k in range(FRAMES):
            img, sk = ctx.render(wl.method, wl.cam, wl.light, wl.params, SIDE, SIDE)
            assert np.array_equal(img, first), k
            assert (sk.samples, sk.shaded_samples, sk.aux_fetches) == (st.samples, st.shaded_samples, st.aux_fetches)
        # a new transfer function of the same shape: other sums, other tables
        tf = scene.TransferFunction(rgb=wl.tf.rgb, alpha=[(0.0, 0), (0.1, 80), (0.3, 160), (0.8, 255)])
        ctx.set_transfer_function(tf)
        ctx.build_sat(tf.ext_per_value(wl.dtype))
        a, _ = ctx.render(wl.method, wl.cam, wl.light, wl.params, 96, 96)
    finally:
        abi.check(ctx.lib.cvr_set_compact_sat(ctx.h, 1), ctx.h)
        abi.check(ctx.lib.cvr_set_walk_tables(ctx.h, 1), ctx.h)
    wl.tf = tf
    orc = oracle.Oracle()
    oracle.prepare(orc, wl)
    ref, _, _ = orc.render(wl.method, wl.cam, wl.light, wl.params, 96, 96, precision=64)
    compare(a, ref, f"box tables, light {direction}")


def test_box_tables_follow_the_light(ctx):
    """Lights that share a walk axis add their widths to one set of tables;
    another axis, and the way back, start it over: the images do not depend on
    what was rendered before."""
    wl = scene.workload("extinction", n=40, image=96)
    scene.prepare(ctx, wl)
    lights = []
    for d in ((0.2, 0.9, 0.1), (0.45, 0.8, -0.3), (0.9, 0.2, 0.2), (-0.3, -0.9, 0.3), (0.2, 0.9, 0.1)):
        f, u, r = scene.light_frame(d)
        lights.append(scene.light(abi.LIGHT_DIRECTIONAL, position=tuple(120.0 * np.array(f)), forward=f, up=u, right=r))
    after = [ctx.render(wl.method, wl.cam, lt, wl.params, 96, 96)[0] for lt in lights]
    for lt, img in zip(lights, after):
        fresh = scene.Context(0)
        try:
            scene.prepare(fresh, wl)
            alone, _ = fresh.render(wl.method, wl.cam, lt, wl.params, 96, 96)
        finally:
            fresh.close()
        assert np.array_equal(alone, img)
