"""Which way a frame takes (on a fake CUDA runtime): the bands of the sample
lists, the direct marchers and the box tables, at the sizes that the GPU tests
of the same images use; and those images under a memory limit (GPU)."""
import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi, scene
from tests import fakegpu
from tests.test_box_tables import FRAMES, N, SIDE
from tests.test_deferred import GAPS, gt_workload

# 93 x 61 pixels are 8 rows of 6 tiles; a row's lists take ROW bytes (24 warps
# of 16 chunks of 256 records)
IMAGE = (93, 61)
ROW = 24 * 16 * (256 * 24 + 4)
LIMITS = [(8 * ROW + 512, 1), (3 * ROW + 512, 3), (7 * ROW + 512, 2), (ROW + 512, 8), (ROW, 0), (0, 0)]


def banded_workload():
    return gt_workload((32, 32, 32), (1.0, 1.0, 1.0), IMAGE, GAPS)


def frame(ctx, wl):
    return ctx.render(wl.method, wl.cam, wl.light, wl.params, wl.width, wl.height)


@pytest.fixture
def fake():
    c = fakegpu.Context(fakegpu.load())
    yield c
    c.close()


@pytest.mark.parametrize("limit,bands", LIMITS)
def test_bands(fake, limit, bands):
    wl = banded_workload()
    scene.prepare(fake, wl)
    abi.check(fake.lib.cvr_set_cache_limit(fake.h, limit), fake.h)
    frame(fake, wl)
    assert fake.launches("k_collect") == fake.launches("k_light_gt") == fake.launches("k_resolve") == bands
    assert fake.launches("k_march_gt") == (1 if bands == 0 else 0)


@pytest.mark.gpu
@pytest.mark.parametrize("limit,bands", LIMITS)
def test_bands_give_one_image(ctx, limit, bands):
    wl = banded_workload()
    scene.prepare(ctx, wl)
    whole, sw = frame(ctx, wl)
    abi.check(ctx.lib.cvr_set_cache_limit(ctx.h, limit), ctx.h)
    try:
        img, st = frame(ctx, wl)
    finally:
        abi.check(ctx.lib.cvr_set_cache_limit(ctx.h, 2 ** 64 - 1), ctx.h)
    assert (st.samples, st.shaded_samples, st.aux_fetches) == (sw.samples, sw.shaded_samples, sw.aux_fetches)
    assert np.array_equal(img[..., 3], whole[..., 3]) and whole[..., 3].max() > 0.5
    if bands:
        assert np.array_equal(img, whole)
    else:  # the direct marcher: the light terms' sums in another kernel
        assert np.abs(img - whole).max() <= 1e-5


def test_far_cameras_and_long_rays_are_direct(fake):
    wl = gt_workload((24, 24, 24), (1.0, 1.0, 1.0), (24, 16), scene.BENCH_TF)
    scene.prepare(fake, wl)
    far = scene.camera(scene.orbit_eye(200.0 * wl.diagonal, 20.0, 30.0), fovy=0.4)
    for cam, step, size in ((far, 0.5, (48, 40)), (wl.cam, 1.0e-4, (64, 16))):
        wl.params.step_size = step
        fake.resize(280 << 30)
        fake.render(wl.method, cam, wl.light, wl.params, *size)
        assert fake.launches("k_collect") == 0 and fake.launches("k_march_gt") == 1


def box_workload(direction, radii, angle, interval, shape):
    wl = scene.workload("extinction", n=N, image=SIDE)
    wl.volume = np.ascontiguousarray(wl.volume[:shape[0], :shape[1], :shape[2]])
    wl.params = scene.ext_params(scene.default_step(wl.spacing), wl.diagonal, ao_radii=radii, shadow_type=1,
                                 interval=interval)
    if angle is not None:
        wl.params.sdw_cone_angle_rad = angle
    f, u, r = scene.light_frame(direction)
    wl.light = scene.light(abi.LIGHT_DIRECTIONAL, position=tuple(130.0 * np.array(f)), forward=f, up=u, right=r)
    return wl


@pytest.mark.parametrize("direction,radii,angle,interval,shape", [  # those of test_box_tables_equal_the_sat
    ((0.9, 0.3, 0.2), (2, 6, 16), None, 2.0, (N, N, N)),
    ((-0.2, 0.85, 0.3), (2, 6, 16), None, 2.0, (41, 44, 37)),
    ((0.25, -0.3, -0.9), (1, 3), None, 1.0, (44, 33, 40)),
    ((-0.8, -0.4, 0.3), (2.5, 7.5), 0.05, 3.0, (37, 41, 44)),
])
@pytest.mark.parametrize("compact", [0, 1])
def test_small_frames_come_to_read_box_tables(fake, direction, radii, angle, interval, shape, compact):
    wl = box_workload(direction, radii, angle, interval, shape)
    scene.prepare(fake, wl)
    abi.check(fake.lib.cvr_set_compact_sat(fake.h, compact), fake.h)
    boxes = lambda: fake.launches("k_light_box") + fake.launches("k_march_extinction_box")  # noqa: E731
    frame(fake, wl)
    assert fake.launches("k_light_ext") == 1 and boxes() == 0  # the SAT at first
    for _ in range(FRAMES):
        frame(fake, wl)
    assert boxes() > 0 and fake.launches("k_light_ext") + boxes() == FRAMES + 1
    # a memory limit below the tables: the SAT again
    abi.check(fake.lib.cvr_set_cache_limit(fake.h, 1 << 20), fake.h)
    seen = boxes()
    for _ in range(FRAMES):
        frame(fake, wl)
    assert boxes() == seen


def test_frames_say_what_they_read(fake):
    """cvr_get_frame_tables, and with it the bytes that the benchmark's roofline counts."""
    import ctypes as C

    import bench

    def tables():
        a, b = C.c_int(-1), C.c_int(-1)
        abi.check(fake.lib.cvr_get_frame_tables(fake.h, C.byref(a), C.byref(b)), fake.h)
        return a.value, b.value

    ck = abi.check
    assert tables() == (abi.TABLES_NONE, abi.TABLES_NONE)
    wl = scene.workload("extinction", n=64, image=160)  # a directional light, three AO boxes of whole widths
    scene.prepare(fake, wl)
    frame(fake, wl)
    assert tables() == (abi.TABLES_BOX, abi.TABLES_BOX)
    ck(fake.lib.cvr_set_ray_refill(fake.h, 1), fake.h)
    frame(fake, wl)
    assert tables() == (abi.TABLES_WALK, abi.TABLES_COMPACT)
    ck(fake.lib.cvr_set_walk_tables(fake.h, 0), fake.h)
    frame(fake, wl)
    assert tables() == (abi.TABLES_COMPACT, abi.TABLES_COMPACT)
    ck(fake.lib.cvr_set_compact_sat(fake.h, 0), fake.h)
    frame(fake, wl)
    assert tables() == (abi.TABLES_SAT, abi.TABLES_SAT)
    ck(fake.lib.cvr_set_ray_refill(fake.h, 0), fake.h)
    wl.params.shadow_type = 0  # a point light: occlusion alone has box tables
    frame(fake, wl)
    assert tables() == (abi.TABLES_SAT, abi.TABLES_BOX)
    wl.params.apply_occlusion = 0
    frame(fake, wl)
    assert tables() == (abi.TABLES_SAT, abi.TABLES_NONE)

    st = abi.FrameStats(1000, 100, 100 * 53, 1.0)
    wl.params.apply_occlusion, wl.params.ao_n_shells = 1, 3
    rest = 1000 * 8 * 2 + 160 * 160 * 16
    assert bench.l1_request_bytes(wl, st, abi, (abi.TABLES_BOX, abi.TABLES_BOX)) == rest + 5300 * 32
    assert bench.l1_request_bytes(wl, st, abi, (abi.TABLES_WALK, abi.TABLES_COMPACT)) == rest + 5000 * 128 + 300 * 256
    assert bench.l1_request_bytes(wl, st, abi, (abi.TABLES_SAT, abi.TABLES_BOX)) == rest + 5000 * 512 + 300 * 32


def test_limit_frees_and_bounds(fake):
    """Limit 0: no tables, lists or copies are held or made, in slots and batches."""
    wl = scene.workload("extinction", n=64, image=128)
    scene.prepare(fake, wl)
    frame(fake, wl)
    assert fake.launches("k_box_tables") and fake.launches("k_quad_volume") and fake.launches("k_collect")
    held = fake.lib.fake_used()
    fake.select_volume(1)  # the copy of slot 0 goes too
    abi.check(fake.lib.cvr_set_cache_limit(fake.h, 0), fake.h)
    assert fake.lib.cvr_get_cache_limit(fake.h) == 0
    fake.select_volume(0)
    small = fake.lib.fake_used()
    assert small < held / 20
    fake.resize(280 << 30)
    frame(fake, wl)
    assert fake.launches("k_march_extinction") == 1
    assert not any(fake.launches(k) for k in ("k_box_tables", "k_quad_volume", "k_collect", "k_light"))
    abi.check(fake.lib.cvr_set_cache_limit(fake.h, 2 ** 64 - 1), fake.h)
    frame(fake, wl)
    assert fake.launches("k_box_tables") and fake.launches("k_quad_volume") and fake.launches("k_collect")
