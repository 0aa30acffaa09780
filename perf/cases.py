"""The work a user of this framework has it do, as measurable cases.

Every case is a frame, a table rebuild followed by the frame that reads it, a
batch of frames or a run of network training, called through the C ABI
(include/cvr.h) the way a program that keeps one context per scene calls it:
prepare() is Init() (volume, tables, tuning), run() is one Update() + Redraw().
Volumes, transfer functions and views are seeded and synthetic; the sizes are
those of the benchmark's workloads and of the tests, and odd ones between them.
"""
import ctypes as C
import math

import numpy as np
import torch

from cpp_volume_rendering_gb300 import abi, scene

DEV = "cuda"

# ------------------------------------------------------------------ cases


def listed():
    return [
        # the smallest frame: a 64^3 preview, where launches and latency count
        dict(name="plain_small", kind="plain", w=64, h=64, d=64, bits=8, width=256, height=256, quads=False, tex=False),
        # the largest plain frame: 512^3 at 2048^2 on the x-y quad layout the autotuner picks for it
        dict(name="plain_large", kind="plain", w=512, h=512, d=512, bits=16, width=2048, height=2048, quads=True,
             tex=False),
        # extinction shading as benchmarked: nested shells, three AO boxes, a directional SAT shadow cone
        dict(name="extinction_directional", kind="extinction", w=256, h=256, d=256, bits=16, width=1024, height=1024,
             light="directional", shells="nested", edit=False),
        # extinction shading with the renderer's defaults (15 unit shells, point light) on an uneven scan, 16:9
        dict(name="extinction_point", kind="extinction", w=192, h=256, d=160, bits=8, width=640, height=360,
             light="point", shells="unit", edit=False),
        # the user drags a transfer-function point: new tables, SAT and frame
        dict(name="extinction_edit", kind="extinction", w=200, h=180, d=222, bits=16, width=512, height=512,
             light="directional", shells="nested", edit=True),
        # cone-traced directional occlusion and shadow as benchmarked
        dict(name="cone", kind="cone", w=256, h=256, d=256, bits=8, width=512, height=512, cache=0, edit=False,
             quads=True),
        # a transfer-function edit under the object-space light cache: new pyramid, cache and frame
        dict(name="cone_cache_edit", kind="cone", w=256, h=256, d=256, bits=8, width=1024, height=768, cache=32,
             edit=True, quads=False),
        # the ground-truth integrator as benchmarked: the most expensive frame there is
        dict(name="ground_truth", kind="ground_truth", w=256, h=256, d=256, bits=8, width=512, height=512, quads=True),
        # the learned surrogate in the ground truth's place, its inputs through the texture unit
        dict(name="surrogate", kind="surrogate", w=320, h=320, d=320, bits=8, width=720, height=720),
        # a new time step of a ragged series: upload, gradients, shaded isosurface, 2 x 2 rays per pixel
        dict(name="iso_new_volume", kind="iso", w=301, h=257, d=190, bits=16, width=641, height=361, scale="multi",
             quads=False),
        # many views of many volumes at once, both shadings
        dict(name="batch", kind="batch", side=128, views=3, lights=2, width=256, height=256),
        # training of the surrogate's network (forward, backward, Adam)
        dict(name="train", kind="train", points=131072, batch=4096, epochs=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; the cost of a frame grows with pixels x voxels along a ray."""
    kind = rng.choice(["plain", "plain", "extinction", "extinction", "extinction", "cone", "cone", "ground_truth",
                       "surrogate", "iso", "batch", "train"])
    if kind == "train":
        return dict(kind=kind, points=_log(rng, 8192, 200000), batch=128 * _log(rng, 4, 48), epochs=rng.randint(1, 4))
    if kind == "batch":
        return dict(kind=kind, side=_log(rng, 64, 160), views=rng.randint(1, 4), lights=rng.randint(1, 3),
                    width=_log(rng, 100, 300), height=_log(rng, 100, 300))
    top = {"plain": 400, "extinction": 288, "cone": 256, "ground_truth": 200, "surrogate": 320, "iso": 320}[kind]
    low = 96 if kind == "surrogate" else 48
    # an edit re-renders a view; the pixel counts stay below the listed frames'
    side = {"plain": 1500, "extinction": 900, "cone": 480, "ground_truth": 360, "surrogate": 700, "iso": 800}[kind]
    c = dict(kind=kind, w=_log(rng, low, top), h=_log(rng, low, top), d=_log(rng, low, top), bits=rng.choice([8, 16]),
             width=_log(rng, 120, side), height=_log(rng, 120, side))
    if kind == "plain":
        c.update(quads=rng.random() < 0.5, tex=rng.random() < 0.25)
    elif kind == "extinction":
        c.update(light=rng.choice(["directional", "directional", "point"]), shells=rng.choice(["nested", "unit"]),
                 edit=rng.random() < 0.4)
    elif kind == "cone":
        cached = rng.random() < 0.5
        c.update(cache=_log(rng, 16, 48) if cached else 0, edit=cached and rng.random() < 0.7,
                 quads=rng.random() < 0.5)
    elif kind == "ground_truth":
        c.update(quads=rng.random() < 0.5)
    elif kind == "iso":
        c.update(scale=rng.choice(["none", "multi", "down"]), quads=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ inputs


def _rng(*seed):
    return np.random.default_rng([int(v) for v in seed])


def _to_bits(v, bits):
    top = 255 if bits == 8 else 65535
    q = (v.clamp(0.0, 1.0) * top).round()
    return q.to(torch.uint8) if bits == 8 else q.to(torch.int32).to(torch.uint16)


def _blobs(w, h, d, bits, count, noise, seed):
    """Isotropic Gaussian blobs in the unit cube, over a uniform noise floor of `noise` of 255."""
    r = _rng(seed)
    side = max(w, h, d)
    vol = torch.zeros((d, h, w), device=DEV)
    ax = [(torch.arange(n, device=DEV) + 0.5) / side + 0.5 * (1.0 - n / side) for n in (w, h, d)]
    for _ in range(count):
        c, s, a = r.uniform(0.2, 0.8, 3), r.uniform(0.05, 0.15), r.uniform(0.5, 1.0)
        ex, ey, ez = (torch.exp(-((x - float(m)) ** 2) / (2.0 * s * s)) for x, m in zip(ax, c))
        vol += float(a) * ez[:, None, None] * ey[None, :, None] * ex[None, None, :]
    vol.clamp_(0.0, 1.0)
    if noise:
        g = torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)
        vol += torch.rand((d, h, w), device=DEV, generator=g) * (noise / 255.0)
    return _to_bits(vol, bits)


def _shells(w, h, d, bits, seed):
    """Four-octave value noise (lacunarity 2, gain 0.5) cut into four nested shells."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)
    side, v, amp, norm = max(w, h, d), torch.zeros((d, h, w), device=DEV), 1.0, 0.0
    for o in range(4):
        f = 4 * 2 ** o
        t = torch.rand((f + 2, f + 2, f + 2), device=DEV, generator=g)
        for axis, n in ((0, d), (1, h), (2, w)):
            p = (torch.arange(n, device=DEV) + 0.5) * (f / side)
            i = p.floor().long()
            s = p - i
            s = s * s * (3.0 - 2.0 * s)
            shape = [1, 1, 1]
            shape[axis] = n
            lo, hi = t.index_select(axis, i), t.index_select(axis, i + 1)
            t = lo + (hi - lo) * s.reshape(shape)
        v += amp * t
        norm += amp
        amp *= 0.5
    v /= norm
    k = sum((v > s / 5.0).float() for s in range(1, 5))
    return _to_bits(k / 4.0, bits)


TF_ISO = (0, 80, 160, 255)
TF_RGB = ((0.20, 0.30, 0.90), (0.30, 0.80, 0.40), (0.90, 0.70, 0.20), (1.00, 0.95, 0.90))


def _tf(seed):
    """256-entry (colour, extinction) and (colour, opacity) tables through four control points, opacity jittered."""
    j = _rng(seed, 7).uniform(0.9, 1.1, 4)
    op = np.interp(np.arange(256), TF_ISO, np.array([0.0, 0.05, 0.4, 0.9]) * j).clip(0.0, 0.995).astype(np.float32)
    rgb = np.stack([np.interp(np.arange(256), TF_ISO, [p[k] for p in TF_RGB]) for k in range(3)], 1)
    ext = np.log(1.0 / (1.0 - op.astype(np.float64)))
    rgbt = np.concatenate([rgb, ext[:, None]], 1).astype(np.float32)
    rgba = np.concatenate([rgb, op[:, None]], 1).astype(np.float32)
    return np.ascontiguousarray(rgbt), np.ascontiguousarray(rgba)


def _ext_of_values(rgba, bits):
    """Extinction of every voxel value: the opacity interpolated at value / max, then -log(1 - opacity)."""
    n = 256 if bits == 8 else 65536
    op = np.interp(np.arange(n) / (n - 1.0) * 255.0, np.arange(256), rgba[:, 3].astype(np.float64))
    return np.log(1.0 / (1.0 - op))


def _volume(case, seed):
    dims = case["w"], case["h"], case["d"], case["bits"]
    kind = case["kind"]
    if kind in ("extinction", "iso"):
        return _shells(*dims, seed)
    if kind == "plain":
        return _blobs(*dims, 8, 0.0, seed)
    return _blobs(*dims, 32, 20.0, seed)


def _diag(case):
    return math.sqrt(case["w"] ** 2 + case["h"] ** 2 + case["d"] ** 2)


def _view(case, seed):
    """Spacing, camera, light and method parameters."""
    r = _rng(seed, 3)
    kind, n = case["kind"], max(case["w"], case["h"], case["d"])
    sp = (1.0 / n,) * 3 if kind == "plain" else (1.0, 1.0, 1.0)
    size = n * sp[0]
    eye = scene.orbit_eye(3.0 * size, float(r.uniform(-60, 60)), float(r.uniform(10, 35)))
    cam = scene.camera(eye, fovy=30.0)
    ldir = np.array([r.uniform(-0.5, 0.5), 0.8, r.uniform(0.2, 0.6)])
    ldir /= np.linalg.norm(ldir)
    fwd, up, right = scene.light_frame(ldir)
    directional = case.get("light") == "directional"
    lt = scene.light(abi.LIGHT_DIRECTIONAL if directional else abi.LIGHT_POINT, position=tuple(2.0 * size * ldir),
                     forward=fwd, up=up, right=right)
    step, diag = scene.default_step(sp), _diag(case)
    if kind == "plain":
        p = abi.PlainParams()
        p.step_size = step
    elif kind == "extinction":
        radii = (2, 6, 16) if case["shells"] == "nested" else tuple(range(1, 16))
        p = scene.ext_params(step, diag, ao_radii=radii, shadow_type=1 if directional else 0)
    elif kind == "cone":
        p = scene.dos_params(step, apply_occ=True, apply_sdw=True, shadow_type=0)
    elif kind == "iso":
        p = scene.iso_params(isovalue=0.6, small=0.1, large=0.8, step_range=0.1, color=(0.66, 0.6, 0.05, 0.8))
    else:
        p = scene.gt_params(step, diag, occ_distance=32.0, light_step=1.0, gap=1.0, shadow_type=0)
    return sp, cam, lt, p


def _hemisphere(seed):
    """16 occlusion directions of a wide cone about +z and the light's own direction."""
    r = _rng(seed, 5)
    z = 1.0 - r.uniform(0.0, 1.0, 16) * (1.0 - math.cos(math.radians(80.0)))
    a, s = r.uniform(0.0, 2.0 * math.pi, 16), np.sqrt(1.0 - z * z)
    return np.stack([s * np.cos(a), s * np.sin(a), z], 1).astype(np.float32), np.array([[0, 0, 1]], np.float32)


METHOD = {"plain": abi.PLAIN, "extinction": abi.EXTINCTION, "cone": abi.CONE_DOS, "ground_truth": abi.GROUND_TRUTH,
          "surrogate": abi.SURROGATE, "iso": abi.ISO}


class State:
    """One scene: a context, what stays on the host for its calls, and the frame."""

    def __init__(self, case):
        self.case = case
        self.ctx = scene.Context(0)
        self.lib, self.h = self.ctx.lib, self.ctx.h
        self.batch = None

    def ck(self, code):
        abi.check(code, self.h)

    def __del__(self):
        if self.batch:
            self.lib.cvr_batch_destroy(self.batch)
            self.batch = None
        self.ctx.close()


def _set_volume(s, vol, sp=(1.0, 1.0, 1.0)):
    d, h, w = vol.shape
    dtype = abi.CVR_U8 if vol.dtype == torch.uint8 else abi.CVR_U16
    s.ck(s.lib.cvr_set_volume_device(s.h, vol.data_ptr(), w, h, d, dtype, *sp))


def _set_tf(s):
    s.ck(s.lib.cvr_set_transfer_function(s.h, abi.fptr(s.rgbt), abi.fptr(s.rgba), len(s.rgbt)))


def _tables(s, case):
    """The tables that follow the transfer function."""
    _set_tf(s)
    if case["kind"] == "extinction":
        s.ck(s.lib.cvr_build_sat(s.h, abi.dptr(s.ext), len(s.ext)))
    elif case["kind"] in ("cone", "surrogate"):
        s.ck(s.lib.cvr_build_ext_pyramid(s.h, C.byref(s.pyramid)))


def prepare(case, seed):
    s = State(case)
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(s, case, seed)
    if kind == "batch":
        return _prepare_batch(s, case, seed)
    vol = _volume(case, seed)
    s.rgbt, s.rgba = _tf(seed)
    s.sp, s.cam, s.light, s.params = _view(case, seed)
    torch.cuda.synchronize()
    _set_volume(s, vol, s.sp)
    s.vol = vol if kind == "iso" else None
    if case.get("quads"):
        s.ck(s.lib.cvr_set_volume_layout(s.h, abi.LAYOUT_QUADS))
    if case.get("tex"):
        s.ck(s.lib.cvr_set_sampling(s.h, abi.SAMPLING_TEX_FEATURES | abi.SAMPLING_TEX_VOLUME))
    if kind == "extinction":
        s.ck(s.lib.cvr_set_warp_shape(s.h, 4))
        s.ext = np.ascontiguousarray(_ext_of_values(s.rgba, case["bits"]))
    if kind in ("cone", "surrogate"):
        s.pyramid = abi.PyramidParams()
        s.pyramid.base_dims[:] = [max(1, case[k] // 2) for k in "whd"]
        s.pyramid.sigma0, s.pyramid.n_levels = 1.0, 5 if kind == "cone" else abi.SURROGATE_LEVELS
    if kind == "cone":
        diag = _diag(case)
        s.cones = [scene.cone_table(20.0, 1, 0.5 * diag, 3.0, 0.35, 1.0),
                   scene.cone_table(0.5, 0, 0.75 * diag, 3.0, 1.0, 1.0)]
        s.ck(s.lib.cvr_set_cone_tables(s.h, C.byref(s.cones[0]), C.byref(s.cones[1])))
        s.ck(s.lib.cvr_set_light_cache(s.h, case["cache"], case["cache"], case["cache"]))
    if kind in ("ground_truth", "surrogate"):
        s.ctx.set_gt_kernels(*_hemisphere(seed))
    if kind == "surrogate":
        s.ctx.set_sampling(abi.SAMPLING_TEX_FEATURES | abi.SAMPLING_TEX_VOLUME)
        s.ck(s.lib.cvr_mlp_init(s.h, 11))
        p = s.ctx.mlp_params()  # outputs inside [0, 1], as a trained network's are
        p[-2:] = 0.5
        p[-130:-2] *= 0.05
        s.ctx.mlp_set_params(p)
    if kind == "iso":
        s.grad = abi.GradientParams(abi.GRADIENT_FINITE_DIFFERENCES, 1, 0, 1)
        s.ctx.set_blinn_phong(True)
        mode = {"none": abi.MULTISCALE_SINGLE, "multi": abi.MULTISCALE_MULTISAMPLE,
                "down": abi.MULTISCALE_DOWNSCALE}[case["scale"]]
        s.ctx.set_multiscaling(mode, abi.FILTER_HAT, 2, 2)
    _tables(s, case)
    s.out = torch.zeros((case["height"], case["width"], 4), device=DEV)
    torch.cuda.synchronize()
    s.ck(s.lib.cvr_sync(s.h))
    return s


def _prepare_train(s, case, seed):
    """Features in [0, 1] with smooth targets of them, as the integrator's labels are."""
    r = _rng(seed)
    n = case["points"]
    x = r.uniform(0.0, 1.0, (n, 48)).astype(np.float32)
    wts = r.normal(0.0, 0.4, (48, 2)).astype(np.float32)
    t = (1.0 / (1.0 + np.exp(-(x - 0.5) @ wts))).astype(np.float32)
    s.ck(s.lib.cvr_mlp_init(s.h, 5))
    s.start = s.ctx.mlp_params()
    s.ck(s.lib.cvr_mlp_set_training_data(s.h, abi.fptr(x), abi.fptr(np.ascontiguousarray(t)), n))
    s.loss = np.zeros(case["epochs"], np.float32)
    s.weights = np.zeros(abi.MLP_PARAMS, np.float32)
    return s


def _prepare_batch(s, case, seed):
    """Four resident volumes of uneven size, `views` cameras, `lights` lights, both shadings."""
    n = case["side"]
    dims = [(n, n, n, 8), (3 * n // 4, n, 5 * n // 8, 16), (n, n, n, 8), (3 * n // 2, 3 * n // 2, 3 * n // 2, 16)]
    s.rgbt, s.rgba = _tf(seed)
    _set_tf(s)
    for slot, (w, h, d, bits) in enumerate(dims):
        s.ctx.select_volume(slot)
        vol = _shells(w, h, d, bits, int(seed) * 4 + slot)
        torch.cuda.synchronize()
        _set_volume(s, vol)
        ext = np.ascontiguousarray(_ext_of_values(s.rgba, bits))
        s.ck(s.lib.cvr_build_sat(s.h, abi.dptr(ext), len(ext)))
        s.ctx.build_pyramid(base_dims=(w // 2, h // 2, d // 2), sigma0=1.0, n_levels=abi.SURROGATE_LEVELS)
        s.ck(s.lib.cvr_sync(s.h))
    s.ctx.select_volume(0)
    s.ck(s.lib.cvr_set_warp_shape(s.h, 4))
    s.ck(s.lib.cvr_mlp_init(s.h, 11))
    p = s.ctx.mlp_params()
    p[-2:] = 0.5
    p[-130:-2] *= 0.05
    s.ctx.mlp_set_params(p)
    n_jobs = 4 * case["views"] * case["lights"] * 2
    s.out = torch.zeros((n_jobs, case["height"], case["width"], 4), device=DEV)
    r = _rng(seed, 3)
    views = [np.array([math.cos(a) * math.cos(e), math.sin(e), math.sin(a) * math.cos(e)])
             for a, e in zip(r.uniform(0, 2 * math.pi, case["views"]), r.uniform(-0.6, 0.6, case["views"]))]
    ldirs = [np.array([r.uniform(-0.6, 0.6), r.uniform(0.4, 0.9), r.uniform(-0.6, 0.6)])
             for _ in range(case["lights"])]
    s.jobs, s.params = [], []
    for slot, (w, h, d, _) in enumerate(dims):
        side, diag = max(w, h, d), math.sqrt(w * w + h * h + d * d)
        for v in views:
            cam = scene.camera(tuple(2.6 * side * v), fovy=30.0)
            for ld in ldirs:
                fwd, up, right = scene.light_frame(ld)
                lt = scene.light(abi.LIGHT_DIRECTIONAL, position=tuple(3.0 * side * np.array(fwd)), forward=fwd,
                                 up=up, right=right)
                for m in (abi.EXTINCTION, abi.SURROGATE):
                    step = scene.default_step((1.0, 1.0, 1.0))
                    p = scene.ext_params(step, diag) if m == abi.EXTINCTION else \
                        scene.gt_params(step, diag, occ_distance=32.0, light_step=1.0, gap=1.0, shadow_type=2)
                    j = abi.Job()
                    j.volume, j.method, j.params, j.params_size = slot, m, C.addressof(p), C.sizeof(p)
                    j.camera, j.light, j.width, j.height = cam, lt, case["width"], case["height"]
                    j.out_rgba_dev = s.out[len(s.jobs)].data_ptr()
                    s.jobs.append(j)
                    s.params.append(p)
    b = C.c_void_p()
    torch.cuda.synchronize()
    s.ck(s.lib.cvr_batch_create(s.h, (abi.Job * n_jobs)(*s.jobs), n_jobs, C.byref(b)))
    s.batch = b
    s.ck(s.lib.cvr_sync(s.h))
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "train":
        s.ck(s.lib.cvr_mlp_set_params(s.h, abi.fptr(s.start), abi.MLP_PARAMS))
        s.ck(s.lib.cvr_mlp_train(s.h, case["epochs"], case["batch"], 2e-3, 17, abi.fptr(s.loss)))
        s.ck(s.lib.cvr_mlp_get_params(s.h, abi.fptr(s.weights), abi.MLP_PARAMS))
        return {"weights": s.weights, "loss": s.loss}
    if kind == "batch":
        s.ck(s.lib.cvr_batch_run(s.batch))
        return s.out
    if kind == "iso":
        _set_volume(s, s.vol, s.sp)
        s.ck(s.lib.cvr_build_gradient(s.h, C.byref(s.grad)))
    if case.get("edit"):
        _tables(s, case)
    s.ck(s.lib.cvr_render(s.h, METHOD[kind], C.byref(s.cam), C.byref(s.light), C.byref(s.params), C.sizeof(s.params),
                          s.out.data_ptr(), case["width"], case["height"], None, None))
    return s.out


# ------------------------------------------------------------------ work


def work(case):
    """The volume and the tables of a frame read once, the frame written once; the arithmetic of the steps of its rays
    (a ray through the box takes two steps a voxel; the shaded methods stop after some tens of steps in dense data)."""
    kind = case["kind"]
    if kind == "train":
        steps = case["epochs"] * case["points"]
        return {"bytes": steps * 50 * 4.0, "flops": steps * 3.0 * 14592}
    if kind == "batch":
        jobs, px, n = 4 * case["views"] * case["lights"], case["width"] * case["height"], case["side"]
        vox = n ** 3 * (1 + 0.47 * 2 + 1 + 3.4 * 2)
        return {"bytes": vox + jobs * 2 * px * 16.0, "flops": jobs * 0.4 * px * (25 * 30 * 60.0 + n * 15000.0)}
    vox, px = case["w"] * case["h"] * case["d"], case["width"] * case["height"]
    n = (case["w"] + case["h"] + case["d"]) / 3.0
    hit = 0.45 * px
    size = vox * case["bits"] / 8.0 + px * 16.0
    if kind == "plain":
        return {"bytes": size, "flops": hit * n * 50.0}
    if kind == "extinction":
        boxes = 3 if case["shells"] == "nested" else 15
        return {"bytes": size + vox * 4.0 * (2 if case["edit"] else 1), "flops": hit * 45 * (boxes + n / 6.0) * 60.0}
    if kind == "cone":
        if case["cache"]:
            return {"bytes": size + vox / 8 * 4.0, "flops": hit * n * 80.0 + case["cache"] ** 3 * 2500.0}
        return {"bytes": size + vox / 8 * 4.0, "flops": hit * n * 2500.0}
    if kind == "ground_truth":
        return {"bytes": size, "flops": hit * n * 490 * 40.0}
    if kind == "surrogate":
        return {"bytes": size + vox / 8 * 4.0, "flops": hit * n * (14592.0 + 67 * 20)}
    rays = 1 if case["scale"] == "none" else 4
    return {"bytes": 2.0 * size + vox * 16.0, "flops": hit * rays * n * 40.0}


# ------------------------------------------------------------------ the same in 64 bits


def _d(v):
    return torch.tensor(np.array(v, np.float64), device=DEV)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


class Exact:
    """The frames in 64 bits, plainly: every ray's steps side by side, the shaded samples in large chunks."""

    CHUNK = 1 << 21

    def __init__(self, case, seed):
        self.case = case
        vol = _volume(case, seed)
        self.v = (vol.to(torch.int32) if case["bits"] == 16 else vol).double().reshape(-1) / (2.0 ** case["bits"] - 1)
        self.dims = case["w"], case["h"], case["d"]
        self.rgbt, self.rgba = _tf(seed)
        self.tf = _d(self.rgbt)
        self.sp, self.cam, self.light, self.p = _view(case, seed)
        self.sp = _d(np.float32(self.sp))
        self.grid = _d(self.dims) * self.sp
        scale = 2 if case.get("scale", "none") == "multi" else 1
        self.W, self.H = case["width"] * scale, case["height"] * scale
        self.rays()

    def rays(self):
        eye, ctr, up = (np.array(v[:], np.float64) for v in (self.cam.eye, self.cam.center, self.cam.up))
        f = (ctr - eye) / np.linalg.norm(ctr - eye)
        s = np.cross(f, up)
        s /= np.linalg.norm(s)
        u = np.cross(s, f)
        t = math.tan(math.radians(self.cam.fovy_deg) / 2.0)
        x = ((torch.arange(self.W, device=DEV).double() + 0.5) / self.W * 2 - 1) * t * (self.case["width"] / self.case["height"])
        y = ((torch.arange(self.H, device=DEV).double() + 0.5) / self.H * 2 - 1) * t
        d = x[None, :, None] * _d(s) + y[:, None, None] * _d(u) + _d(f)
        d = _unit(d.reshape(-1, 3))
        self.eye = _d(eye)
        a, b = (-0.5 * self.grid - self.eye) / d, (0.5 * self.grid - self.eye) / d
        near, far = torch.minimum(a, b).amax(1), torch.maximum(a, b).amin(1)
        self.hit = (far > near).nonzero().reshape(-1)
        near = near[self.hit].clamp_min(0.0)
        self.dir, self.D = d[self.hit], (far[self.hit] - near).abs()
        self.tex0 = self.eye + self.dir * near[:, None] + self.grid * 0.5

    def tri(self, data, dims, p):
        """Trilinear, texel centres, clamped to the edge; p in texels."""
        out, idx, w = None, [], []
        for a in range(3):
            fl = p[..., a].floor()
            t, i = p[..., a] - fl, fl.long()
            idx.append((i.clamp(0, dims[a] - 1), (i + 1).clamp(0, dims[a] - 1)))
            w.append((1.0 - t, t))
        for k in range(8):
            i, j, m = k & 1, (k >> 1) & 1, k >> 2
            at = idx[0][i] + dims[0] * (idx[1][j] + dims[1] * idx[2][m])
            term = data[at] * (w[0][i] * w[1][j] * w[2][m])
            out = term if out is None else out + term
        return out

    def density(self, p):
        return self.tri(self.v, self.dims, p / self.sp - 0.5)

    def lookup(self, density, channel=slice(None)):
        u = density * 256.0 - 0.5
        fl = u.floor()
        t, i = u - fl, fl.long()
        a, b = self.tf[i.clamp(0, 255), channel], self.tf[(i + 1).clamp(0, 255), channel]
        t = t[:, None] if a.dim() == 2 else t
        return a + (b - a) * t

    def frame(self, shade):
        """Front-to-back compositing; shade(points, directions) gives the factor of the samples' colours, or is None."""
        n = len(self.hit)
        img = torch.zeros((n, 4), device=DEV, dtype=torch.float64)
        live = torch.arange(n, device=DEV)
        s = torch.zeros(n, device=DEV, dtype=torch.float64)
        step = float(self.p.step_size)
        kept = []
        while len(live):
            sl = s[live]
            h = torch.clamp(self.D[live] - sl, max=step)
            p = self.tex0[live] + self.dir[live] * (sl + h * 0.5)[:, None]
            src = self.lookup(self.density(p))
            a = 1.0 - torch.exp(-src[:, 3] * h)
            wgt = (1.0 - img[live, 3]) * a
            if shade is None:
                img[live, :3] += wgt[:, None] * src[:, :3]
            else:
                m = src[:, 3] > 0
                kept.append((live[m], p[m], wgt[m], src[m, :3]))
            img[live, 3] += wgt
            s[live] = sl + h
            live = live[(s[live] < self.D[live] * (1 - 1e-7)) & (img[live, 3] <= 0.99)]
        if shade is not None and kept:
            ray, p, wgt, rgb = (torch.cat(x) for x in zip(*kept))
            for i in range(0, len(ray), self.CHUNK):
                at = slice(i, i + self.CHUNK)
                f = shade(p[at], self.dir[ray[at]])
                img.index_add_(0, ray[at], torch.nn.functional.pad((wgt[at] * f)[:, None] * rgb[at], (0, 1)))
        return self.image(img)

    def image(self, hits):
        out = torch.zeros((self.H * self.W, 4), device=DEV, dtype=torch.float64)
        out[self.hit] = hits
        out = out.reshape(self.H, self.W, 4)
        if (self.H, self.W) != (self.case["height"], self.case["width"]):
            out = out.reshape(self.case["height"], 2, self.case["width"], 2, 4).mean((1, 3))
        return out.cpu().numpy()

    # -- extinction: ambient-occlusion boxes and the shadow cone's boxes in the summed-area table
    def sat(self):
        w, h, d = self.dims
        ext = _d(_ext_of_values(self.rgba, self.case["bits"]))
        val = ext[(self.v * (2.0 ** self.case["bits"] - 1)).round().long()].reshape(d, h, w)
        self.S = torch.nn.functional.pad(val, (1, 1, 1, 1, 1, 1)).cumsum(0).cumsum(1).cumsum(2).reshape(-1)
        self.sdims = w + 2, h + 2, d + 2

    def box(self, p1, p2):
        lo, hi = self.sp * 0.5, self.grid + self.sp * 1.5
        c = [torch.minimum(torch.maximum(p + self.sp, lo), hi) / self.sp - 0.5 for p in (p1, p2)]
        out = 0.0
        for k in range(8):
            q = torch.stack([c[(k >> a) & 1][:, a] for a in range(3)], 1)
            sign = 1.0 if bin(k).count("1") % 2 else -1.0
            out = out + sign * self.tri(self.S, self.sdims, q)
        return out

    def extinction(self, p, _):
        q = self.p
        radii = [float(q.ao_radii[i]) for i in range(q.ao_n_shells)]
        t = last = 0.0
        for r in radii:
            b = self.box(p - self.sp * r, p + self.sp * r)
            t, last = t + (b - last) / (r * r), b
        ao = torch.exp(-t / radii[-1] ** 2)
        if q.shadow_type == 1:
            c = _unit(_d(self.light.forward[:])).expand(len(p), 3)
        else:
            c = _unit(_d(self.light.position[:]) - (p - self.grid * 0.5))
        a = c.abs()
        axis = torch.where((a[:, 2] > a[:, 0]) & (a[:, 2] > a[:, 1]), 2, torch.where(a[:, 1] > a[:, 0], 1, 0))
        sh = torch.zeros(len(p), device=DEV, dtype=torch.float64)
        for m in range(3):
            at = (axis == m).nonzero().reshape(-1)
            if len(at):
                sh[at] = self.cone_walk(p[at], c[at], m)
        return (ao * q.ka + torch.exp(-sh) * q.kd) / (q.ka + q.kd)

    def cone_walk(self, p, c, m):
        q, sc = self.p, self.sp
        ang, lateral = float(q.sdw_cone_angle_rad), [a for a in range(3) if a != m]
        slopes = []
        for a in lateral:
            n = torch.hypot(c[:, a], c[:, m])
            ca, cm = c[:, a] / n, c[:, m] / n
            slopes.append([(ca * math.cos(g) - cm * math.sin(g)) / (ca * math.sin(g) + cm * math.cos(g)).abs()
                           for g in (-ang, ang)])
        sign = torch.where(c[:, m] < 0, -1.0, 1.0).double()
        gap = float(q.sdw_sample_interval) * sign * sc[m]
        z = float(q.sdw_initial_step) * sign * sc[m]
        out = torch.zeros(len(p), device=DEV, dtype=torch.float64)
        live = torch.arange(len(p), device=DEV)
        lo_v, hi_v = sc[m] * 0.5, self.grid[m] - sc[m] * 0.5
        while True:
            nxt = p[live, m] + z[live] + gap[live]
            live = live[(z[live] / c[live, m] < float(q.sdw_max_distance)) & (nxt > lo_v) & (nxt < hi_v)]
            if not len(live):
                return out
            zm = (z[live] + gap[live] * 0.5).abs()
            lo, hi = torch.empty((len(live), 3), device=DEV).double(), torch.empty((len(live), 3), device=DEV).double()
            for a, sl in zip(lateral, slopes):
                e = sl[0][live] * zm, sl[1][live] * zm
                l, u = torch.minimum(*e), torch.maximum(*e)
                wide = (u - l) / sc[a]
                grow = (wide.ceil() - wide) * 0.5 * sc[a]
                lo[:, a], hi[:, a] = l - grow, u + grow
            lo[:, m] = torch.minimum(z[live], z[live] + gap[live])
            hi[:, m] = torch.maximum(z[live], z[live] + gap[live])
            voxels = ((hi - lo) / sc).prod(1)
            out[live] += self.box(p[live] + lo, p[live] + hi) / voxels * float(q.sdw_ui_weight)
            z = z + gap

    # -- ground truth: transmittance along sampled light rays
    def light_rays(self, p, w, dist):
        q = self.p
        vt = torch.ones(len(p), device=DEV, dtype=torch.float64)
        s = torch.full_like(vt, float(q.light_ray_initial_gap))
        last = self.lookup(self.density(p + w * s[:, None]), 3)
        live = torch.arange(len(p), device=DEV)
        while len(live):
            h = torch.clamp(dist - s[live], max=float(q.light_ray_step_size))
            at = p[live] + w[live] * (s[live] + h)[:, None]
            ok = ((at >= 0) & (at <= self.grid)).all(1)
            live, h, at = live[ok], h[ok], at[ok]
            now = self.lookup(self.density(at), 3)
            vt[live] *= torch.exp(-(last[live] + now) * 0.5 * h)
            last[live] = now
            s[live] += h
            live = live[(1.0 - vt[live] <= 0.99) & (s[live] < dist - 1e-9)]
        return vt

    def ground_truth(self, p, d):
        q, (occ, _) = self.p, self.vectors
        right = _unit(torch.linalg.cross(d, _d([0.0, 1.0, 0.0]).expand_as(d)))
        up = _unit(torch.linalg.cross(-d, right))
        num = den = 0.0
        for v in occ.astype(np.float64):
            w = _unit(right * v[0] + up * v[1] - d * v[2])
            rw = -(w * d).sum(1)
            num = num + self.light_rays(p, w, float(q.occ_distance)) * rw
            den = den + rw
        w = _unit(_d(self.light.position[:]) - (p - self.grid * 0.5))
        return (num / den * q.ka + self.light_rays(p, w, float(q.sdw_distance)) * q.kd) / (q.ka + q.kd)

    # -- isosurface with Blinn-Phong shading from central differences
    def gradient(self):
        w, h, d = self.dims
        v = torch.nn.functional.pad(self.v.reshape(d, h, w), (1, 1, 1, 1, 1, 1))
        c = slice(1, -1)
        g = torch.stack([v[c, c, 2:] - v[c, c, :-2], v[c, 2:, c] - v[c, :-2, c], v[2:, c, c] - v[:-2, c, c]], -1)
        n = g.norm(dim=-1, keepdim=True)
        self.G = torch.where(n > 0, g / n, torch.zeros_like(g)).reshape(-1, 3)

    def phong(self, p):
        q = p / self.sp - 0.5
        n = torch.stack([self.tri(self.G[:, a].contiguous(), self.dims, q) for a in range(3)], 1)
        flat = (n == 0).all(1)
        n = _unit(n)
        wpos = p - self.grid * 0.5
        l = _unit(_d(self.light.position[:]) - wpos)
        hv = _unit(_unit(self.eye - wpos) + l)
        diff = (n * l).sum(1).clamp_min(0.0)
        spec = (hv * n).sum(1).clamp_min(0.0) ** 30.0
        rgb = _d(self.p.color[:3])[None] * (0.5 + 0.5 * diff)[:, None] + (0.8 * spec)[:, None]
        return torch.where(flat[:, None], _d(self.p.color[:3])[None], rgb)

    def iso(self):
        q = self.p
        small, large, rng, iso = (float(v) for v in (q.step_size_small, q.step_size_large, q.step_size_range, q.isovalue))
        a = float(q.color[3])
        n = len(self.hit)
        img = torch.zeros((n, 4), device=DEV, dtype=torch.float64)
        live, s, prev = torch.arange(n, device=DEV), torch.zeros(n, device=DEV).double(), self.density(self.tex0)
        while len(live):
            sl, pv = s[live], prev[live]
            h = torch.minimum(torch.where((pv - iso).abs() < rng, small, large).double(), self.D[live] - sl)
            d = self.density(self.tex0[live] + self.dir[live] * (sl + h)[:, None])
            m = ((pv <= iso) & (d > iso)) | ((pv >= iso) & (d < iso))
            if bool(m.any()):
                at = live[m]
                t = (iso - pv[m]) / (d[m] - pv[m])
                rgb = self.phong(self.tex0[at] + self.dir[at] * (sl[m] + t * h[m])[:, None])
                wgt = (1.0 - img[at, 3]) * a
                img[at, :3] += wgt[:, None] * rgb
                img[at, 3] += wgt
            prev[live], s[live] = d, sl + h
            live = live[(s[live] < self.D[live] * (1 - 1e-7)) & (img[live, 3] <= 0.99)]
        return self.image(img)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cone", "surrogate", "batch", "train") or case.get("tex") or case.get("scale") == "down":
        return None  # the sampler's cone tables, 16-bit operands, hardware filter weights: no plain 64-bit value
    e = Exact(case, seed)
    if kind == "plain":
        return e.frame(None)
    if kind == "extinction":
        e.sat()
        return e.frame(e.extinction)
    if kind == "ground_truth":
        e.vectors = _hemisphere(seed)
        return e.frame(e.ground_truth)
    e.gradient()
    return e.iso()
