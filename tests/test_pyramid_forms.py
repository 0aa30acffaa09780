"""Which form each pyramid takes (on a fake CUDA runtime), and the lattices
against the FP64 oracle: bases of the volume's own size, taps of several
voxels, other ratios per axis, and levels too wide for a tile."""
import numpy as np
import pytest

import oracle
from cpp_volume_rendering_gb300 import abi, scene
from tests import fakegpu

FORMS = ("k_pyr_base_half", "k_pyr_base_window", "k_pyr_lattice_base", "k_pyr_base")


def built(ctx, dims, spacing, base, s0, levels=5):
    """The base's form and the levels that are lattices."""
    ctx.resize(280 << 30)
    w, h, d = dims
    ctx.set_volume(np.zeros((d, h, w), np.uint8), spacing)
    ctx.set_transfer_function(scene.BENCH_TF)
    ctx.build_pyramid(base_dims=base, sigma0=s0, n_levels=levels)
    form = next(k for k in FORMS if ctx.launches(k))
    return form, ctx.launches("k_pyr_lattice_level")


@pytest.mark.parametrize("dims,spacing,base,s0,form,levels", [
    ((64, 64, 64), 1.0, (32, 32, 32), 1.0, "k_pyr_base_half", 0),
    ((32, 32, 32), 1.0, (32, 32, 32), 1.0, "k_pyr_lattice_base", 0),     # a base of the volume's own size
    ((64, 64, 64), 0.5, (32, 32, 32), 1.0, "k_pyr_lattice_base", 0),     # taps of two voxels
    ((32, 32, 32), 0.25, (32, 32, 32), 1.0, "k_pyr_lattice_base", 4),    # of four, on every level
    ((64, 64, 32), 1.0, (32, 32, 32), 1.0, "k_pyr_lattice_base", 0),     # half on two axes
    ((128, 128, 128), 1.0, (32, 32, 32), 1.0, "k_pyr_base_window", 0),   # 73 lattice points a cell
    ((40, 33, 32), 1.0, (20, 16, 16), 1.0, "k_pyr_base_window", 0),      # no whole ratio
    ((32, 32, 32), 1.0, (16, 16, 16), 5.5, "k_pyr_base", 0),             # no whole tap
])
def test_forms(dims, spacing, base, s0, form, levels):
    ctx = fakegpu.Context(fakegpu.load())
    try:
        assert built(ctx, dims, (spacing,) * 3, base, s0) == (form, levels)
    finally:
        ctx.close()


def test_no_room_for_a_lattice():
    """Room for the levels alone: the window; for nothing beside them: in place."""
    lib = fakegpu.load()
    ctx = fakegpu.Context(lib)
    try:
        n = 64
        ctx.set_volume(np.zeros((n, n, n), np.uint8))
        ctx.set_transfer_function(scene.BENCH_TF)
        levels = 4 * sum((n >> l) ** 3 for l in range(5))
        ctx.resize(lib.fake_used() + 2 * levels + 4096)
        ctx.build_pyramid(base_dims=(n, n, n), sigma0=1.0, n_levels=5)
        assert ctx.launches("k_pyr_base_window") == 1 and ctx.launches("k_pyr_lattice_base") == 0
        assert ctx.launches("k_pyr_backtotau") == 0
    finally:
        ctx.close()
    ctx = fakegpu.Context(lib)
    try:
        ctx.set_volume(np.zeros((n, n, n), np.uint8))
        ctx.set_transfer_function(scene.BENCH_TF)
        ctx.resize(lib.fake_used() + levels + 4096)
        ctx.build_pyramid(base_dims=(n, n, n), sigma0=1.0, n_levels=5)
        assert ctx.launches("k_pyr_base_window") == 1 and ctx.launches("k_pyr_backtotau") == 1
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,spacing,base,s0", [
    ((20, 17, 33), (1.0, 1.0, 1.0), (20, 17, 33), 1.0),    # own size, odd
    ((40, 36, 24), (0.5, 0.5, 0.5), (20, 18, 12), 1.0),    # half the size, taps of two voxels
    ((24, 20, 16), (0.25, 0.25, 0.25), (24, 20, 16), 1.0),  # taps of four voxels: the levels too
    ((36, 18, 12), (1.0, 0.5, 0.25), (12, 18, 12), 1.0),   # ratios 3, 1, 1 and taps of 1, 2, 4 voxels
    ((16, 4, 1), (1.0, 1.0, 1.0), (16, 4, 1), 1.0),        # one voxel along z
    ((32, 32, 32), (1.0, 1.0, 1.0), (16, 16, 16), 5.5),    # direct base and levels
])
@pytest.mark.parametrize("dtype", [abi.CVR_U8, abi.CVR_U16])
def test_lattices_match_oracle(ctx, dims, spacing, base, s0, dtype):
    wl = scene.workload("cone", n=32, image=8)
    w, h, d = dims
    wl.volume = scene.synth_blobs(w, h, d, dtype, 8, seed=41, noise_max=20.0)
    wl.spacing = spacing
    wl.pyramid = dict(base_dims=base, sigma0=s0, n_levels=4)
    scene.prepare(ctx, wl)
    levels = ctx.pyramid()
    orc = oracle.Oracle()
    oracle.prepare(orc, wl)
    assert len(levels) == orc.n_levels
    for l, lev in enumerate(levels):
        ref = orc.pyramid_level(l, 64)
        assert lev.shape == ref.shape
        # the bound of the other pyramid tests: FP32 coordinates, 343 FP32 terms
        err = np.abs(lev - ref) / np.maximum(np.abs(ref), 1e-3)
        assert err.max() <= 1e-4, (l, err.max())
