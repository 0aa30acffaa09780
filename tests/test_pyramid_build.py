"""The pyramid builders at the edges of their forms, against the FP64 oracle:
the lattice of a half-size base (partial tiles and z chunks), the window of a
base of any size (upsampled, far coarser than the volume, one voxel thick), the
levels' tiles of both sizes and the direct kernels beside them."""
import numpy as np
import pytest

import oracle
from cpp_volume_rendering_gb300 import abi, scene

pytestmark = pytest.mark.gpu

CASES = [((34, 66, 36), (17, 33, 18), 1.0),   # half: two tiles and a cell, two z chunks
         ((32, 32, 34), (16, 16, 17), 1.0),   # half: whole tiles, one plane in a chunk of its own
         ((33, 21, 40), (16, 10, 20), 1.0),   # window: ragged
         ((64, 20, 1), (5, 3, 1), 1.0),       # window: cells far apart, one voxel along z
         ((8, 9, 3), (16, 9, 3), 1.0),        # window: more cells than voxels
         ((96, 96, 96), (96, 96, 96), 1.0),   # window of as many cells; a level of more than 152 8^3 tiles
         ((32, 32, 32), (16, 16, 16), 5.0)]   # taps too far apart for a tile: direct kernels


@pytest.mark.parametrize("dims,base,s0", CASES)
@pytest.mark.parametrize("dtype", [abi.CVR_U8, abi.CVR_U16])
def test_levels_match_oracle(ctx, dims, base, s0, dtype):
    wl = scene.workload("cone", n=32, image=8)
    w, h, d = dims
    wl.volume = scene.synth_blobs(w, h, d, dtype, 8, seed=37, noise_max=20.0)
    wl.pyramid = dict(base_dims=base, sigma0=s0, n_levels=5)
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
