"""The training step's own rules: features that are only float-aligned take
scalar loads, an update writes the packed operands of the parameters that it
changes, and epochs alternate between two permutation buffers."""
import ctypes as C

import numpy as np
import pytest

from cpp_volume_rendering_gb300 import abi

pytestmark = pytest.mark.gpu


def device_memory():
    """The tests' own device buffers, or a skip."""
    try:
        from tests.devmem import DeviceMemory
        return DeviceMemory()
    except (ImportError, RuntimeError) as e:
        pytest.skip(f"no CUDA runtime for test buffers: {e}")


def data(n, seed):
    rng = np.random.default_rng(seed)
    return (rng.normal(0, 1, size=(n, 48)).astype(np.float32), rng.uniform(0, 1, size=(n, 2)).astype(np.float32))


@pytest.mark.parametrize("n", [1, 127, 128, 129, 500])
@pytest.mark.parametrize("shift", [0, 1, 2])
def test_gradients_of_features_at_any_float(ctx, n, shift):
    lib, h = abi.load(), ctx.h
    abi.check(lib.cvr_mlp_init(h, 3), h)
    x, t = data(n, n)
    ref = np.zeros(abi.MLP_PARAMS, np.float32)
    abi.check(lib.cvr_mlp_gradients(h, abi.fptr(x), abi.fptr(t), n, abi.fptr(ref), None), h)
    buf = device_memory()
    try:
        xd = buf.upload(np.concatenate([np.zeros(shift, np.float32), x.ravel()]))
        td, gd = buf.upload(t), buf.alloc(4 * abi.MLP_PARAMS)
        xp = C.c_void_p(xd.value + 4 * shift)
        abi.check(lib.cvr_mlp_gradients_noalloc(h, xp, td, n, gd, None), h)
        abi.check(lib.cvr_mlp_check(h), h)
        assert np.array_equal(buf.download(gd, abi.MLP_PARAMS), ref)
    finally:
        buf.close()


@pytest.mark.parametrize("n,batch", [(1, 128), (128, 128), (300, 128), (1000, 256)])
def test_an_update_writes_the_packed_operands(ctx, n, batch):
    lib, h = abi.load(), ctx.h
    abi.check(lib.cvr_mlp_init(h, 4), h)
    x, t = data(n, n + 7)
    abi.check(lib.cvr_mlp_set_training_data(h, abi.fptr(x), abi.fptr(t), n), h)
    abi.check(lib.cvr_mlp_train(h, 3, batch, 1e-2, 11, None), h)
    trained, packed = np.zeros((n, 2), np.float32), np.zeros((n, 2), np.float32)
    abi.check(lib.cvr_mlp_forward(h, abi.fptr(x), n, abi.fptr(trained)), h)
    p = np.zeros(abi.MLP_PARAMS, np.float32)
    abi.check(lib.cvr_mlp_get_params(h, abi.fptr(p), abi.MLP_PARAMS), h)
    abi.check(lib.cvr_mlp_set_params(h, abi.fptr(p), abi.MLP_PARAMS), h)  # packs every parameter anew
    abi.check(lib.cvr_mlp_forward(h, abi.fptr(x), n, abi.fptr(packed)), h)
    assert np.array_equal(trained, packed)


@pytest.mark.parametrize("n", [200, 1024])
def test_one_run_equals_the_runs_of_its_epochs(ctx, n):
    """The first epoch of a run depends on the seed alone: a run of one epoch
    and the first of three give the same loss, and the losses of a run repeat."""
    lib, h = abi.load(), ctx.h
    x, t = data(n, n + 1)
    abi.check(lib.cvr_mlp_init(h, 6), h)
    abi.check(lib.cvr_mlp_set_training_data(h, abi.fptr(x), abi.fptr(t), n), h)
    runs = []
    for epochs in (1, 3, 3):
        abi.check(lib.cvr_mlp_init(h, 6), h)
        loss = np.zeros(epochs, np.float32)
        abi.check(lib.cvr_mlp_train(h, epochs, 128, 1e-2, 5, abi.fptr(loss)), h)
        runs.append(loss)
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[1], runs[2])
