"""The fused training step at the edges of its tiling: one tile, a few, and
more tiles than the GPU has SMs (a CTA then accumulates several)."""
import ctypes as C

import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import _lib as L  # noqa: E402
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
NPARAM = 28032


@pytest.mark.parametrize("B", [128, 384, 128 * 155])
def test_gradients_at_tile_edges(gpu_lib, B):
    from oracle import mlp_oracle as M
    lib = gpu_lib.lib()
    acc = A.MakeAccelerator("ray-bvh", S.displaced_icospheres(seed=3, n_inst=4, box=6.0)["tris"])
    acc.learn_enable(True, seed=7)
    params = np.empty(NPARAM, np.float32)
    io = lambda a, get: lib.pbg_learn_params_io(acc.handle, C.c_void_p(a.ctypes.data), C.c_int32(get))  # noqa: E731
    assert io(params, 1) == 0
    g = np.random.default_rng(B)
    x = g.normal(size=(B, 112)).astype(np.float32)
    x[:, 105:] = 0
    y = g.integers(0, 256, size=B).astype(np.int32)
    grads, loss = np.empty(NPARAM, np.float32), C.c_float()
    rc = lib.pbg_learn_gradients(acc.handle, C.c_void_p(x.ctypes.data), C.c_void_p(y.ctypes.data), C.c_int32(B),
                                 C.c_void_p(grads.ctypes.data), C.byref(loss))
    assert rc == 0, L.last_error()
    want, wloss = M.gradients(params, x, y)
    assert abs(loss.value - wloss) <= 1e-3 * max(1.0, abs(wloss))
    k = 0
    for name, n in zip(["W1", "b1", "W2", "b2", "W3", "b3"], M.SIZES):
        a, b = grads[k:k + n].astype(np.float64), want[k:k + n]
        # both round the same values to bf16; a value on a rounding boundary may go the other way (2^-8 of one term)
        err = np.abs(a - b).max() / max(np.abs(b).max(), 1e-12)
        assert err < 2e-2, f"{name}: relative error {err}"
        k += n
    after = np.empty(NPARAM, np.float32)
    assert io(after, 1) == 0 and np.array_equal(after, params)  # gradients leave the parameters alone
    acc.close()
