"""Several SGD steps of one call, whose launches overlap: bit for bit the same
steps taken one call at a time (partial gradients are summed in a fixed order),
and the float64 loop of momentum SGD over the oracle's gradients."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import _lib as L  # noqa: E402
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
TRIS = S.displaced_icospheres(seed=3, n_inst=60, box=16.0)["tris"]
NPARAM = 28032
LR, MOMENTUM = 0.05, 0.9


def learner(batch, corner=False):
    """A scene with `batch` records, and the records' rays and labels."""
    import torch
    acc = A.MakeAccelerator("ray-bvh", TRIS)
    rays = S.random_rays(12 * batch, -8.0, 8.0, seed=batch)
    if corner:
        rays[0:3], rays[3:6] = TRIS.reshape(-1, 3).min(0)[:, None], np.abs(rays[3:6])
    prim = acc.Intersect(rays.copy())[0]
    keep = np.flatnonzero(prim >= 0)
    assert len(keep) >= batch
    rays, prim = rays[:, keep[:batch]], prim[keep[:batch]]
    o4, d4 = (torch.from_numpy(np.ascontiguousarray(rays[k].T)).cuda() for k in ([0, 1, 2, 6], [3, 4, 5, 7]))
    label = torch.empty(batch, dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    acc.clusters_of_device(torch.from_numpy(prim).cuda(), label)
    acc.learn_enable(True, batch=batch, records=batch, lr=LR, momentum=MOMENTUM, seed=5, queries=1)
    out = [torch.empty(batch // 4, dtype=torch.int32, device="cuda")] + [torch.empty(batch // 4, device="cuda") for _ in range(3)]
    for k in range(4):  # a batch appends at most a quarter of the records kept
        part = slice(k * batch // 4, (k + 1) * batch // 4)
        a, b = o4[part].contiguous(), d4[part].contiguous()
        torch.cuda.synchronize()
        acc.intersect_device(a, b, *out)
    assert acc.learn_stats()["records"] == batch
    return acc, rays, label.cpu().numpy().astype(np.int32)


def params(acc, new=None):
    """The parameters, read; or set, which also zeroes their momentum."""
    w = np.zeros(NPARAM, np.float32) if new is None else new
    L.check(L.lib().pbg_learn_params_io(acc.handle, w.ctypes.data_as(L.C.c_void_p), 1 if new is None else 0), "pbg_learn_params_io")
    return w


@pytest.mark.parametrize("batch", [128] + [512 * k for k in range(1, 17)] + [128 * 155])
def test_chained_steps_are_single_steps(gpu_lib, batch):
    acc, _, _ = learner(batch)
    start = params(acc)
    for steps in (1, 2, 3, 5, 8):
        params(acc, start)
        for _ in range(steps):
            acc.learn_train(1)
        want = params(acc)
        assert not np.array_equal(want, start)
        for _ in range(10):
            params(acc, start)
            acc.learn_train(steps)
            np.testing.assert_array_equal(params(acc), want)
    acc.close()


def features(rays):
    """The network's inputs for rays from the least corner of the scene's box,
    where every sine is 0 and every cosine 1 (the device's sines are fast ones,
    which no restatement meets to BF16)."""
    d = rays[3:6].T.astype(np.float64)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    x = np.zeros((rays.shape[1], 112))
    x[:, 0:3], x[:, 3:6], x[:, 6:9] = -1, d, np.minimum(1.0 / np.maximum(d, 1.0 / 16.0), 16) / 16
    x[:, 10:105:2] = 1
    return x.astype(np.float32)


@pytest.mark.parametrize("batch,steps", [(128, 1), (512, 2), (1536, 8), (8192, 3), (128 * 155, 2)])
def test_steps_match_the_oracle(gpu_lib, batch, steps):
    """Each step's gradient is within 2e-2 of a block's largest (values on a
    BF16 rounding boundary); as much again for what earlier steps moved."""
    from oracle import mlp_oracle as M
    acc, rays, label = learner(batch, corner=True)
    start = params(acc)
    acc.learn_train(steps)
    got = params(acc).astype(np.float64) - start
    x = features(rays)
    w, v = start.astype(np.float64), np.zeros(NPARAM)
    for _ in range(steps):
        g, _ = M.gradients(w.astype(np.float32), x, label)
        v = MOMENTUM * v + g
        w = w - LR * v
    k = 0
    for name, n in zip(["W1", "b1", "W2", "b2", "W3", "b3"], M.SIZES):
        a, b = got[k:k + n], (w - start)[k:k + n]
        err = np.abs(a - b).max() / max(np.abs(b).max(), 1e-12)
        assert err < 4e-2, f"{name}: relative error {err}"
        k += n
    acc.close()
