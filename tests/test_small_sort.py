"""Small rayhierarchy batches are ordered by one cluster in one launch: the
answers of the naive accelerator at the edges of its capacity, for image,
6-D and origin keys, with masks, and for kept origin orders."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
TRIS = S.terrain_icospheres(seed=2, grid=24, n_spheres=4)["tris"]


def check(acc, ref, rays, mask):
    kw = {} if mask is None else {"hit": mask.copy()}
    near = {} if mask is None else {"hit": mask.copy(), "bounce": 1}
    for a, b in zip(acc.Intersect(rays.copy(), **near), ref.Intersect(rays.copy(), **near)):
        np.testing.assert_array_equal(a, b)
    shadow = rays.copy()
    for turn in range(3):  # a fresh origin order, a kept one, one whose origins moved
        if turn == 1:
            shadow[3:6] = -shadow[[4, 5, 3]]
        if turn == 2:
            shadow[0, -1] += 0.25
        np.testing.assert_array_equal(acc.IntersectP(shadow, **kw), ref.IntersectP(shadow, **kw))


@pytest.mark.parametrize("w,h,masked", [(1, 1, False), (31, 1, True), (33, 1, False), (255, 1, True), (257, 1, False),
                                        (89, 92, True), (8192, 1, True), (8193, 1, False), (8191, 1, False), (3, 2731, True), (161, 119, True),
                                        (240, 273, False), (13107, 5, True), (256, 256, True), (65537, 1, True), (372, 353, True),
                                        (4096, 32, True), (131073, 1, True)])
def test_small_batches(gpu_lib, w, h, masked):
    n = w * h
    g = np.random.default_rng(n)
    side = int(np.ceil(np.sqrt(n)))
    rays = np.ascontiguousarray(S.pinhole_rays(side, side, (0.0, 9.0, -14.0), (0.0, 0.0, 0.0), 50.0, jitter_seed=n)[:, :n])
    mask = g.random(n) < 0.7 if masked else None
    ref = A.MakeAccelerator("naive", TRIS)
    for image in (True, False):
        acc = A.MakeAccelerator("rayhierarchy", TRIS)
        if image and w <= 32768:
            acc.Preprocess(xres=w, yres=h)
        check(acc, ref, rays, mask)
        acc.close()
    ref.close()
