"""Which camera batches an untuned ray-bvh scene walks in packets: by rays,
triangles and samples per pixel, against either of the walks it takes instead.
Packets count their work the same on every run, so an automatic batch that
counts as walk 4 does took it."""
import math

import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
TRIS = S.terrain_icospheres(seed=2, grid=48, n_spheres=6)["tris"]


def line(wide, samples):
    a, b, c = {False: {1: (0, 2, 0), 2: (0, 1.1, 0), 4: (0, 0.85, 0)}, True: {1: (0.9, 4.2, 0), 2: (0.9, 0.8, 1.6), 4: (0.85, 0, 1.15)}}[wide][samples]
    x = math.sqrt(len(TRIS) / 2.0 ** 20)
    return 2.0 ** 20 * (a + b * x + c * x * x)


def work(acc, rays):
    acc.profile(2)
    acc.Intersect(rays.copy())
    w = acc.stats()["work"]
    acc.profile(False)
    return w


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("samples,declared", [(1, 1), (2, 2), (2, 3), (2, None), (4, 4), (4, 16)])
def test_line(gpu_lib, wide, samples, declared):
    at = line(wide, samples)
    for n, packets in ((int(at * 0.99), False), (int(at * 1.01), True)):
        side = math.ceil(math.sqrt(n))
        rays = np.ascontiguousarray(S.pinhole_rays(side, side, (0.0, 9.0, -14.0), (0.0, 0.0, 0.0), 50.0, jitter_seed=n)[:, :n])
        auto, four = A.MakeAccelerator("ray-bvh", TRIS), A.MakeAccelerator("ray-bvh", TRIS, {"walk": 4})
        if declared is not None:
            auto.Preprocess(xres=64, yres=64, samplesPerPixel=declared)
        if wide:
            auto.IntersectP(rays[:, :100].copy())  # the first shadow batch builds the eight-wide tree
        assert (auto.stats()["wide_nodes"] > 0) == wide
        assert (work(auto, rays) == work(four, rays)) == packets
        auto.close()
        four.close()
