"""The walks that an untuned ray-bvh scene chooses by the batch's size: the
same answers as one thread per ray on both sides of the lines, before and after
the scene has its eight-wide tree."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
SHADOW, CAMERA = 1 << 18, 3 << 18  # the lines


@pytest.mark.parametrize("n", [1, 33, SHADOW - 1, SHADOW, CAMERA - 1, CAMERA])
def test_choice_by_size(gpu_lib, n):
    tris = S.terrain_icospheres(seed=2, grid=48, n_spheres=6)["tris"]
    side = int(np.ceil(np.sqrt(n)))
    rays = np.ascontiguousarray(S.pinhole_rays(side, side, (0.0, 9.0, -14.0), (0.0, 0.0, 0.0), 50.0, jitter_seed=n)[:, :n])
    auto, one = A.MakeAccelerator("ray-bvh", tris), A.MakeAccelerator("ray-bvh", tris, {"walk": 1})
    want = one.Intersect(rays.copy())
    for a, b in zip(auto.Intersect(rays.copy()), want):  # no eight-wide tree yet
        np.testing.assert_array_equal(a, b)
    assert auto.stats()["wide_nodes"] == 0
    np.testing.assert_array_equal(auto.IntersectP(rays), one.IntersectP(rays))
    assert auto.stats()["wide_nodes"] > 0  # the shadow batch built it
    for a, b in zip(auto.Intersect(rays.copy()), want):
        np.testing.assert_array_equal(a, b)
    auto.close()
    one.close()
