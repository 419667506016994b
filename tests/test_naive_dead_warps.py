"""Warps of the naive kernel without a live ray -- masked out, or past the end
of the batch in its last CTA -- load and test nothing; the live ones answer as
without a mask."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
TRIS = S.terrain_icospheres(seed=2, grid=20, n_spheres=2)["tris"]
FLAT = np.repeat(TRIS[:, :3], 3, axis=0).reshape(-1, 9)[:70]  # coincident vertices: tested by every ray
GROUPS = (len(TRIS) + 31) // 32 + 3


def work(acc, call):
    acc.profile(2)
    call()
    w = acc.stats()["work"]
    acc.profile(False)
    return w


@pytest.mark.parametrize("n,live", [(1, []), (32, [0]), (33, [1]), (4096, []), (4096, [5]), (5000, [0, 77, 156]), (70001, [9, 2187])])
def test_dead_warps(gpu_lib, n, live):
    acc = A.MakeAccelerator("naive", np.concatenate([TRIS, FLAT]))
    rays = S.random_rays(n, -6.0, 6.0, seed=n)
    mask = np.zeros(n, bool)
    for w in live:
        mask[32 * w:32 * w + 32:3] = True
    want = acc.Intersect(rays.copy())
    occ = acc.IntersectP(rays)
    got = []
    near = work(acc, lambda: got.extend(acc.Intersect(rays.copy(), hit=mask.copy(), bounce=1)))
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, np.where(mask, b, -1 if b.dtype == np.int32 else 0))
    any_ = work(acc, lambda: got.append(acc.IntersectP(rays, hit=mask.copy())))
    np.testing.assert_array_equal(got[-1], np.where(mask, occ, ord("0")))
    for w in (near, any_):
        assert w["leaves"] <= GROUPS * len(live)
        assert (w["filter_tests"] > 0) == bool(live)
    whole = work(acc, lambda: acc.Intersect(rays.copy()))  # the last CTA's warps past the end
    assert whole["leaves"] <= GROUPS * ((n + 31) // 32)
    acc.close()
