"""Bounds that are NaN reject nothing in pbrt's triangle test: every walk of
ray-bvh, the automatic choice and the scene set's answer such rays as the CPU
loop over all triangles does."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
TRIS = S.terrain_icospheres(seed=2, grid=20, n_spheres=2)["tris"]


@pytest.mark.parametrize("walk", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("n", [31, 5000])
def test_nan_bounds(gpu_lib, oracle, walk, n):
    rays = S.random_rays(n, -6.0, 6.0, seed=n)
    rays[7, ::3] = np.nan
    rays[6, 1::4] = np.nan
    want, occ = oracle.nearest(TRIS, rays.copy()), oracle.anyhit(TRIS, rays)
    assert (want[0][::3] >= 0).any()
    acc = A.MakeAccelerator("ray-bvh", TRIS, {"walk": walk})
    for _ in range(2):  # the automatic walk before and after the scene has its eight-wide tree
        for a, b in zip(acc.Intersect(rays.copy()), want):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(acc.IntersectP(rays) == ord("1"), occ != 0)
    acc.close()


@pytest.mark.parametrize("walk", [1, 2, 3, 4])
def test_nan_bounds_in_a_set(gpu_lib, oracle, walk):
    import torch
    from pbrt_gb300 import batch as B
    rays = S.random_rays(2000, -6.0, 6.0, seed=3)
    rays[7, ::3] = np.nan
    dev = [torch.from_numpy(np.ascontiguousarray(rays[k].T)).cuda() for k in ([0, 1, 2, 6], [3, 4, 5, 7])]
    off = np.array([0, 1200, 2000], np.int64)
    prim, occ = torch.empty(2000, dtype=torch.int32, device="cuda"), torch.empty(2000, dtype=torch.uint8, device="cuda")
    t, b1, b2 = (torch.empty(2000, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    scenes = [TRIS, TRIS[:700]]
    B.SceneSet(scenes).trace(o4n=dev[0], d4n=dev[1], near_offsets=off, prim=prim, t=t, b1=b1, b2=b2, o4s=dev[0], d4s=dev[1],
                             occ_offsets=off, occ=occ, walk=walk)
    torch.cuda.synchronize()
    for k, tris in enumerate(scenes):
        part = slice(off[k], off[k + 1])
        r = np.ascontiguousarray(rays[:, part])
        want = oracle.nearest(tris, r.copy())
        for a, b in zip((prim, t, b1, b2), want):
            np.testing.assert_array_equal(a.cpu().numpy()[part], b)
        np.testing.assert_array_equal(occ.cpu().numpy()[part] != 0, oracle.anyhit(tris, r) != 0)


@pytest.mark.parametrize("walk", [0, 1, 2, 3, 4, 5, 6])
def test_walk_goes_on_behind_a_nan_hit(gpu_lib, oracle, walk):
    """A triangle so small that its divisor is subnormal is hit at a distance
    that is NaN, after which pbrt accepts whatever it hits: what lies behind,
    of higher indices, is found by every walk."""
    tiny = np.array([[0, 0, 0, 1e-15, 0, 0, 0, 1e-27, 0]], np.float32)
    g = np.random.default_rng(1)
    a = g.uniform(-3, 3, (400, 2))
    behind = np.zeros((400, 3, 3))
    behind[:, :, 2] = g.uniform(1, 9, (400, 1))
    behind[:, :, :2] = a[:, None] * 0.02 + np.array([[-1, -1], [1.5, -1], [-1, 1.5]]) * g.uniform(0.02, 4, (400, 1, 1))
    tris = np.concatenate([tiny, behind.reshape(400, 9).astype(np.float32)])
    rays = np.zeros((8, 40), np.float32)
    rays[2], rays[5], rays[7] = -1e-5, 1.0, np.inf
    want = oracle.nearest(tris, rays.copy())
    assert np.isnan(oracle.nearest(tiny, rays.copy())[1]).all() and (want[0] > 0).all()
    acc = A.MakeAccelerator("ray-bvh", tris, {"walk": walk})
    for _ in range(2):
        for a, b in zip(acc.Intersect(rays.copy()), want):
            np.testing.assert_array_equal(a, b)
        assert (acc.IntersectP(rays) == ord("1")).all()
    acc.close()
