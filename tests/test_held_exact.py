"""Rays whose every leaf holds many triangles that pass the filter: the walks
queue exact tests (32 at a time, the rest behind), and take the last of tied
triangles, as the naive accelerator does."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402

pytestmark = pytest.mark.gpu


def sheets(g, n, copies):
    """n parallel sheets of two triangles each, every third of them repeated."""
    q = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]], np.float64)
    v = np.stack([q + [0, y, 0] + g.normal(size=(4, 3)) * 1e-4 for y in np.linspace(0, 0.01, n)])
    t = np.concatenate([v[:, [0, 1, 2]], v[:, [0, 2, 3]]])
    return np.concatenate([t] + [t[::3]] * copies).astype(np.float32).reshape(-1, 9)


@pytest.mark.parametrize("n,copies,rays_n", [(1, 0, 1), (3, 40, 33), (40, 3, 4099), (300, 2, 2000)])
def test_many_candidates(gpu_lib, n, copies, rays_n):
    g = np.random.default_rng(n)
    tris = sheets(g, n, copies)
    r = np.zeros((8, rays_n), np.float32)
    r[0:3] = g.uniform(-1, 1, (3, rays_n))
    r[1] = np.where(g.random(rays_n) < 0.5, 3, -3)
    r[3:6] = (g.uniform(-0.9, 0.9, (3, rays_n)) - r[0:3])
    r[4] = -r[1] + 0.005
    r[7] = np.where(g.random(rays_n) < 0.2, g.uniform(0.9, 1.1, rays_n), np.inf)
    ref = A.MakeAccelerator("naive", tris)
    want, occ = ref.Intersect(r.copy()), ref.IntersectP(r)
    for w in (1, 2, 3, 4, 5, 6):
        acc = A.MakeAccelerator("ray-bvh", tris, {"walk": w})
        for a, b in zip(acc.Intersect(r.copy()), want):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(acc.IntersectP(r), occ)
        acc.close()
    ref.close()
