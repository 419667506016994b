"""The packet walks' fused slab test on rays and scenes of extreme size, as the
eight-wide walks': each answer is the one-thread-per-ray walk's (separate
subtraction and product) or the loop's over all triangles, and none of the
former's hits is lost."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def extreme_rays(g, n, scale):
    """Random rays, then zero and negative-zero components, tiny and long
    directions, origins inside, at the edge and far outside, bounded t."""
    r = np.zeros((8, n))
    r[0:3] = g.uniform(-8, 8, (3, n)) * scale
    r[3:6] = g.normal(size=(3, n))
    k = np.arange(n)
    for a in range(3):
        r[3 + a, k % 7 == a] = 0.0
        r[3 + a, k % 11 == a] = -0.0
        r[3 + a, k % 13 == a] *= 1e-30
        r[3 + a, k % 17 == a] *= 1e-12
    r[3:6] *= np.where(k % 5 == 0, 10.0 ** g.uniform(-15, 15, n), 1.0)
    back = np.where(k % 6 == 0, 10.0 ** g.uniform(0, 6, n), 0.0) * scale
    r[0:3] -= r[3:6] / np.maximum(np.linalg.norm(r[3:6], axis=0), 1e-300) * back
    r[7] = np.where(k % 4 == 0, g.uniform(0, 10, n) * scale, np.inf)
    r[6] = np.where(k % 9 == 0, -np.inf, 0.0)
    return r.astype(np.float32)


@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e7])
@pytest.mark.parametrize("walk", [3, 4])
def test_extreme_rays(gpu_lib, walk, scale):
    g = np.random.default_rng(11)
    tris = (S.displaced_icospheres(seed=3, n_inst=6, box=8.0)["tris"].astype(np.float64) * scale).astype(np.float32)
    rays = extreme_rays(g, 20000, scale)

    def answers(kind, **opts):
        acc = A.MakeAccelerator(kind, tris, opts)
        hit, occ = np.stack([np.asarray(x, np.float64) for x in acc.Intersect(rays.copy())]), acc.IntersectP(rays)
        acc.close()
        return hit, occ == ord("1")

    pairs, pairs_occ = answers("naive")
    ref, ref_occ = answers("ray-bvh", walk=1)
    got, occ = answers("ray-bvh", walk=walk)
    assert (ref[0] >= 0).any()
    assert ((got == ref).all(0) | (got == pairs).all(0)).all()
    assert (occ | ~ref_occ).all() and (pairs_occ | ~occ).all()
