"""rayhierarchy's leaf tests skip triangles that a whole leaf certainly misses
and hold exact tests back: its answers against the naive accelerator for rays
through edges, vertices and slivers, tied triangles, bounded segments, and
both forms of the kernel (a leaf per warp, a pair per warp).  At scales of
1e12 these rays' products overflow to NaN, and answers depend on order."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402

pytestmark = pytest.mark.gpu
LINE = 1 << 19


def surface(g, side, scale):
    """A bumpy grid, a third of its triangles turned into slivers, some doubled."""
    x, y = np.meshgrid(np.linspace(-4, 4, side + 1), np.linspace(-4, 4, side + 1))
    p = np.stack([x, g.normal(size=x.shape) * 0.15, y], -1)
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[:-1, 1:], p[1:, 1:]
    v = np.concatenate([np.stack([a, b, c], -2).reshape(-1, 3, 3), np.stack([c, b, d], -2).reshape(-1, 3, 3)])
    k = g.random(len(v)) < 0.3
    v[k, 2] = v[k, 1] + (v[k, 0] - v[k, 1]) * g.uniform(0, 1, (k.sum(), 1)) + g.normal(size=(k.sum(), 3)) * 10.0 ** g.uniform(-7, -2, (k.sum(), 1))
    v = np.concatenate([v, v[::29]])
    return (v * scale).astype(np.float32).reshape(-1, 9)


def aimed(g, tris, n, scale):
    """Rays from a few eyes through points on the triangles' edges, at their
    vertices or inside, ordered by target so that neighbours stay together."""
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    t = v[np.sort(g.integers(0, len(v), n))]
    w = g.dirichlet([1, 1, 1], n)
    w[g.random(n) < 0.4, 0] = 0.0                      # an edge
    w[g.random(n) < 0.1] = np.eye(3)[g.integers(0, 3)]  # a vertex
    p = (t * (w / w.sum(1, keepdims=True))[:, :, None]).sum(1)
    eye = np.array([[0, 9, 1], [6, 0.4, 0], [-5, 2, -5], [0.3, 30, 0.1]])[(np.arange(n) * 4) // n] * scale
    d = (p - eye) * np.where(g.random((n, 1)) < 0.2, 10.0 ** g.uniform(-6, 6, (n, 1)), 1.0)
    r = np.empty((8, n), np.float32)
    r[0:3], r[3:6], r[6] = eye.T, d.T, 0
    r[7] = np.where(g.random(n) < 0.3, 1.0, np.inf)
    return r


@pytest.mark.parametrize("n,scale", [(33, 1.0), (20000, 1.0), (20000, 1e-5), (20000, 1e5), (20000, 1e8), (LINE, 1.0),
                                     (LINE + 33, 1.0)])
def test_leaf_tests(gpu_lib, n, scale):
    g = np.random.default_rng(n)
    tris = surface(g, 40, scale)
    rays = aimed(g, tris, n, scale)
    ref, acc = A.MakeAccelerator("naive", tris), A.MakeAccelerator("rayhierarchy", tris)
    for a, b in zip(acc.Intersect(rays.copy()), ref.Intersect(rays.copy())):
        np.testing.assert_array_equal(a, b)
    back = rays.copy()  # from a little short of the targets to the eyes: origins spread, directions meet
    unit = np.linalg.norm(rays[3:6], axis=0)
    back[0:3] = rays[0:3] + rays[3:6] / unit * np.linalg.norm(rays[0:3], axis=0) * 0.7
    back[3:6], back[7] = -rays[3:6], np.inf
    np.testing.assert_array_equal(acc.IntersectP(back), ref.IntersectP(back))
    np.testing.assert_array_equal(acc.IntersectP(rays), ref.IntersectP(rays))
    acc.close()
    ref.close()
