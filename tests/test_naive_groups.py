"""The naive accelerator skips groups of triangles that no ray of a warp can
hit: its answers against the all-pairs loop (pbg_intersect_naive_noalloc) on
rays and triangles where a loose bound would lose a hit -- grazing rays,
slivers, far origins, extreme scales, ties -- for batches that split the
groups and batches that do not."""
import ctypes as C

import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def all_pairs(lib, tris, rays):
    import torch
    fn = lib.pbg_intersect_naive_noalloc
    fn.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_int64] + [C.c_void_p] * 5
    n = rays.shape[1]
    v = torch.from_numpy(np.ascontiguousarray(tris)).cuda()
    o4 = torch.from_numpy(np.ascontiguousarray(rays[[0, 1, 2, 6]].T)).cuda()
    d4 = torch.from_numpy(np.ascontiguousarray(rays[[3, 4, 5, 7]].T)).cuda()
    prim = torch.empty(n, dtype=torch.int32, device="cuda")
    out = [torch.empty(n, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    assert fn(v.data_ptr(), len(tris), o4.data_ptr(), d4.data_ptr(), n, prim.data_ptr(),
              *[x.data_ptr() for x in out], None) == 0
    torch.cuda.synchronize()
    return [prim.cpu().numpy()] + [x.cpu().numpy() for x in out]


def soup(g, n, scale, thin):
    """Triangles about a jittered surface; a third of them slivers when thin."""
    c = g.uniform(-1, 1, (n, 1, 3)) * np.array([4.0, 0.2, 4.0])
    v = c + g.normal(size=(n, 3, 3)) * 0.1
    if thin:
        k = g.random(n) < 0.35
        v[k, 2] = v[k, 1] + g.normal(size=(k.sum(), 3)) * (10.0 ** g.uniform(-7, -2, (k.sum(), 1)))
        k = g.random(n) < 0.1
        v[k, 1] = v[k, 0]  # coincident vertices
        v[::17, :, 1] = 0.0  # and some exactly coplanar
    return (v * scale).astype(np.float32).reshape(n, 9)


def ray_set(g, tris, n, scale):
    """Random, axis-parallel, far and grazing rays, some of them segments."""
    v = tris.reshape(-1, 3, 3).astype(np.float64)
    t = v[g.integers(0, len(v), n)]
    w = g.dirichlet([1, 1, 1], n)[:, :, None]
    p = (t * w).sum(1)                      # a point of a triangle
    e = t[:, 1] - t[:, 0] + (t[:, 2] - t[:, 0]) * g.normal(size=(n, 1))
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-300)
    kind = g.integers(0, 4, n)[:, None]
    size = np.linalg.norm(e, axis=1, keepdims=True) + 1e-30
    graze = e / size + nrm * (10.0 ** g.uniform(-9, -1, (n, 1))) * g.choice([-1, 1], (n, 1))
    d = np.where(kind == 0, graze, g.normal(size=(n, 3)))
    d = np.where(kind == 1, np.eye(3)[g.integers(0, 3, n)] * g.choice([-1.0, 1.0], (n, 1)), d)
    d *= 10.0 ** g.uniform(-2, 2, (n, 1))
    back = np.where(kind == 2, 10.0 ** g.uniform(1, 5, (n, 1)), g.uniform(0, 6, (n, 1))) * scale
    o = p + e * g.normal(size=(n, 1)) * 0.3 - d / np.linalg.norm(d, axis=1, keepdims=True) * back
    r = np.empty((8, n), np.float32)
    r[0:3], r[3:6] = o.T, d.T
    r[6] = np.where(g.random(n) < 0.3, 1e-3 * scale, 0)
    r[7] = np.where(g.random(n) < 0.3, g.uniform(0, 8, n) * scale, np.inf)
    r[6, ::41] = -np.inf
    return r


@pytest.mark.parametrize("ntri,n,scale,thin", [(1, 33, 1.0, False), (31, 257, 1.0, True), (33, 4096, 1.0, True),
                                               (700, 70000, 1.0, True), (2500, 3000, 1e-6, True),
                                               (2500, 3000, 1e6, True), (300, 2000, 1e-12, True),
                                               (300, 2000, 1e12, True), (3000, 200, 1.0, False)])
def test_skipping_keeps_every_hit(gpu_lib, ntri, n, scale, thin):
    g = np.random.default_rng(ntri * 31 + n)
    tris = soup(g, ntri, scale, thin)
    if ntri > 100:
        tris[5::50] = tris[4::50][:len(tris[5::50])]  # exact ties
    rays = ray_set(g, tris, n, scale)
    want = all_pairs(gpu_lib.lib(), tris, rays)
    acc = A.MakeAccelerator("naive", tris)
    got = acc.Intersect(rays.copy())
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(acc.IntersectP(rays) == ord("1"), want[0] >= 0)
    mask = g.random(n) < 0.5
    occ = acc.IntersectP(rays, hit=mask.copy())
    np.testing.assert_array_equal(occ == ord("1"), (want[0] >= 0) & mask)
    acc.close()


def test_sphere_scene(gpu_lib):
    cfg = S.config_small_naive()
    g = np.random.default_rng(2)
    for rays in (cfg["rays"], ray_set(g, cfg["tris"], 50000, 1.0)):
        want = all_pairs(gpu_lib.lib(), cfg["tris"], rays)
        acc = A.MakeAccelerator("naive", cfg["tris"])
        for a, b in zip(acc.Intersect(rays.copy()), want):
            np.testing.assert_array_equal(a, b)
        acc.close()
