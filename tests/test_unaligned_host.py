"""Host arrays off a word boundary (rows of a packed file, say) go to the GPU
and back by copies: the answers of aligned arrays, from every host call."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import _lib as L  # noqa: E402
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


def shifted(a, by):
    """a in memory that starts `by` bytes past a word boundary."""
    raw = np.zeros(a.nbytes + 8, np.uint8)
    b = raw[by:by + a.nbytes].view(a.dtype).reshape(a.shape)
    b[...] = a
    assert b.ctypes.data % 4 == by
    return b


@pytest.mark.parametrize("by", [1, 2, 3])
@pytest.mark.parametrize("kind,n", [("naive", 77), ("rayhierarchy", 1000), ("ray-bvh", 4099)])
def test_answers_as_aligned(gpu_lib, kind, n, by):
    acc = A.MakeAccelerator(kind, S.terrain_icospheres(seed=2, grid=16, n_spheres=2)["tris"])
    rays = S.random_rays(n, -6.0, 6.0, seed=by)
    hits = acc.Intersect(rays.copy())
    occ, geo = acc.IntersectP(rays), acc.HitGeometry(rays, *hits)
    assert (hits[0] >= 0).any()
    odd = shifted(rays, by)
    np.testing.assert_array_equal(acc.HitGeometry(rays, *[shifted(x, by) for x in hits]), geo)
    np.testing.assert_array_equal(acc.HitGeometry(odd, *hits), geo)
    np.testing.assert_array_equal(acc.IntersectP(odd), occ)
    out = [shifted(np.zeros_like(x), by) for x in hits]  # results off a boundary too
    h = L.Hits(out[0].ctypes.data_as(L.C.POINTER(L.C.c_int32)), *[A._fptr(x) for x in out[1:]])
    L.check(L.lib().pbg_intersect(acc.handle, L.C.byref(acc._rays_struct(odd, None)), n, L.C.byref(h)), "pbg_intersect")
    for a, b in zip(out, hits):
        np.testing.assert_array_equal(a, b)
    acc.close()
