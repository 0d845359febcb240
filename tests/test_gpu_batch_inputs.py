"""A batch geometry that has triangles but no vertices is refused by the host,
before any kernel takes a vertex in a bad index's place: wherever it stands in
the batch (past the last geometry's vertices there is nothing), by either entry
point.  The scene stays as it was."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("where", [0, 1, 2])
def test_triangles_without_vertices_are_refused(native, layout, where):
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import engine as E
    from heavyrt_gb300 import workload as wl

    meshes = [wl.soup(5 + k, 40 + k) for k in range(3)]
    verts, idx = [m[0] for m in meshes], [m[1] for m in meshes]
    verts[where] = verts[where][:0]
    s = SceneRT(layout=layout)
    with pytest.raises(E.HrtError, match="triangles but no vertices") as e:
        s.add_geoms_batched(verts, idx)
    assert e.value.status == E.HRT_ERR_INVALID_ARGUMENT
    v, i = np.ascontiguousarray(np.concatenate(verts)), np.concatenate(idx)
    voff = np.cumsum([0] + [len(a) for a in verts]).astype(np.uint64)
    ioff = np.cumsum([0] + [a.size for a in idx]).astype(np.uint64)
    p = [C.c_void_p(a.ctypes.data) for a in (v, voff, i, ioff)]
    first = C.c_uint32()
    st = E.lib().hrt_add_geoms_triangles3f_batched(s._h, 3, p[0], p[1], p[2], p[3], 1, 16, C.byref(first))
    assert st == E.HRT_ERR_INVALID_ARGUMENT and "no vertices" in s.ctx.last_error()
    assert s.GetGeomNum() == 0
    verts[where], idx[where] = verts[where][:0], idx[where][:0]  # neither: a geometry without triangles
    assert s.add_geoms_batched(verts, idx) == [0, 1, 2]
    s.AddInstance((where + 1) % 3)
    s.CommitScene()
    k = (where + 1) % 3
    rays = wl.rays_at_triangles(2, verts[k], idx[k], 64)
    assert (s.RayQuery_NearestHit(rays)["geomId"] == k).any()
    s.close()
