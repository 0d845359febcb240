"""Unused slots of 4-wide nodes take no part in the order in which a nearest-hit
ray visits the others: where two triangles are hit at the same distance, the one
that is reported does not depend on whether the ray also passes through the point
that an unused slot's box is (the origin, or the corner of an 8-bit node's
frame).  On meshes with small whole coordinates the three node formats hold the
same boxes and every rounding is exact, so all formats, and the mesh moved by
whole numbers, give the same hits."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(v, f):
    verts = np.ones((len(v), 4), np.float32)
    verts[:, :3] = v
    return verts, np.asarray(f, np.uint32).reshape(-1)


def _shared_edge():
    """Two triangles with an edge through (1, 1, 1) and one far away: a node with one unused slot."""
    return _mesh([[0, 0, 1], [2, 2, 1], [0, 2, 1], [2, 0, 1], [8, 8, 6], [9, 8, 6], [8, 9, 6]],
                 [[0, 1, 2], [0, 3, 1], [4, 5, 6]])


def _cubes(n):
    corners = np.array(list(itertools.product((0, 1), repeat=3)), np.float32)
    faces = np.array([[0, 1, 3], [0, 3, 2], [4, 6, 7], [4, 7, 5], [0, 4, 5], [0, 5, 1], [2, 3, 7], [2, 7, 6],
                      [0, 2, 6], [0, 6, 4], [1, 5, 7], [1, 7, 3]])
    at = list(itertools.product(range(-n, n), repeat=3))
    return _mesh(np.concatenate([corners + np.array(o, np.float32) for o in at]),
                 np.concatenate([faces + 8 * k for k in range(len(at))]))


def _rays(v):
    """Rays of small whole directions through the mesh's vertices, the middles between them and the origin."""
    rng = np.random.default_rng(8)
    p = v[:, :3]
    n = 4000
    a, b = p[rng.integers(0, len(p), n)], p[rng.integers(0, len(p), n)]
    at = np.where(rng.random((n, 1)) < 0.5, a, 0.5 * (a + b))
    at[::5] = 0.0
    d = rng.integers(-2, 3, (n, 3)).astype(np.float32)
    d[(d == 0).all(axis=1)] = 1.0
    d[:8], at[:8] = 1.0, 0.0
    r = np.zeros((n, 8), np.float32)
    r[:, :3], r[:, 4:7], r[:, 7] = at - d * rng.integers(1, 5, (n, 1)), d, 1e6
    return r


@pytest.mark.parametrize("quality", [False, True])
@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("mesh", ["shared_edge", "cubes"])
def test_ties_do_not_depend_on_unused_slots(native, mesh, test, quality):
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import engine as E

    v, idx = _shared_edge() if mesh == "shared_edge" else _cubes(3)
    rays = _rays(v)
    want = None
    for shift in ((0, 0, 0), (64, 32, 16)):
        w, r = v.copy(), rays.copy()
        w[:, :3] += np.array(shift, np.float32)
        r[:, :3] += np.array(shift, np.float32)
        for layout in (1, 2, 3):
            s = SceneRT(layout=layout, triangle_test=test)
            if quality:
                s.set_bvh4_merge(1)
                s.set_morton_frame(E.MORTON_CUBIC)
                s.set_bvh4_collapse(E.BVH4_COLLAPSE_LARGEST_FIRST)
            g = s.AddGeom_Triangles3f(w, len(w), idx, idx.size, vByteStride=16)
            s.AddInstance(g)
            s.CommitScene()
            got = s.RayQuery_NearestHit(r)
            if want is None:
                want = got
                assert 0 < (got["geomId"] == 0).sum() < len(r)
            np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32), err_msg=f"{layout} {shift}")
            s.close()
