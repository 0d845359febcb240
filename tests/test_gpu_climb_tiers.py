"""The walks above the slices at their edges: one tier and two, the last slice
or group with a leaf or two, codes shared by many triangles (fewer leaves than
triangles), and geometries of a batch that lie across slices and groups; boxes
and counts of every node against the oracle, after the build and after a refit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n, per_cell):
    rng = np.random.default_rng(n + per_cell)
    at = rng.uniform(-1, 1, (max(1, n // per_cell), 3))[rng.integers(0, max(1, n // per_cell), n)]
    verts = np.ones((3 * n, 4), np.float32)
    verts[:, :3] = (at[:, None, :] + rng.uniform(-2e-4, 2e-4, (n, 3, 3))).reshape(-1, 3)
    verts[:2, :3] = [[-1, -1, -1], [1, 1, 1]]
    return verts, np.arange(3 * n, dtype=np.uint32)


def _check(s, gid, o, what):
    from heavyrt_gb300 import engine as E

    np.testing.assert_array_equal(s.export(gid, E.EXPORT_LR_NODES).view(np.uint32).reshape(-1),
                                  np.ascontiguousarray(o.lr_nodes()).view(np.uint32).reshape(-1), err_msg=what)
    np.testing.assert_array_equal(s.export(gid, E.EXPORT_LR_COUNTS), o.lr_counts(), err_msg=what)


@pytest.mark.parametrize("n,per_cell", [(513, 1), (600, 40), (16384, 1), (16385, 1), (16900, 1), (40000, 40), (33000, 1),
                                        (525000, 1)])
def test_nodes_above_the_slices(native, n, per_cell):
    from heavyrt_gb300 import SceneRT
    from oracle import oracle as orc

    v, idx = _mesh(n, per_cell)
    o = orc.OracleBVH(v, idx)
    assert (np.diff(np.append(o.run_starts(), n)) <= 127).all()
    s = SceneRT()
    gid = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    _check(s, gid, o, f"{n} triangles")
    s.close()


@pytest.mark.parametrize("n", [700, 17000])
def test_nodes_after_a_refit(native, n):
    """A refit to the same vertices rewrites the same tree."""
    from heavyrt_gb300 import BUILD_REFIT, SceneRT
    from oracle import oracle as orc

    v, idx = _mesh(n, 1)
    o = orc.OracleBVH(v, idx)
    s = SceneRT()
    gid = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    moved = v * np.array([1, 1, 1, 1], np.float32)
    moved[:, :3] += 0.25
    for verts in (moved, v):
        s.UpdateGeom_Triangles3f(gid, verts, len(verts), idx, idx.size, BUILD_REFIT, 16)
    _check(s, gid, o, f"{n} triangles")
    s.close()


@pytest.mark.parametrize("sizes", [[400, 300], [1] * 600 + [1000], [9000, 9000, 20, 40000, 1, 500, 600]])
def test_geometries_of_a_batch(native, sizes):
    from heavyrt_gb300 import SceneRT
    from oracle import oracle as orc

    meshes = [_mesh(n, 1 + k % 3) for k, n in enumerate(sizes)]
    s = SceneRT()
    ids = s.add_geoms_batched([m[0] for m in meshes], [m[1] for m in meshes])
    for k in sorted({0, 1, len(sizes) // 2, len(sizes) - 2, len(sizes) - 1}):
        _check(s, ids[k], orc.OracleBVH(*meshes[k]), f"geometry {k}")
    s.close()
