"""Geometries built by one block, at the edges of its sort, its runs and its
range, against the oracle bit for bit; and instance trees over instances with
and without triangles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513, 1024, 2047, 2049, 4095, 4096, 4097]


def _stages(s, gid):
    from heavyrt_gb300 import engine as E

    what = {"box": E.EXPORT_SCENE_BOX, "unsorted": E.EXPORT_MORTON_UNSORTED, "sorted": E.EXPORT_MORTON_SORTED,
            "codes": E.EXPORT_COMPRESSED, "runs": E.EXPORT_RUN_STARTS, "lr": E.EXPORT_LR_NODES,
            "counts": E.EXPORT_LR_COUNTS, "order": E.EXPORT_PRIM_INDICES, "idx": E.EXPORT_SORTED_INDICES}
    return {k: np.ascontiguousarray(s.export(gid, w)).view(np.uint32).reshape(-1) for k, w in what.items()}


def _expected(o):
    want = {"box": o.scene_box(), "unsorted": o.morton_unsorted(), "sorted": o.morton_sorted(), "codes": o.compressed(),
            "runs": o.run_starts(), "lr": o.lr_nodes(), "counts": o.lr_counts(), "order": o.prim_indices(),
            "idx": o.sorted_indices()}
    return {k: np.ascontiguousarray(w).view(np.uint32).reshape(-1) for k, w in want.items()}


def _mesh(n, shared):
    """n triangles; shared: on a few vertices, so that codes repeat."""
    from heavyrt_gb300 import workload as wl

    if not shared:
        return wl.soup(300 + n, n, off=0.03)
    rng = np.random.default_rng(n)
    verts = np.ones((max(3, n // 7), 4), np.float32)
    verts[:, :3] = rng.integers(-8, 9, (len(verts), 3)) / 8.0
    return verts, rng.integers(0, len(verts), 3 * n).astype(np.uint32)


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_stages(native, n, shared):
    from heavyrt_gb300 import SceneRT
    from oracle import oracle as orc

    v, idx = _mesh(n, shared)
    o = orc.OracleBVH(v, idx)
    assert (np.diff(np.append(o.run_starts(), n)) <= 127).all()
    want = _expected(o)
    for stride in (12, 16, 28):
        raw = np.zeros((len(v), stride // 4), np.float32)
        raw[:, :3] = v[:, :3]
        s = SceneRT()
        gid = s.AddGeom_Triangles3f(raw, len(v), idx, idx.size, vByteStride=stride)
        got = _stages(s, gid)
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{n} triangles, stride {stride}: {k}")
        s.close()


@pytest.mark.parametrize("n,verts", [(5, 12288), (5, 12289), (4096, 12289), (300, 40000)])
def test_vertices_that_no_triangle_uses(native, n, verts):
    from heavyrt_gb300 import SceneRT
    from oracle import oracle as orc

    rng = np.random.default_rng(verts)
    v = np.ones((verts, 4), np.float32)
    v[:, :3] = rng.uniform(-1, 1, (verts, 3))
    idx = rng.integers(0, verts, 3 * n).astype(np.uint32)
    want = _expected(orc.OracleBVH(v, idx))
    s = SceneRT()
    got = _stages(s, s.AddGeom_Triangles3f(v, verts, idx, idx.size, vByteStride=16))
    for k in want:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
    s.close()


def test_bad_indices_and_crowded_codes_are_refused(native):
    from heavyrt_gb300 import HrtError, SceneRT
    from heavyrt_gb300 import workload as wl

    s = SceneRT()
    v, idx = wl.soup(5, 100, off=0.03)
    bad = idx.copy()
    bad[250] = len(v)
    with pytest.raises(HrtError):
        s.AddGeom_Triangles3f(v, len(v), bad, bad.size, vByteStride=16)
    with pytest.raises(HrtError):  # 200 triangles at one place
        s.AddGeom_Triangles3f(v, len(v), np.tile(idx[:3], 200), 600, vByteStride=16)
    s.close()


@pytest.mark.parametrize("count", [2, 40, 600])
@pytest.mark.parametrize("empty", [False, True])
def test_instance_trees(native, count, empty):
    """An instance tree gives what testing every instance gives, with an
    instance of a geometry without triangles among them or not."""
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    v, idx = wl.soup(9, 60, off=0.2)
    rays = torch.from_numpy(wl.sphere_rays(10, 4000)).cuda()
    got = []
    for tlas in (True, False):
        s = SceneRT()
        s.set_tlas(tlas)
        g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
        none = s.AddGeom_Triangles3f(v, len(v), idx[:0], 0, vByteStride=16)
        r = np.random.default_rng(count)
        for k in range(count):
            m = np.eye(4, dtype=np.float32)
            m[:3, 3] = r.uniform(-1, 1, 3)
            m[:3, :3] *= 0.3
            s.AddInstance(none if empty and k == count // 2 else g, m)
        s.CommitScene()
        hits = torch.zeros((4000, 8), device="cuda")
        s.query_device(0, rays.data_ptr(), 4000, hits.data_ptr())
        torch.cuda.synchronize()
        got.append(hits.cpu().numpy().view(np.uint32))
        s.close()
    np.testing.assert_array_equal(got[0], got[1])
    assert (got[0][:, 2] != 0xFFFFFFFF).any()
