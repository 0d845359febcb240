"""The build's kernels at their edges: slices of 512 leaves and chunks of 512
triangles (runs that cross them, runs of a hundred triangles), scan tiles past
one look-back window, the walks that leave a slice, the largest-first roles
above and below one block's frontier, and geometries of a batch that share a
slice; every stage against the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stages(s, gid):
    from heavyrt_gb300 import engine as E

    return {"box": s.export(gid, E.EXPORT_SCENE_BOX).view(np.uint32), "unsorted": s.export(gid, E.EXPORT_MORTON_UNSORTED),
            "sorted": s.export(gid, E.EXPORT_MORTON_SORTED), "codes": s.export(gid, E.EXPORT_COMPRESSED),
            "runs": s.export(gid, E.EXPORT_RUN_STARTS), "lr": s.export(gid, E.EXPORT_LR_NODES).view(np.uint32),
            "counts": s.export(gid, E.EXPORT_LR_COUNTS), "order": s.export(gid, E.EXPORT_PRIM_INDICES),
            "idx": s.export(gid, E.EXPORT_SORTED_INDICES)}


def _expected(o):
    return {"box": o.scene_box().view(np.uint32), "unsorted": o.morton_unsorted(), "sorted": o.morton_sorted(),
            "codes": o.compressed(), "runs": o.run_starts(), "lr": np.asarray(o.lr_nodes()).view(np.uint32),
            "counts": o.lr_counts(), "order": o.prim_indices(), "idx": o.sorted_indices()}


def _check(got, want, what):
    for k in want:
        np.testing.assert_array_equal(np.asarray(got[k]).reshape(-1), np.asarray(want[k]).reshape(-1), err_msg=f"{what}: {k}")


def _clustered(seed, n, per_cell):
    """n small triangles, about per_cell of them in each of the cells they fall in."""
    rng = np.random.default_rng(seed)
    cells = max(1, n // per_cell)
    at = rng.uniform(-1, 1, (cells, 3))[rng.integers(0, cells, n)]
    v = at[:, None, :] + rng.uniform(-2e-4, 2e-4, (n, 3, 3))
    verts = np.ones((3 * n, 4), np.float32)
    verts[:, :3] = v.reshape(-1, 3)
    verts[:2, :3] = [[-1, -1, -1], [1, 1, 1]]  # the box of every size
    return verts, np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("n,per_cell", [(511, 0), (512, 0), (513, 0), (1024, 0), (1025, 0), (3000, 60), (20000, 3),
                                        (70000, 40), (135000, 0), (300001, 0)])
def test_stages_at_the_edges(native, n, per_cell):
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    v, idx = _clustered(n, n, per_cell) if per_cell else wl.soup(n, n, off=0.01)
    o = orc.OracleBVH(v, idx)
    if (np.diff(np.append(o.run_starts(), n)) > 127).any():
        pytest.skip("more than 127 triangles in a cell")
    want = _expected(o)
    for stride in (16, 12, 28):
        raw = np.zeros((len(v), stride // 4), np.float32)
        raw[:, :3] = v[:, :3]
        s = SceneRT()
        gid = s.AddGeom_Triangles3f(raw, len(v), idx, idx.size, vByteStride=stride)
        _check(_stages(s, gid), want, f"{n} triangles, stride {stride}")
        s.close()


@pytest.mark.parametrize("merge", [0, 1, 4])
@pytest.mark.parametrize("n,per_cell", [(600, 0), (2100, 0), (20000, 3), (30000, 0)])
def test_largest_first_nodes_past_the_frontier(native, n, per_cell, merge):
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import engine as E
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    v, idx = _clustered(n, n, per_cell) if per_cell else wl.soup(n, n, off=0.01)
    o = orc.OracleBVH(v, idx)
    s = SceneRT(layout="bvh4")
    s.set_bvh4_merge(merge)
    s.set_bvh4_collapse(E.BVH4_COLLAPSE_LARGEST_FIRST)
    gid = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    want = orc.collapse4(o.lr_nodes(), o.lr_counts(), o.run_starts(), o.n_tris, merge, 1)
    np.testing.assert_array_equal(s.export(gid, E.EXPORT_NODES4).view(np.uint32).reshape(-1, 32), want)
    s.close()


@pytest.mark.parametrize("layout", [0, 2])
def test_batches_across_slices(native, layout):
    """Geometries of uneven sizes, many to a slice and many slices to one."""
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import engine as E
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    sizes = [1, 2, 3, 500, 12, 1, 6000, 511, 513, 40, 1500, 1, 9000]
    meshes = [wl.soup(40 + k, n, off=0.02) if k % 4 else _clustered(k, n, 9) for k, n in enumerate(sizes)]
    s = SceneRT(layout=layout)
    s.set_bvh4_collapse(E.BVH4_COLLAPSE_LARGEST_FIRST)
    ids = s.add_geoms_batched([m[0] for m in meshes], [m[1] for m in meshes])
    for gid, (v, idx) in zip(ids, meshes):
        o = orc.OracleBVH(v, idx)
        _check(_stages(s, gid), _expected(o), f"geometry {gid}")
        if layout == 2:
            want = orc.collapse4(o.lr_nodes(), o.lr_counts(), o.run_starts(), o.n_tris, 0, 1)
            got = s.export(gid, E.EXPORT_NODES4).view(np.uint32).reshape(-1, 16)
            np.testing.assert_array_equal(got[:, 12:16], want[:, 24:28])
    s.close()


def _off(a, words):
    """A copy of `a` that starts `words` 4-byte words past a 16-byte boundary."""
    buf = np.zeros(a.size + 8, a.dtype)
    at = (-buf.ctypes.data // 4) % 4 + words
    out = buf[at:at + a.size].reshape(a.shape)
    out[...] = a
    return out


@pytest.mark.parametrize("words", [0, 1, 3])
@pytest.mark.parametrize("columns", [3, 4, 6])
def test_inputs_in_place(native, columns, words):
    """Host arrays of any alignment and stride, device arrays, and a batch's
    arrays apart and joined give the arrays of a plain load."""
    import ctypes as C

    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import engine as E
    from heavyrt_gb300 import workload as wl

    meshes = [wl.soup(60 + k, n, off=0.02) for k, n in enumerate((1, 5, 700, 3001))]
    s = SceneRT()
    plain = [s.AddGeom_Triangles3f(v, len(v), i, i.size, vByteStride=16) for v, i in meshes]
    want = [_stages(s, g) for g in plain]
    raw = []
    for v, i in meshes:
        r = np.full((len(v), columns), 7.0, np.float32)
        r[:, :3] = v[:, :3]
        raw.append((_off(r, words), _off(i, words)))
    for k, (r, i) in enumerate(raw):  # host, then device (the C entry takes addresses)
        g = s.AddGeom_Triangles3f(r, len(r), i, i.size, vByteStride=4 * columns)
        _check(_stages(s, g), want[k], f"mesh {k}")
        dr, di = torch.zeros(r.size + 4, device="cuda"), torch.zeros(i.size + 4, dtype=torch.int32, device="cuda")
        dr[words:words + r.size] = torch.from_numpy(r.copy()).reshape(-1).cuda()
        di[words:words + i.size] = torch.from_numpy(i.view(np.int32).copy()).cuda()
        torch.cuda.synchronize()
        gid = C.c_uint32()
        s.ctx.check(E.lib().hrt_add_geom_triangles3f(s._h, C.c_void_p(dr.data_ptr() + 4 * words), len(r),
                                                     C.c_void_p(di.data_ptr() + 4 * words), i.size, 2, 4 * columns,
                                                     C.byref(gid)), "device arrays")
        _check(_stages(s, gid.value), want[k], f"mesh {k} on the device")
    for k, g in enumerate(s.add_geoms_batched([r for r, _ in raw], [i for _, i in raw])):
        _check(_stages(s, g), want[k], f"batch {k}")
    # an array of another width among them: all are widened
    mixed = [raw[0][0][:, :3].copy()] + [r for r, _ in raw[1:]]
    for k, g in enumerate(s.add_geoms_batched(mixed, [i for _, i in raw])):
        _check(_stages(s, g), want[k], f"mixed batch {k}")
    v = _off(np.concatenate([r for r, _ in raw]), words)
    i = _off(np.concatenate([i for _, i in raw]), words)
    voff = np.cumsum([0] + [len(r) for r, _ in raw]).astype(np.uint64)
    ioff = np.cumsum([0] + [x.size for _, x in raw]).astype(np.uint64)
    first = C.c_uint32()
    s.ctx.check(E.lib().hrt_add_geoms_triangles3f_batched(s._h, len(raw), E._ptr(v), E._ptr(voff), E._ptr(i), E._ptr(ioff),
                                                          2, 4 * columns, C.byref(first)), "joined")
    for k in range(len(raw)):
        _check(_stages(s, first.value + k), want[k], f"joined batch {k}")
    with pytest.raises(ValueError):
        s.AddGeom_Triangles3f(raw[0][0], len(raw[0][0]), raw[0][1], raw[0][1].size + 3, vByteStride=4 * columns)
    s.close()
