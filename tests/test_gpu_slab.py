"""The traversal kernels' packed slab test at its edges: every sign pattern of
the direction (zeros of both signs among them), origins on the planes of the
boxes, empty and unbounded intervals, lone leaves and nodes with unused slots,
rays through the point that an unused slot's box is, and rays that are not
numbers; single-instance and segmented launches, both triangle tests, against
the oracle."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MISS = 0xFFFFFFFF


def _rays(rng, v, n_each):
    """n_each rays of each of the 26 sign patterns, aimed past and through the mesh's vertices."""
    p = v[:, :3]
    out = []
    for signs in itertools.product((-1, 0, 1), repeat=3):
        if signs == (0, 0, 0):
            continue
        d = rng.uniform(0.2, 1.0, (n_each, 3)) * np.asarray(signs, float)
        d[::2][:, [s == 0 for s in signs]] = -0.0
        at = p[rng.integers(0, len(p), n_each)].astype(np.float64) + rng.uniform(-0.03, 0.03, (n_each, 3))
        o = at - d * rng.uniform(0.0, 3.0, (n_each, 1))
        plane = rng.integers(0, 3, n_each)  # every fourth origin lies on a plane of some box
        rows = np.arange(0, n_each, 4)
        o[rows, plane[rows]] = p[rng.integers(0, len(p), len(rows)), plane[rows]]
        r = np.zeros((n_each, 8), np.float32)
        r[:, 0:3], r[:, 4:7], r[:, 7] = o, d, 1e9
        out.append(r)
    r = np.concatenate(out)
    r[1::7, 3] = 0.5
    r[2::11, 7] = np.inf
    r[3::13, 7] = 0.1  # short, and behind tNear for some
    through = rng.uniform(-1, 1, (64, 3))  # through the origin, the box of an unused slot
    z = np.zeros((64, 8), np.float32)
    z[:, 0:3], z[:, 4:7], z[:, 7] = through, -through, 1e9
    return np.concatenate([r, z])


@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_every_direction_sign(native, layout, test):
    import torch

    from heavyrt_gb300 import SceneRT, engine
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    rng = np.random.default_rng(11)
    meshes = [wl.soup(700 + n, n, off=0.05) for n in (1, 2, 3, 4, 5, 33, 4000)]
    scene = SceneRT(layout=layout, triangle_test=test)
    want_all, rays_all, counts = [], [], []
    for v, idx in meshes:
        rays = _rays(rng, v, 40)
        o = orc.OracleBVH(v, idx)
        want, any_want = o.trace(rays, watertight=test == "watertight"), o.trace(rays, any_hit=True,
                                                                                watertight=test == "watertight")
        one = SceneRT(layout=layout, triangle_test=test)
        one.AddInstance(one.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16))
        one.CommitScene()
        for persistent in (0, 1):
            one.set_trace_config(0, persistent=persistent)
            one.set_trace_config(1, persistent=persistent)
            got = one.RayQuery_NearestHit(rays)
            np.testing.assert_array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
            np.testing.assert_array_equal(got["geomId"] == MISS, want["geomId"] == MISS)
            if layout == 0:
                np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
            np.testing.assert_array_equal(one.RayQuery_AnyHit(rays), any_want)
        one.close()
        scene.AddInstance(scene.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16))
        want_all.append(want), rays_all.append(rays), counts.append(len(rays))
    # the same rays as one segmented launch; the last segment names no instance
    extra = rays_all[-1][:40]
    scene.CommitScene()
    rays = torch.from_numpy(np.concatenate(rays_all + [extra])).cuda()
    off = torch.from_numpy(np.cumsum([0] + counts + [len(extra)]).astype(np.int32)).cuda()
    seg = torch.tensor(list(range(len(meshes))) + [99], dtype=torch.int32, device="cuda")
    hits = torch.zeros((len(rays), 8), device="cuda")
    for persistent in (0, 1):
        scene.set_trace_config(0, persistent=persistent)
        scene.query_multi(engine.query_desc(0, rays.data_ptr(), len(rays), hits.data_ptr(), off.data_ptr(),
                                            seg.data_ptr(), len(seg)))
        torch.cuda.synchronize()
        got = hits.cpu().numpy().view(np.uint32)
        at = 0
        for k, want in enumerate(want_all):
            g = got[at:at + counts[k]]
            found = want["geomId"] != MISS
            np.testing.assert_array_equal(g[:, 0], want["t"].view(np.uint32))
            np.testing.assert_array_equal(g[:, 2], np.where(found, k, MISS))
            np.testing.assert_array_equal(g[:, 3], np.where(found, k, MISS))
            at += counts[k]
        assert (got[at:, 1:4] == MISS).all()
        np.testing.assert_array_equal(got[at:, 0], extra[:, 7].view(np.uint32))
    scene.close()


@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_rays_that_are_not_numbers_miss(native, layout):
    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    v, idx = wl.soup(3, 500, off=0.1)
    s = SceneRT(layout=layout)
    s.AddInstance(s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16))
    s.CommitScene()
    base = wl.rays_at_triangles(5, v, idx, 64)
    for column in (0, 1, 2, 3, 4, 5, 6, 7):
        for value in (np.nan, np.inf, -np.inf):
            if column == 3 and value == -np.inf or column == 7 and value == np.inf:
                continue  # an unbounded interval
            rays = base.copy()
            rays[:, column] = value
            assert (s.RayQuery_NearestHit(rays)["primId"] == MISS).all(), (column, value)
            assert not s.RayQuery_AnyHit(rays).any(), (column, value)
    s.close()
