"""Rays that are not numbers end at the root: whatever the layout, the kind of
query and the instance's transform (which spreads one bad component over all
three axes), such a ray visits one node and misses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MISS = 0xFFFFFFFF
NAN, INF = np.nan, np.inf


@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("layout", [0, 1, 2, 3])
@pytest.mark.parametrize("place", ["as_is", "moved", "tree"])
def test_one_visit_a_ray(native, layout, test, place):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    v, idx = wl.soup(3, 2000, off=0.05)
    s = SceneRT(layout=layout, triangle_test=test)
    g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    turned = np.eye(4, dtype=np.float32)
    turned[:3, :3] = [[0.48, -0.6, 0.64], [0.8, 0.6, 0.0], [-0.36, 0.52, 0.77]]
    s.AddInstance(g, None if place == "as_is" else turned)
    if place == "tree":
        s.AddInstance(g, np.diag([1, 2, 1, 1]).astype(np.float32))
    s.CommitScene()
    base = wl.rays_at_triangles(5, v, idx, 64)
    bad = [((0, 1, 2), NAN), ((3,), NAN), ((7,), NAN), ((0, 1, 2, 4, 5, 6), NAN), ((0, 1, 2, 7), NAN)]
    if place == "moved":  # one component is enough
        bad += [((0,), NAN), ((1,), NAN), ((2,), NAN), ((0, 1, 2), INF)]
    for columns, value in bad:
        rays = base.copy()
        rays[:, columns] = value
        d = torch.from_numpy(rays).cuda()
        for kind in (0, 1):
            assert s.query_counters(kind, d.data_ptr(), len(rays)) == (len(rays), 0), (columns, value, kind)
        assert (s.RayQuery_NearestHit(rays)["primId"] == MISS).all(), (columns, value)
        assert not s.RayQuery_AnyHit(rays).any(), (columns, value)
    s.close()
