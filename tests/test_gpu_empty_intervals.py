"""The counters are those of the reference's comparisons also for rays whose tFar
lies before their tNear: such a ray misses, and visits the boxes that the
reference's walk visits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MISS = 0xFFFFFFFF


@pytest.mark.parametrize("near,far", [(0.7, 0.5), (0.0, -1.0), (1e10, 1e9), (2.5, 2.0)])
def test_counters_of_empty_intervals(native, near, far):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    v, idx = wl.soup(77, 3000, off=0.08)
    rays = np.concatenate([wl.rays_at_triangles(3, v, idx, 1000), wl.sphere_rays(4, 1000, radius=0.5)])
    rays[::3, 3], rays[::3, 7] = near, far
    o = orc.OracleBVH(v, idx)
    want, counts, _ = o.trace(rays, counters=True)
    d = torch.from_numpy(rays).cuda()
    for layout in (0, 1, 2, 3):
        s = SceneRT(layout=layout)
        s.AddInstance(s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16))
        s.CommitScene()
        got = s.RayQuery_NearestHit(rays)
        np.testing.assert_array_equal(got["t"].view(np.uint32), want["t"].view(np.uint32))
        assert (got["primId"][::3] == MISS).all() and not s.RayQuery_AnyHit(rays)[::3].any()
        if layout == 0:
            assert s.query_counters(0, d.data_ptr(), len(rays)) == counts
        s.close()
