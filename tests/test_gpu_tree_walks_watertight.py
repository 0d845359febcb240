"""An instance tree's walks under the watertight test: batches on both sides of
the lines between one thread per ray, the pool without a vote and the pool by
vote give each ray the result that testing every instance in turn gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_results_do_not_depend_on_the_walk(native, layout):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    spread, resident, vote = 13 * 16 * sms, 24 * 32 * sms, 128 * 32 * sms
    top = vote + 33
    v, idx = wl.soup(23, 500, off=0.05)
    rays = torch.from_numpy(wl.sphere_rays(24, top)).cuda()
    want = None
    for tree in (False, True):
        s = SceneRT(layout=layout, triangle_test="watertight")
        s.set_tlas(tree)
        g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
        rng = np.random.default_rng(6)
        for _ in range(9):
            m = np.eye(4, dtype=np.float32)
            m[:3, :3] *= 0.4
            m[:3, 3] = rng.uniform(-1, 1, 3)
            s.AddInstance(g, m)
        s.CommitScene()
        for n in [top] if not tree else [spread, spread + 1, resident, resident + 1, vote, vote + 1, top]:
            hits = torch.zeros((n, 8), device="cuda")
            flags = torch.zeros(n, dtype=torch.uint8, device="cuda")
            s.query_device(0, rays.data_ptr(), n, hits.data_ptr())
            s.query_device(1, rays.data_ptr(), n, flags.data_ptr())
            torch.cuda.synchronize()
            got = hits.view(torch.int32), flags
            if want is None:
                want = got
                assert 0 < int(flags.sum()) < n
            else:
                assert torch.equal(got[0], want[0][:n]) and torch.equal(got[1], want[1][:n]), n
        s.close()
