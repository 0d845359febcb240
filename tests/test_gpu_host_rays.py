"""Rays in host memory: batches around the lines at which a host query is cut
into chunks give the results of device memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("n", [1, (2 << 17) - 1, 2 << 17, (2 << 17) + 1, (8 << 17) + 3])
def test_chunks_of_a_host_query(native, n, aligned):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    v, idx = wl.soup(51, 2000, off=0.03)
    s = SceneRT(layout=2)
    g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    s.AddInstance(g)
    s.CommitScene()
    block = np.empty(8 * n + 8, np.float32)
    at = (-block.ctypes.data // 4) % 4 + (0 if aligned else 1)  # 16-byte aligned, or four bytes past it
    rays = block[at:at + 8 * n].reshape(n, 8)
    rays[:] = wl.sphere_rays(52, n)
    dev = torch.from_numpy(rays.copy()).cuda()
    hits = torch.zeros((n, 8), device="cuda")
    flags = torch.zeros(n, dtype=torch.uint8, device="cuda")
    s.query_device(0, dev.data_ptr(), n, hits.data_ptr())
    s.query_device(1, dev.data_ptr(), n, flags.data_ptr())
    torch.cuda.synchronize()
    got = s.RayQuery_NearestHit(rays)
    np.testing.assert_array_equal(got.view(np.uint32).reshape(n, 8), hits.cpu().numpy().view(np.uint32))
    np.testing.assert_array_equal(s.RayQuery_AnyHit(rays), flags.cpu().numpy().astype(bool))
