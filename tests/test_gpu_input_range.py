"""Arrays that are page-locked in their first part only give the results that
pageable arrays give where kernels read them in place: builds, host queries and a
server's rays."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 65536


def _partly_locked(a):
    """A copy of a at a page boundary whose first half (in whole pages) is page-locked; release() ends that."""
    import torch

    room = mmap.mmap(-1, (a.nbytes + 2 * PAGE) // PAGE * PAGE + PAGE)
    raw = np.frombuffer(room, np.uint8)
    at = -raw.ctypes.data % PAGE
    b = raw[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
    b[...] = a
    locked = a.nbytes // 2 // PAGE * PAGE
    assert locked and int(torch.cuda.cudart().cudaHostRegister(b.ctypes.data, locked, 0)) == 0
    return b, lambda: torch.cuda.cudart().cudaHostUnregister(b.ctypes.data)


@pytest.mark.parametrize("layout", [0, 2])
def test_partly_page_locked_arrays(native, layout):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300.engine import SCENE_READY, Server
    from heavyrt_gb300 import workload as wl

    torch.cuda.init()
    v, idx = wl.soup(31, 20000, off=0.02)
    rays = wl.rays_at_triangles(7, v, idx, 30000, jitter=0.02)
    whole = v, idx  # a server copies a scene's arrays, which refuses one that is locked in part
    want = None
    for part in (False, True):
        done = []
        if part:
            (v, d0), (idx, d1), (rays, d2) = _partly_locked(v), _partly_locked(idx), _partly_locked(rays)
            done = [d0, d1, d2]
        s = SceneRT(layout=layout)
        g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
        s.AddInstance(g)
        s.AddInstance(s.add_geoms_batched([v, v], [idx, idx])[1])
        s.CommitScene()
        got = [s.RayQuery_NearestHit(rays).view(np.uint32).reshape(-1, 8), s.RayQuery_AnyHit(rays)]
        srv = Server(layout=layout)
        sid = srv.add_scene(*whole)
        assert srv.scene_state(sid, 30.0) == SCENE_READY
        hits, flags = np.zeros((len(rays), 8), np.uint32), np.zeros(len(rays), np.uint8)
        tickets = [srv.submit_array(sid, 0, rays, hits), srv.submit_array(sid, 1, rays, flags)]
        assert all(srv.wait(t, 30.0)[0] == 0 for t in tickets)
        got += [hits, flags]
        if want is None:
            want = got
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
        srv.close()
        s.close()
        for d in done:
            assert int(d()) == 0
