"""Rays in host memory: batches around the lines at which a host query is cut
into chunks, and server batches whose requests' rays lie in page-locked,
pageable and differently aligned memory; every result equals the one from
device memory, or from the request alone."""
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


@pytest.mark.parametrize("layout", [0, 2, 3])
@pytest.mark.parametrize("count", [2, 9])
def test_one_batch_of_rays_from_everywhere(native, layout, count):
    from heavyrt_gb300 import PinnedBuffer
    from heavyrt_gb300 import engine as E
    from heavyrt_gb300 import workload as wl

    sizes = [1, 31, 32, 33, 1000, 5, 20000, 64, 7][:count]
    v, idx = wl.soup(61, 4000, off=0.03)
    srv = E.Server(slot_rays=1 << 18, slots=1, max_batch_requests=count, layout=layout)
    sid = srv.add_scene(v, idx, evictable=False)
    assert srv.scene_state(sid, timeout=120) == E.SCENE_READY
    rays = [wl.rays_at_triangles(70 + j, v, idx, n, jitter=0.05) for j, n in enumerate(sizes)]
    want = []
    for j, r in enumerate(rays):
        out = np.empty((len(r), 8), np.uint32) if j % 2 == 0 else np.empty(len(r), np.uint8)
        assert srv.wait(srv.submit_array(sid, j % 2, np.ascontiguousarray(r), out))[0] == 0
        want.append(out)
    most = 1
    for attempt in range(8):
        buffers, outs, tickets = [], [], []
        for j, r in enumerate(rays):
            # page-locked on 32 and on 16 bytes, page-locked on 4, pageable
            shift = (0, 4, 1)[j % 4] if j % 4 < 3 else None
            if shift is None:
                buffers.append(np.ascontiguousarray(r))
                at = buffers[-1].ctypes.data
            else:
                buffers.append(PinnedBuffer(r.nbytes + 64))
                buffers[-1].array(np.float32)[shift:shift + r.size] = r.reshape(-1)
                at = buffers[-1].ptr + 4 * shift
            outs.append((at, np.full_like(want[j], 0xAB)))
        # a request in flight keeps the one slot busy, so the others are batched
        big = wl.sphere_rays(80 + attempt, 200000)
        flags = np.empty(len(big), np.uint8)
        first = srv.submit_array(sid, 1, big, flags)
        for j, (at, out) in enumerate(outs):
            tickets.append(srv.submit(sid, j % 2, at, len(rays[j]), out.ctypes.data))
        assert srv.wait(first)[0] == 0
        for t in tickets:
            st, info = srv.wait(t)
            assert st == 0
            most = max(most, info["batchRequests"])
        for j, (at, out) in enumerate(outs):
            np.testing.assert_array_equal(out, want[j], err_msg=f"request {j}")
        for b in buffers:
            if isinstance(b, PinnedBuffer):
                b.free()
        if most == count:
            break
    assert most > 1
    srv.close()
