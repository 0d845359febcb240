"""Batches around the lines of the launch rule (few rays a warp, one thread per
ray, the persistent pool): the first n rays of a batch give the same results
whatever n, on one geometry, on its segments and on an instance tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MISS = 0xFFFFFFFF


def _lines(sms):
    spread, resident = 13 * sms, 36 * 32 * sms
    return sorted({1, 2, 31, 32, 33, spread, spread + 1, 2 * spread, 2 * spread + 1, 16 * spread, 16 * spread + 1,
                   resident - 1, resident, resident + 1, resident + 1000})


def _query(scene, kind, rays, n, out, seg=None):
    import torch

    from heavyrt_gb300 import engine

    out.zero_()
    if seg is None:
        scene.query_device(kind, rays.data_ptr(), n, out.data_ptr())
    else:
        off = torch.tensor([0, min(n, 7), n], dtype=torch.int32, device="cuda")
        scene.query_multi(engine.query_desc(kind, rays.data_ptr(), n, out.data_ptr(), off.data_ptr(), seg.data_ptr(), 2))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert not got[n:].any()  # nothing past the batch
    return got[:n].view(np.uint32) if kind == 0 else got[:n]


@pytest.mark.parametrize("given", [False, True])
@pytest.mark.parametrize("layout", [0, 2, 3])
def test_results_do_not_depend_on_the_batch_size(native, layout, given):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl
    from oracle import oracle as orc

    lines = _lines(torch.cuda.get_device_properties(0).multi_processor_count)
    top = lines[-1]
    v, idx = wl.soup(91, 3000, off=0.03)
    host = np.concatenate([wl.rays_at_triangles(9, v, idx, top // 2, jitter=0.02), wl.sphere_rays(10, top - top // 2)])
    host = host[np.random.default_rng(3).permutation(top)]
    o = orc.OracleBVH(v, idx)
    want, want_any = o.trace(host), o.trace(host, any_hit=True)
    rays = torch.from_numpy(host).cuda()
    hits = torch.zeros((top, 8), device="cuda")
    flags = torch.zeros(top, dtype=torch.uint8, device="cuda")

    one = SceneRT(layout=layout)
    g = one.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    one.AddInstance(g)
    one.CommitScene()
    many = SceneRT(layout=layout)  # an instance tree; instance 2 is the geometry as it is
    g = many.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    for k in range(5):
        m = np.eye(4, dtype=np.float32)
        m[:3, 3] = 0.0 if k == 2 else (3.0 * (k - 2), 0.3 * k, 0.0)
        many.AddInstance(g, m)
    many.CommitScene()
    seg = torch.tensor([2, 2], dtype=torch.int32, device="cuda")
    if given:
        for s in (one, many):
            s.set_trace_config(0, 256, 1, 5, 3)
            s.set_trace_config(1, 64, 0)
    tree = _query(many, 0, rays, top, hits), _query(many, 1, rays, top, flags)
    for n in lines:
        got = _query(one, 0, rays, n, hits)
        np.testing.assert_array_equal(got[:, 0], want["t"][:n].view(np.uint32))
        np.testing.assert_array_equal(got[:, 3] == MISS, want["geomId"][:n] == MISS)
        np.testing.assert_array_equal(_query(one, 1, rays, n, flags) != 0, want_any[:n])
        part = _query(many, 0, rays, n, hits, seg)
        np.testing.assert_array_equal(part[:, 0], got[:, 0])
        np.testing.assert_array_equal(part[:, 1], got[:, 1])
        np.testing.assert_array_equal(_query(many, 1, rays, n, flags, seg) != 0, want_any[:n])
        np.testing.assert_array_equal(_query(many, 0, rays, n, hits), tree[0][:n])
        np.testing.assert_array_equal(_query(many, 1, rays, n, flags), tree[1][:n])
    one.close()
    many.close()
