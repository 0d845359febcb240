"""The launch shape that a caller sets is the one that is launched: threads a
block, pool or one thread per ray, and the part of the stack in shared memory, on
one geometry, on segments and on an instance tree, read from the nodes of a
captured graph.  The only exception is a pool in a batch so small that it would
refill nothing (13 x 16 rays an SM), which goes one thread per ray.  Shapes that
the autotuner compares are therefore launched too, and the one that it leaves is
one of those it timed."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNEL, MEMSET = 0, 2


class _KernelParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS (version 2)
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _launched(query):
    """(blocks, threads, shared bytes, cleared a counter) of the one kernel that query(stream) launches."""
    import torch

    cu = C.CDLL("libcuda.so.1")
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g, capture_error_mode="relaxed"):
        query(torch.cuda.current_stream().cuda_stream)
    graph, n = C.c_void_p(g.raw_cuda_graph()), C.c_size_t()
    assert cu.cuGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0
    kinds, found = [], []
    for node in nodes:
        t = C.c_int()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(t)) == 0
        kinds.append(t.value)
        if t.value == KERNEL:
            p = _KernelParams()
            assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
            found.append((p.grid[0], p.block[0], p.shared))
    assert len(found) == 1
    return (*found[0], MEMSET in kinds)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("place", ["one", "segments", "turns", "tree"])
@pytest.mark.parametrize("small", [True, False])
def test_a_given_shape_is_launched(native, small, place, layout, kind):
    import torch

    from heavyrt_gb300 import SceneRT, engine
    from heavyrt_gb300 import workload as wl

    n = 13 * 16 * torch.cuda.get_device_properties(0).multi_processor_count + (not small)  # all resident at once
    v, idx = wl.soup(31, 2000, off=0.02)
    rays = torch.from_numpy(wl.sphere_rays(3, n)).cuda()
    out = torch.zeros((n, 8), device="cuda")
    off = torch.tensor([0, 7, n], dtype=torch.int32, device="cuda")
    seg = torch.tensor([1, 0], dtype=torch.int32, device="cuda")
    s = SceneRT(layout=layout)
    s.set_tlas(place == "tree")
    g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    s.AddInstance(g)
    if place != "one":
        s.AddInstance(g, np.diag([2, 1, 1, 1]).astype(np.float32))
    s.CommitScene()
    if place == "segments":
        desc = engine.query_desc(kind, rays.data_ptr(), n, out.data_ptr(), off.data_ptr(), seg.data_ptr(), 2)
        query = lambda stream: s.query_multi(desc, stream)
    else:
        query = lambda stream: s.query_device(kind, rays.data_ptr(), n, out.data_ptr(), stream)
    depth = (32 if layout == 0 else 48) + (32 if place == "tree" else 0)
    for threads, persistent, stack in ((64, 1, 0), (128, 1, 0), (256, 1, 16), (128, 0, 0), (256, 0, depth), (64, 0, 20)):
        s.set_trace_config(kind, threads, persistent, 5, 3, stack)
        blocks, block, shared, cleared = _launched(query)
        assert (block, cleared) == (threads, bool(persistent) and not small), (threads, persistent, stack)
        entries = stack if 0 < stack < depth else depth
        assert shared == 4 * threads * entries, (threads, persistent, stack)
        if cleared:
            assert blocks <= -(-n // threads)
    s.close()


@pytest.mark.parametrize("n", [5000, 60000])
def test_autotune_leaves_a_shape_that_it_launched(native, n):
    import torch

    from heavyrt_gb300 import SceneRT, engine
    from heavyrt_gb300 import workload as wl

    v, idx = wl.soup(31, 2000, off=0.02)
    rays = torch.from_numpy(wl.sphere_rays(3, n)).cuda()
    out = torch.zeros((n, 8), device="cuda")
    s = SceneRT(layout=2)
    s.AddInstance(s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16))
    s.CommitScene()
    cfg, _ = s.autotune(engine.query_desc(0, rays.data_ptr(), n, out.data_ptr()), repeats=2)
    _, block, shared, cleared = _launched(lambda stream: s.query_device(0, rays.data_ptr(), n, out.data_ptr(), stream))
    assert (block, cleared) == (cfg["threadsPerBlock"], bool(cfg["persistent"]))
    assert shared == 4 * block * min(cfg["stackEntries"] or 48, 48)
    s.close()
