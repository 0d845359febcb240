"""On an instance tree the shape that a caller sets decides where the traversal
stack lies, as on a single geometry: 0, or a value at or above the depth bound,
keeps the whole of it in shared memory, a smaller one that many entries of it
(read from the node of a captured graph)."""
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
@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_a_given_stack_is_in_shared_memory(native, layout, kind):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    n = 150000  # more than the GPU holds at once
    v, idx = wl.soup(31, 2000, off=0.02)
    rays = torch.from_numpy(wl.sphere_rays(3, n)).cuda()
    out = torch.zeros((n, 8), device="cuda")
    s = SceneRT(layout=layout)
    g = s.AddGeom_Triangles3f(v, len(v), idx, idx.size, vByteStride=16)
    s.AddInstance(g)
    s.AddInstance(g, np.diag([2, 1, 1, 1]).astype(np.float32))
    s.CommitScene()
    results = []
    depth = (32 if layout == 0 else 48) + 32
    for threads, stack in ((64, 0), (128, 0), (256, 0), (128, depth), (128, depth + 1), (128, depth - 1), (64, 1)):
        s.set_trace_config(kind, threads, 1, 5, 3, stack)
        query = lambda stream: s.query_device(kind, rays.data_ptr(), n, out.data_ptr(), stream)
        _, block, shared, _ = _launched(query)
        assert (block, shared) == (threads, 4 * threads * (stack if 0 < stack < depth else depth)), (threads, stack)
        query(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        results.append(out.clone())
        assert torch.equal(results[0].view(torch.int32), out.view(torch.int32))
    s.close()
