"""The blob of a batch-built geometry is that of the same geometry built alone,
byte for byte: nothing in it is what the memory held before.  (A geometry without
triangles differs in its header's frame; its unused words are zero too.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("test", ["mt", "watertight"])
@pytest.mark.parametrize("layout", [0, 1, 2, 3])
def test_blob_of_a_batch_geometry(native, tmp_path, layout, test):
    import torch

    from heavyrt_gb300 import SceneRT
    from heavyrt_gb300 import workload as wl

    sizes = (1, 2, 40, 513, 5000, 0)
    meshes = [wl.soup(60 + n, n, off=0.05) if n else (np.ones((4, 4), np.float32), np.zeros(0, np.uint32)) for n in sizes]
    for k, n in enumerate((3, 300, 2000, 20000, 70000)):
        v, i = wl.soup(90 + k, n, off=0.02)
        s = SceneRT(layout=layout, triangle_test=test)
        s.AddGeom_Triangles3f(v, len(v), i, i.size, vByteStride=16)
        s.ClearGeom()  # the pool's memory has held indices, codes and nodes
        ids = s.add_geoms_batched([v for v, _ in meshes], [i for _, i in meshes])
        one = SceneRT(layout=layout, triangle_test=test)
        for g, (v, i) in zip(ids, meshes):
            a = one.AddGeom_Triangles3f(v, len(v), i, i.size, vByteStride=16)
            s.save_geom(g, tmp_path / "batch")
            one.save_geom(a, tmp_path / "alone")
            got = (tmp_path / "batch").read_bytes()
            assert got[88:96] == bytes(8)
            if i.size:
                assert got == (tmp_path / "alone").read_bytes(), (k, i.size // 3)
        s.close()
        one.close()
    torch.cuda.synchronize()
