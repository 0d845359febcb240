"""The frame's AO slots: images of less than a block of rays, a block more or
less, ragged sides (rays in rows, not tiles), many samples and none hit; slots
follow the traced order, each slot's rays start at its pixel's hit, and pixels
without a hit are 0 also where an earlier frame had hits."""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples", [1, 3, 16])
@pytest.mark.parametrize("width,height", [(1, 1), (8, 8), (16, 16), (17, 15), (257, 1), (64, 40), (331, 203), (1024, 520)])
def test_slots_and_cleared_pixels(native, width, height, samples):
    import torch

    from heavyrt_gb300 import Frame, SceneRT, rtao_qmc_tile
    from heavyrt_gb300 import engine as E

    z = dict(np.load(GOLDEN / "render_frames.npz"))
    s = SceneRT(layout=2)
    g = s.AddGeom_Triangles3f(z["verts"], len(z["verts"]), z["idx"], z["idx"].size, vByteStride=16)
    s.AddInstance(g)
    s.CommitScene()
    f = Frame()
    f.set_ao_tile(rtao_qmc_tile(samples), samples)
    f.set_normals(g, z["normals"])
    n = width * height
    colors = torch.full((n,), 0x7F, dtype=torch.int32, device="cuda")
    view = z["a_world_view_inv"].astype(np.float32)
    away = view.copy()
    away[:3, 3] += 1.0e4
    seen = []
    for v in (view, away, view):
        f.render_rtao(s, z["a_proj_inv"], v, width, height, colors.data_ptr(), ao_max_radius=1.0)
        torch.cuda.synchronize()
        hits, pixel, pos = f.read(E.FRAME_EYE_HITS), f.read(E.FRAME_RAY_PIXEL), f.read(E.FRAME_POSITIONS)
        slots, rays, vis = f.read(E.FRAME_AO_PIXEL), f.read(E.FRAME_AO_RAYS), f.read(E.FRAME_VISIBILITY)
        hit = hits.view(np.uint32)[:, 3] != 0xFFFFFFFF
        np.testing.assert_array_equal(slots, pixel[hit])
        assert rays.shape[0] == samples * len(slots)
        # every ray starts at its slot's hit, within the offset
        near = np.abs(rays.reshape(-1, samples, 8)[:, :, :3] - pos[slots][:, None, :3])
        assert near.size == 0 or near.max() <= 1.0e-4 * max(1.0, np.abs(pos[slots][:, :3]).max())
        other = np.setdiff1d(np.arange(n), slots)
        got = colors.cpu().numpy()
        assert not got[other].any() and not vis[other].any()
        assert (got[slots].view(np.uint32) >> 24 == 255).all()
        seen.append((len(slots), got, vis))
    assert seen[1][0] == 0 and seen[0][0] == seen[2][0]
    np.testing.assert_array_equal(seen[0][1], seen[2][1])
    np.testing.assert_array_equal(seen[0][2], seen[2][2])
    f.close()
    s.close()
