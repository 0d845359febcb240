"""What is timed of this engine, and on which inputs.

A case is a dict of plain values.  prepare() makes what a program has in hand
before the call (meshes, rays, a built scene, a server), run() makes one pass
through the public entry points of heavyrt_gb300, work() says what a pass
cannot do without, and exact() gives the same outputs by brute force in 64
bits where that is quick.

The operations:
  trace      query_device on device arrays: the batched RayQuery_* of a host
             that keeps its rays on the GPU
  host       RayQuery_NearestHit / RayQuery_AnyHit on numpy arrays
  build      a mesh loaded: ClearGeom, AddGeom, AddInstance, CommitScene, the
             primitive order read back, and a first few rays
  refit      one frame of a deforming mesh: UpdateGeom (BUILD_REFIT),
             CommitScene, the frame's eye rays
  instances  one frame of a scene of instances in which one moves:
             UpdateInstance, CommitScene, the frame's eye rays
  batch      many small scenes loaded at once: add_geoms_batched and a first
             few rays of each
  graph      the rays of many small scenes, nearest and any hit, by one
             captured graph
  frame      a frame of the ambient-occlusion renderer
  served     a burst of requests to a server's resident scenes
"""
import math

import numpy as np
import torch

from heavyrt_gb300 import BUILD_HIGH, BUILD_REFIT, Frame, SceneRT, rtao_qmc_tile
from heavyrt_gb300 import engine

NEAREST, ANY = 0, 1
CAMERA = ((0.0, -2.5, 1.5), (0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 60.0)  # a heightfield from its side
FRONT = ((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 60.0)  # a soup from +z
FAR = 100.0
LAYOUTS = ("bvh2", "bvh4_f32", "bvh4_f16", "bvh4_q8")
BRUTE_LIMIT = 1.0e10  # ray-triangle pairs that exact() takes on


def listed():
    return [
        # the smallest call: a picking or visibility query of a few rays, all latency
        {"name": "trace_tiny", "op": "trace", "mesh": "soup", "tris": 2003, "layout": "bvh2", "tree": "reference",
         "test": "mt", "query": "nearest", "rays": "random", "count": 96, "shape": "default"},
        # a full-HD primary pass with a scene and a launch shape left at their defaults
        {"name": "eye_bvh2", "op": "trace", "mesh": "field", "tris": 2097152, "layout": "bvh2", "tree": "reference",
         "test": "mt", "query": "nearest", "rays": "eye", "width": 1920, "height": 1080, "shape": "default"},
        # the ambient-occlusion pass of the benchmark's frame, on its tree and launch shape
        {"name": "ao_any_f16", "op": "trace", "mesh": "field", "tris": 2097152, "layout": "bvh4_f16",
         "tree": "quality", "test": "mt", "query": "any", "rays": "ao", "count": 4000000, "shape": "tuned"},
        # incoherent rays (path tracing, particle transport) with the watertight test
        {"name": "random_q8_watertight", "op": "trace", "mesh": "soup", "tris": 1000003, "layout": "bvh4_q8",
         "tree": "reference", "test": "watertight", "query": "nearest", "rays": "random", "count": 1048579,
         "shape": "default"},
        # the small configuration (65,536 triangles, 512 x 512 eye rays) through numpy arrays
        {"name": "host_eye_bvh2", "op": "host", "mesh": "soup", "tris": 65536, "layout": "bvh2", "tree": "reference",
         "test": "mt", "query": "nearest", "rays": "eye", "width": 512, "height": 512},
        # loading the benchmark's mesh
        {"name": "build_field_f16", "op": "build", "mesh": "field", "tris": 2097152, "layout": "bvh4_f16",
         "tree": "quality", "test": "mt"},
        # loading a set of small meshes at once
        {"name": "batch_build_f16", "op": "batch", "scenes": 48, "tris_lo": 1024, "tris_hi": 32768,
         "layout": "bvh4_f16", "rays_each": 1024},
        # a deforming mesh, frame after frame
        {"name": "refit_field_f16", "op": "refit", "mesh": "field", "tris": 500000, "layout": "bvh4_f16",
         "tree": "reference", "test": "mt", "width": 640, "height": 360},
        # a scene of instances, one of which moves in each frame
        {"name": "instances_f32", "op": "instances", "instances": 240, "geoms": 3, "tris": 20000,
         "layout": "bvh4_f32", "width": 1280, "height": 720},
        # the rays of many small scenes in one captured graph
        {"name": "graph_f16", "op": "graph", "scenes": 64, "tris_lo": 1024, "tris_hi": 65536, "rays_lo": 4096,
         "rays_hi": 65536, "layout": "bvh4_f16"},
        # a frame of the ambient-occlusion renderer
        {"name": "rtao_frame_f16", "op": "frame", "tris": 1048352, "layout": "bvh4_f16", "width": 1280, "height": 720,
         "samples": 16},
        # a burst of requests of uneven sizes to a server
        {"name": "served_f16", "op": "served", "scenes": 8, "tris_lo": 10000, "tris_hi": 200000, "requests": 24,
         "rays_lo": 1000, "rays_hi": 200000, "layout": "bvh4_f16"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def tree(layout):
        return rng.choice(("reference", "quality")) if layout != "bvh2" else "reference"

    op = rng.choice(("trace", "trace", "trace", "host", "build", "batch", "refit", "instances", "graph", "frame",
                     "served"))
    layout = rng.choice(LAYOUTS)
    if op in ("trace", "host"):
        c = {"op": op, "mesh": rng.choice(("field", "soup")), "tris": log_int(1000, 2000000 if op == "trace" else 65536),
             "layout": layout, "tree": tree(layout), "test": rng.choice(("mt", "mt", "watertight")),
             "query": rng.choice(("nearest", "any"))}
        c["rays"] = rng.choice(("eye", "random", "ao")) if c["mesh"] == "field" else rng.choice(("eye", "random"))
        most = 2000000 if op == "trace" else 262144
        if c["rays"] == "eye":
            c["width"] = log_int(16, math.sqrt(1.7 * most))
            c["height"] = max(9, int(c["width"] * rng.uniform(0.4, 0.56)))
        else:
            c["count"] = log_int(64, most)
        if op == "trace":
            c["shape"] = rng.choice(("default", "tuned"))
        return c
    if op == "build":
        return {"op": op, "mesh": rng.choice(("field", "soup")), "tris": log_int(500, 1500000), "layout": layout,
                "tree": tree(layout), "test": rng.choice(("mt", "mt", "watertight"))}
    if op == "batch":
        return {"op": op, "scenes": log_int(2, 48), "tris_lo": 500, "tris_hi": log_int(2000, 32768), "layout": layout,
                "rays_each": 1024}
    if op == "refit":
        return {"op": op, "mesh": "field", "tris": log_int(2000, 500000), "layout": layout, "tree": tree(layout),
                "test": rng.choice(("mt", "watertight")), "width": 640, "height": 360}
    if op == "instances":
        width = log_int(160, 1280)
        return {"op": op, "instances": log_int(2, 240), "geoms": rng.randint(1, 4), "tris": log_int(1000, 20000),
                "layout": layout, "width": width, "height": width * 9 // 16}
    if op == "graph":
        return {"op": op, "scenes": log_int(2, 64), "tris_lo": 1024, "tris_hi": log_int(4096, 65536), "rays_lo": 1024,
                "rays_hi": log_int(4096, 65536), "layout": layout}
    if op == "frame":
        width = log_int(160, 1280)
        return {"op": op, "tris": log_int(5000, 1000000), "layout": layout, "width": width, "height": width * 9 // 16,
                "samples": rng.choice((1, 4, 8, 16))}
    return {"op": op, "scenes": log_int(1, 8), "tris_lo": 10000, "tris_hi": log_int(20000, 200000),
            "requests": log_int(1, 24), "rays_lo": 1000, "rays_hi": log_int(4000, 200000), "layout": layout}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000003 + 17)


def _uniform(gen, shape, lo=-1.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo


def _soup(gen, tris):
    """Random small triangles in [-1,1]^3, sized so that they overlap as 65,536 of offset 0.02 do."""
    off = 0.02 * (65536.0 / tris) ** (1.0 / 3.0)
    v = _uniform(gen, (tris, 1, 3)) + _uniform(gen, (tris, 3, 3), -off, off)
    return v.reshape(-1, 3).contiguous(), torch.arange(3 * tris, device="cuda", dtype=torch.int32)


def _quads(tris):
    return max(1, int(round(math.sqrt(tris / 2.0))))


def _heights(gen, x, y):
    """z of a sum of eight sines, amplitudes 0.1 / 2^k."""
    f, p = _uniform(gen, (8, 2), -3.0, 3.0).tolist(), _uniform(gen, (8,), 0.0, 2.0 * math.pi).tolist()
    z = torch.zeros_like(x)
    for k in range(8):
        z += 0.1 / 2**k * torch.sin((f[k][0] * x + f[k][1] * y) * 1.7**k + p[k])
    return z


def _field(gen, tris):
    """A heightfield mesh over [-1,1]^2: vertices, indices and the grid of heights."""
    q = _quads(tris)
    a = torch.linspace(-1.0, 1.0, q + 1, device="cuda")
    y, x = torch.meshgrid(a, a, indexing="ij")
    z = _heights(gen, x, y)
    v = torch.stack([x, y, z], dim=-1).reshape(-1, 3).contiguous()
    i = torch.arange(q, device="cuda")
    c = (i[:, None] * (q + 1) + i[None, :]).reshape(-1)
    idx = torch.stack([c, c + 1, c + q + 2, c, c + q + 2, c + q + 1], dim=-1)
    return v, idx.reshape(-1).to(torch.int32), z


def _mesh(case, gen):
    if case["mesh"] == "soup":
        v, idx = _soup(gen, case["tris"])
        return v, idx, None
    return _field(gen, case["tris"])


def _camera_rays(view, width, height, far=FAR):
    eye, target, up, fov = view
    e, t, u = (np.asarray(a, np.float64) for a in (eye, target, up))
    f = (t - e) / np.linalg.norm(t - e)
    r = np.cross(f, u)
    r /= np.linalg.norm(r)
    u = np.cross(r, f)
    s = math.tan(math.radians(fov) / 2.0)
    px = ((torch.arange(width, device="cuda", dtype=torch.float64) + 0.5) / width * 2 - 1) * s * width / height
    py = (1 - (torch.arange(height, device="cuda", dtype=torch.float64) + 0.5) / height * 2) * s
    d = px[None, :, None] * torch.tensor(r, device="cuda") + py[:, None, None] * torch.tensor(u, device="cuda")
    d = d + torch.tensor(f, device="cuda")
    d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)
    rays = torch.zeros((width * height, 8), device="cuda")
    rays[:, 0:3] = torch.tensor(e, device="cuda").float()
    rays[:, 4:7] = d.float()
    rays[:, 7] = far
    return rays


def _sphere_rays(gen, n):
    """Rays from a sphere of radius 3 towards uniform points of [-1,1]^3."""
    o = torch.randn((n, 3), generator=gen, device="cuda")
    o = 3.0 * o / o.norm(dim=-1, keepdim=True)
    d = _uniform(gen, (n, 3)) - o
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 0:3] = o
    rays[:, 4:7] = d / d.norm(dim=-1, keepdim=True)
    rays[:, 7] = FAR
    return rays


def _ao_rays(gen, z, n):
    """16 cosine-weighted rays from each of a raster of points of the heightfield (z: its grid of heights)."""
    q = z.shape[0] - 1
    points = (n + 15) // 16
    side = int(math.ceil(math.sqrt(points)))
    k = torch.arange(points, device="cuda")
    g = torch.stack([k % side, k // side], dim=-1) + torch.rand((points, 2), generator=gen, device="cuda")
    p = (g / side * 0.96 + 0.02) * q  # in cells, off the border
    c = p.floor().clamp(0, q - 1)
    f, c = p - c, c.long()
    z00, z10 = z[c[:, 1], c[:, 0]], z[c[:, 1], c[:, 0] + 1]
    z01, z11 = z[c[:, 1] + 1, c[:, 0]], z[c[:, 1] + 1, c[:, 0] + 1]
    low = f[:, 0] >= f[:, 1]
    sx, sy = torch.where(low, z10 - z00, z11 - z01), torch.where(low, z11 - z10, z01 - z00)
    h = 2.0 / q
    normal = torch.stack([-sx / h, -sy / h, torch.ones_like(sx)], dim=-1)
    normal = normal / normal.norm(dim=-1, keepdim=True)
    pos = torch.stack([p[:, 0] * h - 1, p[:, 1] * h - 1, z00 + f[:, 0] * sx + f[:, 1] * sy], dim=-1) + 1e-4 * normal
    a = torch.zeros_like(normal)
    a[:, 0] = 1.0
    tangent = torch.linalg.cross(normal, a)
    tangent = tangent / tangent.norm(dim=-1, keepdim=True)
    other = torch.linalg.cross(normal, tangent)
    u = torch.rand((points, 16, 2), generator=gen, device="cuda")
    r, phi = u[..., 0:1].sqrt(), 2.0 * math.pi * u[..., 1:2]
    d = r * phi.cos() * tangent[:, None] + r * phi.sin() * other[:, None] + (1 - u[..., 0:1]).sqrt() * normal[:, None]
    rays = torch.zeros((points, 16, 8), device="cuda")
    rays[..., 0:3] = pos[:, None]
    rays[..., 4:7] = d / d.norm(dim=-1, keepdim=True)
    rays[..., 7] = 0.28  # a tenth of the scene's diagonal
    return rays.reshape(-1, 8)[:n].contiguous()


def _rays(case, gen, z):
    if case["rays"] == "eye":
        return _camera_rays(CAMERA if case["mesh"] == "field" else FRONT, case["width"], case["height"])
    if case["rays"] == "random":
        return _sphere_rays(gen, case["count"])
    return _ao_rays(gen, z, case["count"])


def _log_uniform(n, lo, hi, start=0.5):
    """n sizes spread log-uniformly over [lo, hi], the same for every seed (a golden-ratio sequence)."""
    return [int(round(lo * (hi / lo) ** ((start + 0.6180339887498949 * k) % 1.0))) for k in range(n)]


def _matrices(gen, n):
    """Rotations and scales spread over [-1,1]^3 (row-major 4x4, float32)."""
    a = torch.randn((n, 4), generator=gen, device="cuda", dtype=torch.float64)
    w, x, y, z = (a / a.norm(dim=-1, keepdim=True)).unbind(-1)
    r = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=-1).reshape(n, 3, 3)
    s = _uniform(gen, (n,), 0.15, 0.35).double()
    m = torch.zeros((n, 4, 4), device="cuda", dtype=torch.float64)
    m[:, :3, :3] = r * s[:, None, None]
    m[:, :3, 3] = _uniform(gen, (n, 3)).double()
    m[:, 3, 3] = 1.0
    return m.float().cpu().numpy()


def _inputs(case, seed):
    """The meshes, rays and matrices of a case, all on the GPU (matrices on the host)."""
    gen, op = _generator(seed), case["op"]
    if op in ("trace", "host"):
        v, idx, z = _mesh(case, gen)
        return {"verts": v, "idx": idx, "rays": _rays(case, gen, z)}
    if op == "build":
        v, idx, _ = _mesh(case, gen)
        return {"verts": v, "idx": idx,
                "rays": _sphere_rays(gen, 4096) if case["mesh"] == "soup" else _camera_rays(CAMERA, 64, 64)}
    if op == "refit":
        v, idx, _ = _mesh(case, gen)
        moved = v.clone()
        moved[:, 2] += 0.05 * torch.sin(4.0 * v[:, 0] + _uniform(gen, (1,), 0.0, 6.0))
        return {"verts": v, "idx": idx, "moved": moved, "rays": _camera_rays(CAMERA, case["width"], case["height"])}
    if op == "instances":
        meshes = [_field(gen, case["tris"])[:2] if k % 2 == 0 else _soup(gen, case["tris"]) for k in range(case["geoms"])]
        return {"meshes": meshes, "matrices": _matrices(gen, case["instances"]), "moved": _matrices(gen, 1)[0],
                "rays": _camera_rays(FRONT, case["width"], case["height"])}
    if op in ("batch", "graph"):
        tris = _log_uniform(case["scenes"], case["tris_lo"], case["tris_hi"])
        n = ([case["rays_each"]] * case["scenes"] if op == "batch" else
             _log_uniform(case["scenes"], case["rays_lo"], case["rays_hi"], 0.2))
        return {"meshes": [_soup(gen, t) for t in tris], "rays": [_sphere_rays(gen, k) for k in n]}
    if op == "frame":
        v, idx, z = _field(gen, case["tris"])
        h = 2.0 / _quads(case["tris"])
        dy, dx = torch.gradient(z, spacing=h)
        nrm = torch.stack([-dx, -dy, torch.ones_like(dx)], dim=-1).reshape(-1, 3)
        nrm = torch.nn.functional.pad(nrm / nrm.norm(dim=-1, keepdim=True), (0, 1))
        return {"verts": v, "idx": idx, "normals": nrm}
    tris = _log_uniform(case["scenes"], case["tris_lo"], case["tris_hi"])
    meshes = [_soup(gen, t) if k % 2 else _field(gen, t)[:2] for k, t in enumerate(tris)]
    n = _log_uniform(case["requests"], case["rays_lo"], case["rays_hi"], 0.2)
    return {"meshes": meshes, "rays": [_sphere_rays(gen, k) for k in n]}


# ---------------------------------------------------------------- states
def _scene(case):
    s = SceneRT(layout=case["layout"], triangle_test=case.get("test", "mt"))
    if case.get("tree") == "quality":
        s.set_bvh4_merge(1)
        s.set_morton_frame(engine.MORTON_CUBIC)
        s.set_bvh4_collapse(engine.BVH4_COLLAPSE_LARGEST_FIRST)
    return s


def _host_mesh(mesh):
    return mesh[0].cpu().numpy(), mesh[1].cpu().numpy().view(np.uint32)


def _add(scene, verts, idx):
    return scene.AddGeom_Triangles3f(verts, len(verts), idx, idx.size, BUILD_HIGH, 12)


def _hit_views(hits):
    """The views of an array of hits that a program reads: t, the three ids, the coordinates."""
    return {"t": hits[:, 0], "ids": hits.view(torch.int32)[:, 1:4], "coords": hits[:, 4:8]}


def _hit_buffer(n):
    hits = torch.zeros((n, 8), device="cuda")
    return hits, _hit_views(hits)


def _segments(counts):
    off = np.zeros(len(counts) + 1, np.int32)
    off[1:] = np.cumsum(counts)
    return torch.from_numpy(off).cuda(), torch.arange(len(counts), device="cuda", dtype=torch.int32)


def _prepare_trace(case, d, st):
    s = st["scene"] = _scene(case)
    v, idx = _host_mesh((d["verts"], d["idx"]))
    s.AddInstance(_add(s, v, idx))
    s.CommitScene()
    st["kind"] = NEAREST if case["query"] == "nearest" else ANY
    if case["op"] == "host":
        st["rays"] = d["rays"].cpu().numpy()
        return
    st["rays"], st["n"] = d["rays"], d["rays"].shape[0]
    if case["shape"] == "tuned":  # the shapes that the autotuner picks for the benchmark's frame
        if st["kind"] == NEAREST:
            s.set_trace_config(NEAREST, 128, 0, 16, 24, imageWidth=case.get("width", 0))
        else:
            s.set_trace_config(ANY, 128, 1, 8, 8)
    if st["kind"] == NEAREST:
        st["buffer"], st["out"] = _hit_buffer(st["n"])
    else:
        st["buffer"] = st["out"] = torch.zeros(st["n"], device="cuda", dtype=torch.uint8)


def _prepare_build(case, d, st):
    st["scene"] = _scene(case)
    st["verts"], st["idx"] = _host_mesh((d["verts"], d["idx"]))
    st["rays"] = d["rays"]
    st["buffer"], st["out"] = _hit_buffer(d["rays"].shape[0])


def _prepare_refit(case, d, st):
    s = st["scene"] = _scene(case)
    v, st["idx"] = _host_mesh((d["verts"], d["idx"]))
    st["geom"] = _add(s, v, st["idx"])
    s.AddInstance(st["geom"])
    s.CommitScene()
    st["moved"], st["rays"] = d["moved"].cpu().numpy(), d["rays"]
    st["buffer"], st["out"] = _hit_buffer(d["rays"].shape[0])


def _prepare_instances(case, d, st):
    s = st["scene"] = _scene(case)
    ids = [_add(s, *_host_mesh(m)) for m in d["meshes"]]
    for k, m in enumerate(d["matrices"]):
        s.AddInstance(ids[k % len(ids)], m)
    s.CommitScene()
    st["moved"], st["rays"] = d["moved"], d["rays"]
    st["buffer"], st["out"] = _hit_buffer(d["rays"].shape[0])


def _prepare_many(case, d, st):
    s = st["scene"] = _scene(dict(case, tree="quality"))
    meshes = [_host_mesh((torch.nn.functional.pad(v, (0, 1), value=1.0), idx)) for v, idx in d["meshes"]]
    st["verts"], st["idx"] = [m[0] for m in meshes], [m[1] for m in meshes]  # float4 vertices, as the engine keeps them
    st["rays"] = torch.cat(d["rays"])
    n = st["rays"].shape[0]
    st["offsets"], st["instances"] = _segments([r.shape[0] for r in d["rays"]])
    st["buffer"], st["out"] = _hit_buffer(n)
    desc = [engine.query_desc(NEAREST, st["rays"].data_ptr(), n, st["buffer"].data_ptr(), st["offsets"].data_ptr(),
                              st["instances"].data_ptr(), len(meshes))]
    if case["op"] == "batch":
        st["desc"] = desc[0]
        return
    for g in s.add_geoms_batched(st["verts"], st["idx"]):
        s.AddInstance(g)
    s.CommitScene()
    st["any"] = torch.zeros(n, device="cuda", dtype=torch.uint8)
    desc.append(engine.query_desc(ANY, st["rays"].data_ptr(), n, st["any"].data_ptr(), st["offsets"].data_ptr(),
                                  st["instances"].data_ptr(), len(meshes)))
    st["graph"] = s.capture(desc)


def _prepare_frame(case, d, st):
    from heavyrt_gb300.workload import camera_inverses

    s = st["scene"] = _scene(dict(case, tree="quality"))
    g = _add(s, *_host_mesh((d["verts"], d["idx"])))
    s.AddInstance(g)
    s.CommitScene()
    f = st["frame"] = Frame()
    f.set_normals(g, d["normals"].cpu().numpy())
    f.set_ao_tile(rtao_qmc_tile(case["samples"]), case["samples"])
    st["camera"] = camera_inverses(*CAMERA, case["width"], case["height"])
    st["size"] = (case["width"], case["height"])
    st["colors"] = torch.zeros(case["width"] * case["height"], device="cuda", dtype=torch.int32)


def _prepare_served(case, d, st):
    sv = st["server"] = engine.Server(memory_budget=8 << 30, slot_rays=4 << 20, layout=case["layout"], bvh4_merge=1,
                                      morton_frame=engine.MORTON_CUBIC)
    st["scenes"] = [sv.add_scene(*_host_mesh(m), evictable=False) for m in d["meshes"]]
    for k in st["scenes"]:
        if sv.scene_state(k, -1.0) != engine.SCENE_READY:
            raise RuntimeError("a served scene was not built")
    st["requests"], st["buffers"], st["out"] = [], [], []
    for k, r in enumerate(d["rays"]):
        kind = k % 2
        if kind == NEAREST:
            buffer = torch.zeros((r.shape[0], 8), pin_memory=True)
            out = _hit_views(buffer)
        else:
            buffer = out = torch.zeros(r.shape[0], dtype=torch.uint8, pin_memory=True)
        rays = r.cpu().pin_memory()
        st["buffers"].append((rays, buffer))
        st["requests"].append((st["scenes"][k % len(st["scenes"])], kind, rays.data_ptr(), r.shape[0],
                               buffer.data_ptr()))
        st["out"].append(out)


_PREPARE = {"trace": _prepare_trace, "host": _prepare_trace, "build": _prepare_build, "refit": _prepare_refit,
            "instances": _prepare_instances, "batch": _prepare_many, "graph": _prepare_many, "frame": _prepare_frame,
            "served": _prepare_served}


def prepare(case, seed):
    st = {"op": case["op"], "stream": torch.cuda.current_stream().cuda_stream}
    _PREPARE[case["op"]](case, _inputs(case, seed), st)
    torch.cuda.synchronize()  # the engine's own streams do not wait for the inputs' kernels
    return st


# ---------------------------------------------------------------- passes
def _run_trace(st):
    st["scene"].query_device(st["kind"], st["rays"].data_ptr(), st["n"], st["buffer"].data_ptr(), st["stream"])
    return st["out"]


def _run_host(st):
    if st["kind"] == ANY:
        return st["scene"].RayQuery_AnyHit(st["rays"])
    h = st["scene"].RayQuery_NearestHit(st["rays"])
    return {"t": h["t"], "ids": h.view(np.uint32).reshape(-1, 8)[:, 1:4], "coords": h["coords"]}


def _trace_rays(st):
    st["scene"].query_device(NEAREST, st["rays"].data_ptr(), st["rays"].shape[0], st["buffer"].data_ptr(), st["stream"])


def _run_build(st):
    s = st["scene"]
    s.ClearGeom()
    g = _add(s, st["verts"], st["idx"])
    s.AddInstance(g)
    s.CommitScene()
    _trace_rays(st)
    return {"order": s.export(g, engine.EXPORT_PRIM_INDICES), "boxes": s.GetGeomBoxes(), "hits": st["out"]}


def _run_refit(st):
    s, v, idx = st["scene"], st["moved"], st["idx"]
    s.UpdateGeom_Triangles3f(st["geom"], v, len(v), idx, idx.size, BUILD_REFIT, 12)
    s.CommitScene()
    _trace_rays(st)
    return {"boxes": s.GetGeomBoxes(), "hits": st["out"]}


def _run_instances(st):
    st["scene"].UpdateInstance(0, st["moved"])
    st["scene"].CommitScene()
    _trace_rays(st)
    return st["out"]


def _run_batch(st):
    s = st["scene"]
    s.ClearGeom()
    for g in s.add_geoms_batched(st["verts"], st["idx"]):
        s.AddInstance(g)
    s.CommitScene()
    s.query_multi(st["desc"], st["stream"])
    return {"boxes": s.GetGeomBoxes(), "hits": st["out"]}


def _run_graph(st):
    st["graph"].launch(st["stream"])
    return {"hits": st["out"], "any": st["any"]}


def _run_frame(st):
    st["frame"].render_rtao(st["scene"], *st["camera"], *st["size"], st["colors"].data_ptr(), ao_max_radius=0.28,
                            stream=st["stream"])
    return st["colors"]


def _run_served(st):
    sv = st["server"]
    for t in [sv.submit(*r) for r in st["requests"]]:
        status, _ = sv.wait(t)
        if status != engine.HRT_OK:
            raise RuntimeError("a request failed")
    return st["out"]


_RUN = {"trace": _run_trace, "host": _run_host, "build": _run_build, "refit": _run_refit, "instances": _run_instances,
        "batch": _run_batch, "graph": _run_graph, "frame": _run_frame, "served": _run_served}


def run(state):
    return _RUN[state["op"]](state)


# ---------------------------------------------------------------- work
def work(case):
    """Rays in and results out once, the meshes in once where they are built, and for each ray one path down a 4-wide
    tree (four boxes of 22 operations a level) and one triangle test (52), with the 36 bytes of that triangle."""
    op = case["op"]

    def mean(lo, hi):
        return (hi - lo) / math.log(hi / lo) if hi > lo else lo

    def traced(rays, tris, result):
        levels = max(1.0, math.log(max(tris, 4), 4))
        return np.array([rays * (32.0 + result) + 36.0 * min(rays, tris), rays * (levels * 88.0 + 52.0)])

    def built(tris, verts):
        # vertices and indices in; 48 B a triangle and 64 B a 4-wide node (a third as many) out
        return np.array([12.0 * verts + 12.0 * tris + (48.0 + 21.0) * tris, 40.0 * tris])

    if op in ("trace", "host"):
        n = case["width"] * case["height"] if case["rays"] == "eye" else case["count"]
        w = traced(n, case["tris"], 32 if case["query"] == "nearest" else 1)
    elif op in ("build", "refit"):
        t = case["tris"]
        w = built(t, t / 2 if case["mesh"] == "field" else 3 * t)
        w += traced(4096 if op == "build" else case["width"] * case["height"], t, 32)
        w[0] += 4.0 * t if op == "build" else 0.0
    elif op == "instances":
        w = traced(case["width"] * case["height"], case["tris"] * case["geoms"], 32) + 112.0 * case["instances"]
    elif op == "batch":
        t = mean(case["tris_lo"], case["tris_hi"])
        w = case["scenes"] * (built(t, 3 * t) + traced(case["rays_each"], t, 32))
    elif op == "graph":
        t, n = mean(case["tris_lo"], case["tris_hi"]), mean(case["rays_lo"], case["rays_hi"])
        w = case["scenes"] * (traced(n, t, 32) + traced(n, t, 1))
    elif op == "frame":
        # the heightfield covers about an eighth of the image
        n = case["width"] * case["height"]
        w = traced(n, case["tris"], 32) + traced(n * case["samples"] / 8.0, case["tris"], 1) + 4.0 * n
    else:
        t, n = mean(case["tris_lo"], case["tris_hi"]), mean(case["rays_lo"], case["rays_hi"])
        w = case["requests"] / 2.0 * (traced(n, t, 32) + traced(n, t, 1))
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ---------------------------------------------------------------- 64 bits
def _brute(tris, rays, slack):
    """t and coordinates of the nearest hit of every ray, in 64 bits: tris [T, 3, 3], rays [n, 8]."""
    a, e1, e2 = tris[:, 0], tris[:, 1] - tris[:, 0], tris[:, 2] - tris[:, 0]
    n, t_count = rays.shape[0], tris.shape[0]
    t_out, coords = rays[:, 7].clone(), torch.zeros((n, 4), device="cuda", dtype=torch.float64)
    block_t = min(t_count, 1 << 18)
    block_r = max(1, (1 << 24) // block_t)
    for r0 in range(0, n, block_r):
        o, d = rays[r0:r0 + block_r, None, 0:3], rays[r0:r0 + block_r, None, 4:7]
        near, best = rays[r0:r0 + block_r, 3:4], t_out[r0:r0 + block_r]
        for t0 in range(0, t_count, block_t):
            E1, E2, A = e1[None, t0:t0 + block_t], e2[None, t0:t0 + block_t], a[None, t0:t0 + block_t]

            def cross(x, y):
                return (x[..., 1] * y[..., 2] - x[..., 2] * y[..., 1], x[..., 2] * y[..., 0] - x[..., 0] * y[..., 2],
                        x[..., 0] * y[..., 1] - x[..., 1] * y[..., 0])

            p = cross(d, E2)
            tv = o - A
            det = E1[..., 0] * p[0] + E1[..., 1] * p[1] + E1[..., 2] * p[2]
            inv = 1.0 / det
            v = (tv[..., 0] * p[0] + tv[..., 1] * p[1] + tv[..., 2] * p[2]) * inv
            q = cross(tv, E1)
            u = (d[..., 0] * q[0] + d[..., 1] * q[1] + d[..., 2] * q[2]) * inv
            t = (E2[..., 0] * q[0] + E2[..., 1] * q[1] + E2[..., 2] * q[2]) * inv
            ok = (u >= -slack) & (v >= -slack) & (u + v <= 1.0 + slack) & (t > near) & (t < best[:, None])
            t = torch.where(ok, t, torch.full((), math.inf, device="cuda", dtype=torch.float64))
            m, k = t.min(dim=1)
            better = m < best
            rows = torch.nonzero(better).reshape(-1)
            best[rows] = m[rows]
            coords[r0 + rows, 0] = u[rows, k[rows]]
            coords[r0 + rows, 1] = v[rows, k[rows]]
    return {"t": t_out, "ids": None, "coords": coords}


def _corners(verts, idx):
    return verts.double()[idx.long()].reshape(-1, 3, 3)


def _boxes(verts_list):
    one = torch.ones(1, device="cuda", dtype=torch.float64)
    return torch.stack([torch.cat([v.double().amin(0), one, v.double().amax(0), one]) for v in verts_list])


def exact(case, seed):
    got = _exact(case, seed)

    def some(v):
        return any(map(some, v.values() if isinstance(v, dict) else v)) if isinstance(v, (dict, list)) else v is not None

    return got if some(got) else None


def _exact(case, seed):
    op = case["op"]
    if op == "frame" or case.get("query") == "any":
        return None  # whole numbers only
    d = _inputs(case, seed)
    slack = 0.0 if case.get("test") == "watertight" else 1e-6

    def hits(tris, rays):
        if float(tris.shape[0]) * rays.shape[0] > BRUTE_LIMIT:
            return {"t": None, "ids": None, "coords": None}
        return _brute(tris, rays.double(), slack)

    if op in ("trace", "host"):
        return hits(_corners(d["verts"], d["idx"]), d["rays"])
    if op == "build":
        return {"order": None, "boxes": _boxes([d["verts"]]), "hits": hits(_corners(d["verts"], d["idx"]), d["rays"])}
    if op == "refit":
        return {"boxes": _boxes([d["moved"]]), "hits": hits(_corners(d["moved"], d["idx"]), d["rays"])}
    if op == "instances":
        matrices = torch.from_numpy(np.concatenate([d["moved"][None], d["matrices"][1:]])).cuda().double()
        if case["instances"] * case["tris"] * float(d["rays"].shape[0]) > BRUTE_LIMIT:
            return {"t": None, "ids": None, "coords": None}
        tris = [_corners(*d["meshes"][k % len(d["meshes"])]) @ m[:3, :3].T + m[:3, 3] for k, m in enumerate(matrices)]
        return hits(torch.cat(tris), d["rays"])
    pairs = sum(float(m[1].numel() / 3) * r.shape[0] for m, r in zip(d["meshes"], d["rays"]))
    none = {"t": None, "ids": None, "coords": None}
    if op == "served":
        if pairs > BRUTE_LIMIT:
            return [none if k % 2 == NEAREST else None for k in range(case["requests"])]
        return [_brute(_corners(*d["meshes"][k % case["scenes"]]), r.double(), slack) if k % 2 == NEAREST else None
                for k, r in enumerate(d["rays"])]
    got = none
    if pairs <= BRUTE_LIMIT:
        each = [_brute(_corners(*m), r.double(), slack) for m, r in zip(d["meshes"], d["rays"])]
        got = {"t": torch.cat([e["t"] for e in each]), "ids": None, "coords": torch.cat([e["coords"] for e in each])}
    if op == "graph":
        return {"hits": got, "any": None}
    return {"boxes": _boxes([m[0] for m in d["meshes"]]), "hits": got}
