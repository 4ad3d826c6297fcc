"""The workloads that say how fast this library is: what a renderer has it do,
through its public entry points, from the smallest frame to the largest.

  frame       one frame of the reference's pass order (Context.render_frame, or
              Context.render_frame_host for a program whose planes are on the
              host)
  passes      a program that runs the passes itself with biased spatial reuse
  visibility  a batch of shadow segments (Context.visibility_batch)
  gbuffer     the primary-ray G-buffer (Context.trace_gbuffer)
  tree        the reference's tree built on the device (rg_build_bvh_device)
  infer       the learned proposal's inference over a frame
  gradients   one gradient of the learned proposal (a training step's work)
  batch       many views of one scene, one launch per pass (passes.Batch)

Scenes are the three of restir_gb300.scenes: "boxes" (config 1: 768 cube
triangles in a room, uniform source pdf), "soup" (config 2: random triangles,
power-proportional pdf) and "rocks" (config 3: instanced rocks, clustered
heavy-tailed lights), reseeded and resized.  Every pass of a case is the same
work: a frame with temporal reuse reads a previous frame that `prepare`
rendered and that the frame does not overwrite.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "restir-vulkan_gb300"))

from restir_gb300 import _lib, scenes  # noqa: E402
from restir_gb300.passes import Batch, Context, DeviceGBuffer, reservoirs  # noqa: E402

FRAME = {"kind": "frame", "scene": "soup", "triangles": 100_000, "lights": 65_536, "width": 1920, "height": 1080,
         "candidates": 32, "unbiased": True, "spatial": 2, "neighbors": 5, "temporal": True, "samples": 1, "mis": 0,
         "host": False}


def listed():
    return [
        # the smallest frame: config 1, biased reuse, one still image; four launches, so latency counts
        {**FRAME, "name": "frame_boxes_256", "scene": "boxes", "triangles": 780, "lights": 1024, "width": 256,
         "height": 256, "unbiased": False, "spatial": 1, "temporal": False},
        # the benchmark's frame: config 3, 1.05M triangles and 1M lights, three chained unbiased passes
        {**FRAME, "name": "frame_rocks_1080p", "scene": "rocks", "triangles": 1_048_576, "lights": 1_048_576,
         "spatial": 3},
        # config 2 for a program whose G-buffer is on the host: planes copied in, image copied out
        {**FRAME, "name": "host_frame_soup_1080p", "host": True},
        # the reference's RESERVOIR_SIZE 2 and UNBIASED_MIS build, its own NUM_NEIGHBORS, an odd window
        {**FRAME, "name": "frame_mis2_641x359", "triangles": 20_000, "lights": 4096, "width": 641, "height": 359,
         "spatial": 1, "neighbors": 3, "samples": 2, "mis": 1},
        # the reference's default mode: temporal and two biased dispatches, on a device that offers SNORM
        # normals, RGB32F positions and D24 depth (the first formats of the reference's lists)
        {"name": "passes_biased_720p", "kind": "passes", "scene": "soup", "triangles": 100_000, "lights": 65_536,
         "width": 1280, "height": 720, "candidates": 32, "neighbors": 5, "formats": "compact"},
        # a small odd batch of shadow queries: one launch that cannot fill the chip
        {"name": "visibility_2003", "kind": "visibility", "scene": "boxes", "triangles": 780, "lights": 1024,
         "segments": 2003},
        # a large batch of shadow queries against the largest scene
        {"name": "visibility_rocks_2m", "kind": "visibility", "scene": "rocks", "triangles": 1_048_576,
         "lights": 65_536, "segments": 2_000_000},
        # the G-buffer of the benchmark's frame, for a program without a rasteriser
        {"name": "gbuffer_rocks_1080p", "kind": "gbuffer", "scene": "rocks", "triangles": 1_048_576, "lights": 1024,
         "width": 1920, "height": 1080},
        # the tree of the largest scene, rebuilt for moved geometry
        {"name": "tree_rocks_1m", "kind": "tree", "scene": "rocks", "triangles": 1_048_576},
        # config 4's inference, once per frame
        {"name": "infer_1080p_4096", "kind": "infer", "width": 1920, "height": 1080, "clusters": 4096,
         "lights": 65_536, "candidates": 32},
        # config 4's training batch
        {"name": "gradients_64k_4096", "kind": "gradients", "width": 1920, "height": 1080, "clusters": 4096,
         "lights": 65_536, "rows": 65_536},
        # config 5 at a quarter of its views
        {"name": "batch_soup_16", "kind": "batch", "scene": "soup", "triangles": 100_000, "lights": 65_536,
         "views": 16, "min_width": 320, "max_width": 1920, "candidates": 32, "spatial": 2, "neighbors": 5,
         "learned": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_scene(rng):
    kind = rng.choice(["boxes", "soup", "soup", "rocks"])
    if kind == "boxes":
        return {"scene": kind, "triangles": 780, "lights": 1024}
    if kind == "soup":
        return {"scene": kind, "triangles": _log_int(rng, 500, 150_000), "lights": _log_int(rng, 64, 100_000)}
    return {"scene": kind, "triangles": 32 * _log_int(rng, 4, 32) ** 3, "lights": _log_int(rng, 5000, 500_000)}


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "passes", "visibility", "gbuffer", "tree", "infer", "gradients",
                       "batch"])
    size = {"width": _log_int(rng, 33, 1920), "height": _log_int(rng, 19, 1080)}
    if kind == "frame":
        samples = rng.choice([1, 1, 1, 2])
        return {"kind": kind, **_draw_scene(rng), **size, "candidates": rng.randint(4, 32),
                "unbiased": rng.random() < 0.75, "spatial": rng.randint(1, 2 if samples == 2 else 3),
                "neighbors": rng.randint(1, 5), "temporal": rng.random() < 0.7, "samples": samples,
                "mis": rng.choice([0, 0, 1]), "host": rng.random() < 0.25}
    if kind == "passes":
        return {"kind": kind, **_draw_scene(rng), **size, "candidates": rng.randint(4, 32),
                "neighbors": rng.randint(1, 8), "formats": rng.choice(["default", "compact"])}
    if kind == "visibility":
        return {"kind": kind, **_draw_scene(rng), "segments": _log_int(rng, 300, 4_000_000)}
    if kind == "gbuffer":
        return {"kind": kind, **_draw_scene(rng), **size}
    if kind == "tree":
        if rng.random() < 0.5:
            return {"kind": kind, "scene": "soup", "triangles": _log_int(rng, 100, 1_000_000)}
        return {"kind": kind, "scene": "rocks", "triangles": 32 * _log_int(rng, 3, 32) ** 3}
    clusters = 64 * _log_int(rng, 2, 64)
    if kind == "infer":
        return {"kind": kind, **size, "clusters": clusters, "lights": clusters * rng.randint(1, 24),
                "candidates": rng.randint(1, 32)}
    if kind == "gradients":
        return {"kind": kind, "width": 640, "height": 360, "clusters": clusters,
                "lights": clusters * rng.randint(1, 24), "rows": _log_int(rng, 500, 131_072)}
    return {"kind": "batch", "scene": "soup", "triangles": _log_int(rng, 1000, 100_000), "lights": 64 * 256,
            "views": rng.randint(2, 12), "min_width": 96, "max_width": _log_int(rng, 160, 960),
            "candidates": rng.randint(8, 32), "spatial": rng.randint(1, 2), "neighbors": rng.randint(1, 5),
            "learned": rng.random() < 0.4}


# ---------------------------------------------------------------- scenes
def _rock_grid(triangles):
    a = max(1, round((triangles / 32) ** (1 / 3)))
    return (2 * a, a, a)


def _scene(case, seed, width, height, frames):
    """A reseeded scene whose camera path has `frames` frames."""
    n, lights = case["triangles"], case["lights"]
    if case["scene"] == "boxes":
        s = scenes.config1(seed=seed, width=width, height=height)
        s.cameras = scenes.camera_path(np.random.default_rng(seed + 77), frames, width / height)
        return s
    if case["scene"] == "soup":
        return scenes.config2(seed=seed, width=width, height=height, n_tris=n, n_lights=lights, frames=frames)
    return scenes.config3(seed=seed, width=width, height=height, grid=_rock_grid(n), n_lights=lights,
                          n_clusters=max(1, min(4096, lights // 16)), frames=frames)


def _trace(ctx, scene, frame):
    g = DeviceGBuffer(scene.width, scene.height)
    ctx.trace_gbuffer(scene.cameras[frame], g)
    return g


def _set(scene, case):
    scene.candidates = case["candidates"]
    scene.neighbors = case["neighbors"]
    scene.unbiased = bool(case.get("unbiased", False))
    scene.spatial_passes = case.get("spatial", 1)
    scene.temporal = bool(case.get("temporal", False))
    return scene


def _reservoir_parts(buf, samples=1, mis=0):
    """The fields of a reservoir buffer (int32 words per pixel): floats as floats, light index and count as integers."""
    f = buf.view(torch.float32)
    words = 16 if mis else 12
    out = {"count": buf[:, samples * words]}
    for j in range(samples):
        w = j * words
        out[f"sample{j}"] = f[:, w:w + 8]
        out[f"light{j}"] = buf[:, w + 8]
        out[f"weights{j}"] = f[:, w + 9:w + (13 if mis else 12)]
    return out


class _Span:
    """Device memory of a context; the tensors made from it keep the context."""

    def __init__(self, ctx, ptr, nbytes):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (nbytes // 4,), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _words(ctx, ptr, nbytes):
    return torch.as_tensor(_Span(ctx, ptr, nbytes), device="cuda")


class CompactGBuffer:
    """A G-buffer's planes as RGB16_SNORM normals, RGB32F positions and D24S8 depth."""

    def __init__(self, g):
        self.width, self.height = g.width, g.height
        n = g.planes["normal"].view(torch.float16)[..., :3].float().clamp(-1.0, 1.0)
        d = (g.planes["depth"].double().clamp(0.0, 1.0) * 16777215.0).round()
        self.planes = {"albedo": g.planes["albedo"], "material": g.planes["material"],
                       "normal": (n * 32767.0).round().to(torch.int16).contiguous(),
                       "world_pos": g.planes["world_pos"][..., :3].contiguous(), "depth": d.to(torch.int32)}

    def struct(self):
        p = self.planes
        return _lib.GBuffer(self.width, self.height, p["albedo"].data_ptr(), p["normal"].data_ptr(),
                            p["material"].data_ptr(), p["world_pos"].data_ptr(), p["depth"].data_ptr(),
                            _lib.FORMAT_R16G16B16_SNORM, _lib.FORMAT_R32G32B32_SFLOAT,
                            _lib.FORMAT_D24_UNORM_S8_UINT, 0)


# ---------------------------------------------------------------- the learned proposal's inputs, in plain torch
def _room_gbuffer(width, height, seed, dtype=torch.float32):
    """Positions and unit normals of a camera's pixels in the empty unit room, and the camera's position."""
    rng = np.random.default_rng(seed)
    cam = rng.uniform(0.25, 0.75, 3)
    fwd = rng.normal(size=3)
    fwd /= np.linalg.norm(fwd)
    right = np.cross(fwd, [0.0, 1.0, 0.0])
    right /= np.linalg.norm(right)
    up = np.cross(right, fwd)
    y, x = torch.meshgrid(torch.arange(height, dtype=torch.float64), torch.arange(width, dtype=torch.float64),
                          indexing="ij")
    vx = ((x + 0.5) / width * 2 - 1).cuda()[..., None] * (width / height)
    vy = ((y + 0.5) / height * 2 - 1).cuda()[..., None]
    t = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")  # noqa: E731
    d = vx * t(right) - vy * t(up) + t(fwd)
    c = t(cam.astype(np.float32).astype(np.float64))
    dist, axis = torch.where(d > 0, (1.0 - c) / d, -c / d).min(-1)
    pos = (c + dist[..., None] * d).float()
    normal = torch.zeros_like(pos)
    normal.scatter_(-1, axis[..., None], -torch.gather(d, -1, axis[..., None]).sign().float())
    return pos.reshape(-1, 3), normal.reshape(-1, 3), [float(v) for v in c]


def _network(case, seed):
    """Lights, their clusters and the network's parameters (He-uniform hidden layers, a spread logit layer)."""
    rng = np.random.default_rng(seed + 1)
    n, c = case["lights"], case["clusters"]
    pos = rng.uniform(0.0, 1.0, (n, 3))
    lum = np.exp(rng.uniform(math.log(0.01), math.log(100.0), n))
    cell = np.floor(pos * 16).astype(np.int64)
    order = np.lexsort((pos[:, 2], cell[:, 1], cell[:, 0]))
    cluster = np.empty(n, np.int32)
    cluster[order] = (np.arange(n) * c // n).astype(np.int32)
    w1 = np.zeros((16, 64))
    w1[:9] = rng.uniform(-1, 1, (9, 64)) * math.sqrt(6 / 9)
    w2, w3 = (rng.uniform(-1, 1, (64, 64)) * math.sqrt(6 / 64) for _ in range(2))
    w4 = rng.normal(0.0, 0.25, (64, c))
    b1, b2, b3 = (rng.normal(0.0, 0.1, 64) for _ in range(3))
    power = np.bincount(cluster, weights=lum, minlength=c)
    b4 = np.log(power)
    parts = [w1, b1, w2, b2, w3, b3, w4, b4]
    return pos, lum, cluster, np.concatenate([p.ravel() for p in parts]).astype(np.float32)


def _unpack(params, c):
    shapes = [(16, 64), (64,), (64, 64), (64,), (64, 64), (64,), (64, c), (c,)]
    out, at = [], 0
    for s in shapes:
        k = int(np.prod(s))
        out.append(torch.from_numpy(params[at:at + k].reshape(s)).double().cuda())
        at += k
    return out


def _bf16(t):
    return t.float().to(torch.bfloat16).double()


def _targets(case, seed):
    rng = np.random.default_rng(seed + 2)
    px = case["width"] * case["height"]
    rows = (np.arange(case["rows"], dtype=np.int64) * 31 + int(rng.integers(px))) % px
    target = rng.integers(0, case["clusters"], case["rows"]).astype(np.int32)
    target[rng.uniform(size=case["rows"]) < 0.05] = -1  # pixels whose reservoir kept no light
    return rows.astype(np.int32), target


def _learned_context(case, seed):
    s = scenes.config1(seed=seed, width=64, height=64)
    pos, lum, cluster, params = _network(case, seed)
    s.point_lights = scenes.make_point_lights(pos, np.repeat(lum[:, None], 3, 1))
    s.alias = scenes.build_alias(s.point_lights)
    ctx = Context(0)
    ctx.upload_scene(s)
    ctx.create_proposal(cluster, case["clusters"], mix=0.9, learning_rate=1e-2, batch=65536, seed=seed)
    ctx.set_proposal_params(params)
    p, n, cam = _room_gbuffer(case["width"], case["height"], seed)
    g = DeviceGBuffer(case["width"], case["height"])
    g.planes["world_pos"].view(-1, 4)[:, :3] = p
    g.planes["world_pos"].view(-1, 4)[:, 3] = 1.0
    g.planes["normal"].view(torch.float16).view(-1, 4)[:, :3] = n.half()
    return ctx, g, cam


def _features(pos, normal, cam):
    c = torch.tensor(cam, dtype=torch.float64, device="cuda")
    v = c - pos.double()
    v = v / v.norm(dim=-1, keepdim=True)
    x = torch.cat([(pos.double() - 0.5) * 2.0, normal.double(), v], -1)
    return _bf16(torch.cat([x, torch.zeros(len(x), 7, dtype=torch.float64, device="cuda")], -1))


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_frame(case, seed):
    s = _set(_scene(case, seed, case["width"], case["height"], 2), case)
    ctx = Context(0)
    ctx.set_reservoir_format(case["samples"], case["mis"])
    ctx.upload_scene(s)
    g = [_trace(ctx, s, f) for f in range(2)]
    image = torch.zeros((s.height, s.width, 4), dtype=torch.float32, device="cuda")
    st = {"case": case, "ctx": ctx, "g": g, "image": image, "params": s.frame_params(1), "scene": s}
    if not case["unbiased"]:
        # biased reuse writes through the previous frame's buffer: a still image, whose frames are all alike
        st["params"] = s.frame_params(0)
    if case["host"]:
        pin = lambda a: torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).pin_memory()  # noqa: E731
        st["planes"] = [{k: pin(v) for k, v in d.to_host().items()} for d in g]
        st["host_image"] = torch.zeros((s.height, s.width, 4), dtype=torch.float32).pin_memory()
        if case["unbiased"] and case["temporal"]:
            _host_frame(st, 0, s.frame_params(0))
    elif case["unbiased"] and case["temporal"]:
        ctx.render_frame(g[0], None, 0, s.frame_params(0), image)
    return st


def _host_frame(st, f, params):
    planes = {k: v.numpy() for k, v in st["planes"][f].items()}
    st["ctx"].render_frame_host(planes, params, st["host_image"].numpy())


def _prepare_passes(case, seed):
    s = _set(_scene(case, seed, case["width"], case["height"], 2), {**case, "temporal": True})
    ctx = Context(0)
    ctx.upload_scene(s)
    g = [_trace(ctx, s, f) for f in range(2)]
    if case["formats"] == "compact":
        g = [CompactGBuffer(x) for x in g]
    n = s.width * s.height
    res = [reservoirs(n) for _ in range(4)]
    ctx.initial_temporal(g[0], None, None, res[0], s.uniforms(0))
    return {"case": case, "ctx": ctx, "g": g, "res": res, "u": s.uniforms(1), "lu": s.lighting_uniforms(1),
            "image": torch.zeros((s.height, s.width, 4), dtype=torch.float32, device="cuda")}


def _prepare_visibility(case, seed):
    """Segments from surface points to lights, as the passes trace them."""
    n = case["segments"]
    w = max(8, min(1024, int(math.sqrt(n))))
    s = _scene(case, seed, w, w, 1)
    ctx = Context(0)
    ctx.upload_scene(s)
    g = _trace(ctx, s, 0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    px = (torch.arange(n, device="cuda") * (w * w) // n).clamp_(max=w * w - 1)  # neighbours in the image stay so
    p1 = g.planes["world_pos"].view(-1, 4)[px].contiguous()
    lights = torch.from_numpy(np.ascontiguousarray(s.point_lights["pos"])).cuda()
    p2 = lights[torch.randint(0, len(lights), (n,), generator=gen, device="cuda")].contiguous()
    return {"case": case, "ctx": ctx, "p1": p1, "p2": p2, "out": torch.zeros(n, dtype=torch.uint8, device="cuda")}


def _prepare_gbuffer(case, seed):
    s = _scene(case, seed, case["width"], case["height"], 1)
    ctx = Context(0)
    ctx.upload_scene(s)
    return {"case": case, "ctx": ctx, "camera": s.cameras[0], "g": DeviceGBuffer(s.width, s.height)}


def _triangles(case, seed):
    """The scene's triangles on the device, without its host-built tree."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = lambda lo, hi, *shape: lo + (hi - lo) * torch.rand(shape, generator=gen, device="cuda")  # noqa: E731
    room = torch.from_numpy(scenes.room_triangles()).cuda()
    if case["scene"] == "soup":
        n = case["triangles"]
        edge = torch.exp(u(math.log(1e-3), math.log(0.1), n, 1, 1))
        tris = u(0.0, 1.0, n, 1, 3) + edge * u(-0.5, 0.5, n, 3, 3)
        return torch.cat([room, tris.reshape(n, 9)]).contiguous()
    grid = _rock_grid(case["triangles"])
    n = grid[0] * grid[1] * grid[2]
    rng = np.random.default_rng(seed)
    verts, faces = scenes.rock_mesh(rng, n)
    rot = scenes.random_rotations(rng, n)
    cell = 1.0 / np.array(grid)
    ijk = np.stack(np.meshgrid(*(np.arange(k) for k in grid), indexing="ij"), -1).reshape(-1, 3)
    centers = (ijk + rng.uniform(0.25, 0.75, (n, 3))) * cell
    scale = rng.uniform(0.15, 0.35, (n, 1, 1)) * cell.min()
    to = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    world = torch.einsum("nij,nvj->nvi", to(rot), to(verts)) * to(scale) + to(centers)[:, None, :]
    return torch.cat([room, world[:, to(faces), :].reshape(n * 16, 9).float()]).contiguous()


def _prepare_tree(case, seed):
    xyz = _triangles(case, seed)
    n = len(xyz)
    return {"case": case, "ctx": Context(0), "xyz": xyz,
            "nodes": torch.zeros((n - 1) * 80, dtype=torch.uint8, device="cuda"),
            "tris": torch.zeros(n * 48, dtype=torch.uint8, device="cuda")}


def _prepare_infer(case, seed):
    ctx, g, cam = _learned_context(case, seed)
    u = _lib.RestirUniforms()
    u.camera_pos[:] = cam + [1.0]
    u.screen_size[:] = [case["width"], case["height"]]
    u.frame = 1
    u.initial_light_sample_count = case["candidates"]
    return {"case": case, "ctx": ctx, "g": g, "u": u}


def _prepare_gradients(case, seed):
    ctx, g, cam = _learned_context(case, seed)
    rows, target = _targets(case, seed)
    return {"case": case, "ctx": ctx, "g": g, "cam": cam, "rows": torch.from_numpy(rows).cuda(),
            "targets": torch.from_numpy(target).cuda()}


def _prepare_batch(case, seed):
    lo, hi = case["min_width"], case["max_width"]
    base = scenes.config2(seed=seed, width=lo, height=lo, n_tris=case["triangles"], n_lights=case["lights"], frames=1)
    rng = np.random.default_rng(seed + 5)
    ctx = Context(0)
    ctx.upload_scene(base)
    if case["learned"]:
        order = np.lexsort(np.floor(base.point_lights["pos"][:, :3].T * 16))
        cluster = np.empty(len(order), np.int32)
        cluster[order] = np.arange(len(order)) * 256 // len(order)
        ctx.create_proposal(cluster, 256, seed=seed)
    sizes = np.random.default_rng(5)  # the views' sizes are the case's, their cameras the seed's
    views = []
    for _ in range(case["views"]):
        w = int(round(math.exp(sizes.uniform(math.log(lo), math.log(hi)))))
        h = int(round(w * sizes.uniform(0.5, 0.8)))
        cam = scenes.camera_path(rng, 1, w / h)[0]
        s = _set(base.view(cam, w, h), {**case, "unbiased": True, "temporal": True})
        s.cameras = [cam, cam]  # a still camera: its own previous frame
        g = _trace(ctx, s, 0)
        u = s.uniforms(1)
        if case["learned"]:
            u.flags |= _lib.RG_FLAG_LEARNED_PROPOSAL
        views.append({"cur": g, "prev": g, "res0": reservoirs(w * h), "res1": reservoirs(w * h),
                      "tmp": reservoirs(w * h), "image": torch.zeros((h, w, 4), device="cuda"), "uniforms": u})
    b = Batch(ctx, views, s.frame_params(1))
    b.run(1)  # the previous frame of every later run: reservoirs[1]
    return {"case": case, "ctx": ctx, "batch": b, "views": views}


# ---------------------------------------------------------------- run
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_frame(st):
    case, ctx = st["case"], st["ctx"]
    if case["host"]:
        f = 1 if case["unbiased"] else 0
        _host_frame(st, f, st["params"])
        image, slot = st["host_image"], st["params"].uniforms.frame & 1
    else:
        cur, prev, slot = (st["g"][1], st["g"][0], 1) if case["unbiased"] else (st["g"][0], None, 0)
        ctx.render_frame(cur, prev, slot, st["params"], st["image"])
        image = st["image"]
    words = ctx.reservoir_bytes() // 4
    n = case["width"] * case["height"]
    res = _words(ctx, ctx.frame_reservoirs_ptr(slot), n * words * 4).view(n, words)
    return {"image": image[..., :3], "reservoirs": _reservoir_parts(res, case["samples"], case["mis"])}


def _run_passes(st):
    ctx, (prev, cur), (pr, r0, r1, r2), u = st["ctx"], st["g"], st["res"], st["u"]
    ctx.initial_temporal(cur, prev, pr, r0, u)
    ctx.spatial_biased(cur, r0, r1, u, 0)
    ctx.spatial_biased(cur, r1, r2, u, 1)
    ctx.shade(cur, r2, st["lu"], st["image"])
    return {"image": st["image"][..., :3], "ris": _reservoir_parts(r0), "reservoirs": _reservoir_parts(r2)}


def _run_visibility(st):
    st["ctx"].visibility_batch(st["p1"], st["p2"], st["out"])
    return st["out"]


def _run_gbuffer(st):
    st["ctx"].trace_gbuffer(st["camera"], st["g"])
    return dict(st["g"].planes)


def _run_tree(st):
    n = len(st["xyz"])
    undefined = C.c_int32(-1)
    count = _lib.check(_lib.lib().rg_build_bvh_device(
        st["ctx"]._h, st["xyz"].data_ptr(), n, st["nodes"].data_ptr(), st["tris"].data_ptr(), C.byref(undefined),
        torch.cuda.current_stream().cuda_stream))
    return {"nodes": st["nodes"], "triangles": st["tris"], "count": count, "undefined": undefined.value}


def _run_infer(st):
    case, ctx = st["case"], st["ctx"]
    ctx.proposal_infer(st["g"], st["u"])
    n, c = case["width"] * case["height"], case["candidates"]
    cand, stat = C.c_void_p(), C.c_void_p()
    _lib.check(_lib.lib().rg_proposal_buffers(ctx._h, C.byref(cand), C.byref(stat)))
    cd = _words(ctx, cand.value, n * 32 * 8).view(n, 32, 2)[:, :c]
    sv = _words(ctx, stat.value, n * 16).view(n, 4)
    return {"key": cd[..., 0], "q": cd.view(torch.float32)[..., 1], "lse": sv[:, 0].view(torch.float32),
            "mode": sv[:, 1], "mode_q": sv[:, 2].view(torch.float32)}


def _run_gradients(st):
    grad, loss = st["ctx"].proposal_gradients(st["g"], st["cam"], st["rows"], st["targets"])
    return {"grad": grad, "loss": loss}


def _run_batch(st):
    st["batch"].run(0)
    return [{"image": v["image"][..., :3], **_reservoir_parts(v["res0"])} for v in st["views"]][:12]


# ---------------------------------------------------------------- exact
def exact(case, seed):
    """64-bit values of what has one: a reservoir's random choices do not, the network's outputs do."""
    if case["kind"] == "infer":
        return _exact_infer(case, seed)
    if case["kind"] == "gradients":
        return _exact_gradients(case, seed)
    return None


def _hidden(x, net):
    w1, b1, w2, b2, w3, b3, _, _ = net
    h1 = _bf16(torch.relu(x @ _bf16(w1) + b1))
    h2 = _bf16(torch.relu(h1 @ _bf16(w2) + b2))
    return h1, h2, _bf16(torch.relu(h2 @ _bf16(w3) + b3))


def _exact_infer(case, seed):
    _, _, _, params = _network(case, seed)
    net = _unpack(params, case["clusters"])
    pos, normal, cam = _room_gbuffer(case["width"], case["height"], seed)
    w4, b4 = _bf16(net[6]), net[7]
    lse, top = [], []
    for at in range(0, len(pos), 32768):
        h = _hidden(_features(pos[at:at + 32768], normal[at:at + 32768], cam), net)[2]
        z = h @ w4 + b4
        l = torch.logsumexp(z, -1)
        lse.append(l)
        top.append(torch.exp(z.max(-1).values - l))
    return {"key": None, "q": None, "lse": torch.cat(lse), "mode": None, "mode_q": torch.cat(top)}


def _exact_gradients(case, seed):
    _, _, _, params = _network(case, seed)
    c = case["clusters"]
    net = _unpack(params, c)
    pos, normal, cam = _room_gbuffer(case["width"], case["height"], seed)
    rows, target = (torch.from_numpy(a).long().cuda() for a in _targets(case, seed))
    w2, w3, w4 = (_bf16(net[k]) for k in (2, 4, 6))
    grads = [torch.zeros_like(p) for p in net]
    loss = torch.zeros((), dtype=torch.float64, device="cuda")
    for at in range(0, len(rows), 16384):
        r, t = rows[at:at + 16384], target[at:at + 16384]
        x = _features(pos[r], normal[r], cam)
        h1, h2, h3 = _hidden(x, net)
        z = h3 @ w4 + net[7]
        lse = torch.logsumexp(z, -1)
        has = (t >= 0).double()
        zt = torch.gather(z, 1, t.clamp(min=0)[:, None])[:, 0]
        loss += ((lse - zt) * has).sum()
        dz = torch.exp(z - lse[:, None])
        dz.scatter_add_(1, t.clamp(min=0)[:, None], -torch.ones_like(zt)[:, None])
        dz *= (has / len(rows))[:, None]
        d3 = (dz @ w4.T) * (h3 > 0)
        d2 = (d3 @ w3.T) * (h2 > 0)
        d1 = (d2 @ w2.T) * (h1 > 0)
        for k, g in enumerate([x.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ d3, d3.sum(0), h3.T @ dz, dz.sum(0)]):
            grads[k] += g
    return {"grad": torch.cat([g.reshape(-1) for g in grads]), "loss": float(loss)}


# ---------------------------------------------------------------- work
# Bytes: G-buffer 36 B, reservoir 52 B of fields, image 16 B a pixel, a tree node 64 B and a triangle 36 B, a light
# 32 B and its alias column 16 B, each read or written once.  Operations: about 100 for a target function's value,
# and for a shadow segment two box tests of 25 at each level of a balanced tree.
def _segment_flops(triangles):
    return 50.0 * max(1.0, math.log2(max(2, triangles)))


def _scene_bytes(case):
    return case["triangles"] * 100.0 + case["lights"] * 48.0


def _frame_work(case, pixels):
    spatial = case["spatial"] * (1 if case["unbiased"] else 2)
    segments = 1 + (case["spatial"] * (case["neighbors"] + 1) if case["unbiased"] else 0)
    merges = case["candidates"] + (1 if case["temporal"] else 0) + spatial * case["neighbors"]
    s = case.get("samples", 1)
    per_pixel = 36 + 52.0 * s + 16 + (28 + 52.0 * s if case["temporal"] else 0)
    return {"bytes": per_pixel * pixels + _scene_bytes(case),
            "flops": pixels * s * (100.0 * merges + segments * _segment_flops(case["triangles"]))}


def work(case):
    kind = case["kind"]
    pixels = case.get("width", 0) * case.get("height", 0)
    if kind == "frame":
        return _frame_work(case, pixels)
    if kind == "passes":
        return _frame_work({**case, "spatial": 1, "unbiased": False, "temporal": True}, pixels)
    if kind == "visibility":
        return {"bytes": case["segments"] * 33.0 + case["triangles"] * 100.0,
                "flops": case["segments"] * _segment_flops(case["triangles"])}
    if kind == "gbuffer":
        return {"bytes": pixels * 36.0 + case["triangles"] * 108.0,
                "flops": pixels * _segment_flops(case["triangles"])}
    if kind == "tree":
        n = case["triangles"]
        return {"bytes": n * (36.0 + 80 + 48), "flops": n * 60.0 * max(1.0, math.log2(n))}
    if kind == "infer":
        c = case["clusters"]
        return {"bytes": pixels * (24.0 + 16 + 8 * case["candidates"]) + c * 64 * 2.0,
                "flops": 2.0 * pixels * (9 * 64 + 2 * 64 * 64 + 64 * c)}
    if kind == "gradients":
        n, c = case["rows"], case["clusters"]
        return {"bytes": n * (24.0 + 8) + c * 65 * 8.0, "flops": 6.0 * n * (9 * 64 + 2 * 64 * 64 + 64 * c)}
    rng = np.random.default_rng(5)
    lo, hi = case["min_width"], case["max_width"]
    total = 0
    for _ in range(case["views"]):
        w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        total += w * int(round(w * rng.uniform(0.5, 0.8)))
    w = _frame_work({**case, "unbiased": True, "temporal": True}, total)
    if case["learned"]:
        w["flops"] += 2.0 * total * (9 * 64 + 2 * 64 * 64 + 64 * 256)
    return w
