"""Timed workloads of the rasterizer: what a program draws with it, as calls of the Python
mirror of the reference's API (Rasterizer, VertexProcessor, BatchRenderer, DiffRenderer).

A case is a dict of plain values; `prepare` makes its inputs on the GPU from a seed and the
objects a program keeps between frames, `run` draws one frame (or one training step) and
returns the target's buffers, `work` counts the bytes and operations the frame cannot do
without, and `exact` restates the frame's computed numbers (depths, images, gradients) in
64 bits with plain torch.

Colours, drawPixel counts and winning primitives are whole numbers decided by comparisons,
so `exact` has no value for them; nor for the soup and the overwriting shaders, whose
frames write no other number or would take the plain rasterizer below too long.
"""
import math

import numpy as np
import torch

from softwarerenderer_gb300 import scenes
from softwarerenderer_gb300.abi import CullMode, DrawMode, PS, RasterMode, VS, make_uniforms
from softwarerenderer_gb300.batch import BatchRenderer
from softwarerenderer_gb300.device import DeviceTarget
from softwarerenderer_gb300.diff import DiffRenderer, render
from softwarerenderer_gb300.renderer import Rasterizer, VertexProcessor

CLEAR_DEPTH = 1.0  # the far end of the default depth range
SHADERS = {  # name: (vertex shader, pixel shader, texture edge, vertex bytes)
    "lambert": (VS.POS_NRM_UV, PS.LAMBERT, 0, 32),
    "lambert_tex": (VS.POS_NRM_UV, PS.LAMBERT_TEX, 512, 32),
    "texture": (VS.POS_NRM_UV, PS.TEX_NEAREST, 256, 32),
    "color": (VS.POS_RGB, PS.VCOLOR, 0, 24),
}
RASTER = {"span": RasterMode.Span, "block": RasterMode.Block, "adaptive": RasterMode.Adaptive}


# ---------------------------------------------------------------------------------------
# the cases

def listed():
    return [
        # The smallest program: the textured cube of the reference's tutorial, one synchronous
        # draw a frame.  Launches and host latency are all of it.
        {"name": "cube", "kind": "cube", "width": 640, "height": 480, "mip": False},
        # The reference's Box example: the same cube through the mip-mapped anisotropic sampler.
        {"name": "box_mip", "kind": "cube", "width": 640, "height": 480, "mip": True},
        # A viewer's ordinary frame: a mid-size textured mesh in a window of an odd size, the
        # reference's default Span mode, the per-pixel records a picking program reads.
        {"name": "mesh_span", "kind": "mesh", "tris": 20480, "width": 1283, "height": 717, "shader": "lambert_tex",
         "raster": "span", "graph": False, "sync": True, "records": True},
        # The headline frame: the dense icosphere at 1080p in Block mode, frames queued ahead
        # and replayed as CUDA graphs, as a renderer's main loop does.
        {"name": "mesh_dense", "kind": "mesh", "tris": 327680, "width": 1920, "height": 1080, "shader": "lambert",
         "raster": "block", "graph": True, "sync": False, "records": False},
        # The stress frame: a million independent triangles of all sizes at 4K, clipped at the
        # near and far planes, half of them culled.
        {"name": "soup_4k", "kind": "soup", "tris": 1048576, "width": 3840, "height": 2160, "raster": "adaptive"},
        # The reference's own Benchmark program: large random triangles over each other, an
        # overwriting pixel shader, no depth test.
        {"name": "benchmark", "kind": "overdraw", "tris": 40960, "width": 640, "height": 480, "raster": "span"},
        # Many meshes, each with its own camera, texture and target, in one submission.
        {"name": "batch_256", "kind": "batch", "meshes": 256, "max_tris": 200000},
        # A training step of differentiable rendering: forward, fused L2 loss, backward.
        {"name": "diff_16", "kind": "diff", "views": 16, "level": 6, "size": 512, "texture": 1024, "autograd": False},
        # A small step through torch.autograd, as an optimisation loop on one object runs it.
        {"name": "diff_small", "kind": "diff", "views": 2, "level": 4, "size": 129, "texture": 64, "autograd": True},
        # A wireframe overlay: every edge of a mesh drawn in Line mode.
        {"name": "wireframe", "kind": "lines", "lines": 122880, "width": 1920, "height": 1080},
        # A scanner's point cloud in Point mode.
        {"name": "points", "kind": "points", "points": 1000000, "width": 1920, "height": 1080},
        # A program with its own vertex stage: screen-space records straight to the Rasterizer.
        {"name": "triangle_list", "kind": "list", "tris": 60000, "width": 1280, "height": 720, "raster": "adaptive"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cube", "mesh", "mesh", "soup", "overdraw", "batch", "diff", "diff", "lines", "points", "list"])
    size = {"width": _log_int(rng, 161, 1920), "height": _log_int(rng, 121, 1080)}
    raster = rng.choice(["span", "block", "adaptive"])
    if kind == "cube":
        return {"kind": kind, **size, "mip": rng.random() < 0.5}
    if kind == "mesh":
        return {"kind": kind, "tris": _log_int(rng, 200, 327680), **size, "shader": rng.choice(sorted(SHADERS)),
                "raster": raster, "graph": rng.random() < 0.5, "sync": rng.random() < 0.5, "records": rng.random() < 0.5}
    if kind == "soup":
        return {"kind": kind, "tris": _log_int(rng, 2000, 1048576), "width": _log_int(rng, 640, 3840),
                "height": _log_int(rng, 480, 2160), "raster": raster}
    if kind == "overdraw":
        return {"kind": kind, "tris": _log_int(rng, 512, 40960), "width": _log_int(rng, 65, 640),
                "height": _log_int(rng, 65, 480), "raster": raster}
    if kind == "batch":
        return {"kind": kind, "meshes": _log_int(rng, 2, 200), "max_tris": _log_int(rng, 1000, 200000)}
    if kind == "diff":
        return {"kind": kind, "views": rng.randint(1, 16), "level": rng.randint(2, 6), "size": _log_int(rng, 48, 512),
                "texture": _log_int(rng, 16, 1024), "autograd": rng.random() < 0.5}
    if kind == "lines":
        return {"kind": kind, "lines": _log_int(rng, 300, 300000), **size}
    if kind == "points":
        return {"kind": kind, "points": _log_int(rng, 1000, 1000000), **size}
    return {"kind": kind, "tris": _log_int(rng, 100, 100000), **size, "raster": raster}


def _raster_pixels(case):
    return case["width"] * case["height"]


# Mean area of a soup triangle: 15 octaves from 0.5 px^2, uniform inside each, half culled.
_SOUP_AREA = sum(0.75 * 2.0 ** e for e in range(14)) / 15 + 9096.0 / 15


def work(case):
    """Bytes: each index, vertex and texel read once, each target pixel's buffers written
    once.  Operations: the arithmetic per vertex, triangle setup and fragment."""
    k = case["kind"]
    if k == "cube":
        px = _raster_pixels(case)
        tex = 4 * 256 * 256 * (4 / 3 if case["mip"] else 1)
        return {"bytes": 24 * 20 + 36 * 4 + tex + px * (4 if case["mip"] else 8), "flops": 24 * 60 + 12 * 150 + 0.1 * px * (400 if case["mip"] else 40)}
    if k == "mesh":
        px, vs = _raster_pixels(case), SHADERS[case["shader"]]
        verts = 10 * 4 ** _level(case["tris"]) + 2
        out = px * (16 if case["records"] else 8)
        return {"bytes": case["tris"] * 12 + verts * vs[3] + 4 * vs[2] ** 2 + out,
                "flops": verts * 60 + case["tris"] * 100 + 0.15 * px * 100}
    if k == "soup":
        px, t = _raster_pixels(case), case["tris"]
        return {"bytes": t * (12 + 72) + px * 8, "flops": t * 3 * 60 + t * 100 + 0.35 * t * _SOUP_AREA * 10}
    if k == "overdraw":
        px, t = _raster_pixels(case), case["tris"]
        return {"bytes": t * (12 + 72) + px * 4, "flops": t * 3 * 60 + t * 150 + t * px / 4 * 11 / 144 * 4}
    if k == "batch":
        n = case["meshes"]
        tris = n * (case["max_tris"] - 100) / math.log(case["max_tris"] / 100)
        px = sum((256 * (1 + i % 4)) ** 2 for i in range(n))
        return {"bytes": tris * 12 + tris * 0.75 * 32 + n * 4 * 512 ** 2 + px * 8, "flops": tris * 145 + 0.3 * px * 100}
    if k == "diff":
        v, px = case["views"], case["views"] * case["size"] ** 2
        verts, tris, tex = 10 * 4 ** case["level"] + 2, 20 * 4 ** case["level"], case["texture"] ** 2
        # image written and read back, target (or image gradient) read, parameters, gradients
        return {"bytes": px * 48 + 12 * tris + verts * 64 + tex * 32, "flops": v * (verts * 60 + tris * 100) + 0.35 * px * 500}
    if k == "lines":
        px, n = _raster_pixels(case), case["lines"]
        return {"bytes": n * 8 + n / 3 * 24 + px * 8, "flops": n / 3 * 60 + n * 40 + _line_fragments(case) * 15}
    if k == "points":
        px, n = _raster_pixels(case), case["points"]
        return {"bytes": n * 4 + n * 24 + px * 8, "flops": n * 75}
    px, t = _raster_pixels(case), case["tris"]
    return {"bytes": t * (12 + 3 * 144) + px * 8, "flops": t * 100 + t * _LIST_AREA / 2 * 30}


_LIST_AREA = 1000.0 / math.log(2000.0)


def _line_fragments(case):
    return case["lines"] * max(1.0, 2.0 * min(case["width"], case["height"]) / math.sqrt(case["lines"]))


# ---------------------------------------------------------------------------------------
# inputs

def _level(tris):
    level = 0
    while 20 * 4 ** level < tris:
        level += 1
    return level


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rotation(rng):
    q = rng.standard_normal(4)
    w, x, y, z = q / np.linalg.norm(q)
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w), 0],
                     [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w), 0],
                     [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y), 0], [0, 0, 0, 1]])


def _camera(rng, aspect, distance, far=100.0):
    """60 degree perspective, a seeded rotation, the object `distance` in front."""
    proj = np.array(scenes.perspective(aspect, 0.1, far))
    view = np.array(scenes.translate(0.0, 0.0, -distance))
    return (proj @ view @ _rotation(rng)).astype(np.float32).reshape(16)


_SPHERES = {}


def _sphere(level):
    """Unit icosphere on the GPU: positions (float64), triangles (int32)."""
    if level not in _SPHERES:
        p, f = scenes.icosphere(level)
        _SPHERES[level] = (torch.from_numpy(p).cuda(), torch.from_numpy(f.astype(np.int32)).cuda())
    return _SPHERES[level]


def _bumps(p, c):
    """Radial deformation of unit vectors by a cubic polynomial with coefficients c (6,)."""
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    r = 1.0 + c[0] * x * y + c[1] * y * z + c[2] * z * x + c[3] * x * x + c[4] * y * y * y + c[5] * z
    return p * r[:, None]


def _checker(rng, size):
    """RGBA8 checker of two seeded colours with a ramp."""
    i = np.arange(size, dtype=np.uint32)
    sq = max(1, size // int(rng.integers(8, 33)))
    a, b = rng.integers(0, 2 ** 24, 2).astype(np.uint32)
    on = ((i // sq)[:, None] + (i // sq)[None, :]) & 1
    return (np.where(on == 1, a, b) ^ (i & 15)[None, :] ^ ((i & 15) << np.uint32(8))[:, None]) | np.uint32(0xFF000000)


def _mesh_inputs(case, seed):
    """(attribute streams, indices, mvp, texture) of a mesh case."""
    rng = np.random.default_rng([11, int(seed)])
    p, f = _sphere(_level(case["tris"]))
    f = f[:case["tris"]]
    q = _bumps(p, rng.random(6) * 0.3 - 0.15)
    mvp = _camera(rng, case["width"] / case["height"], 2.2 + 1.8 * rng.random())
    if case["shader"] == "color":
        rgb = torch.rand(q.shape, generator=_generator(seed), device="cuda", dtype=torch.float64)
        streams = [(torch.cat([q, rgb], 1).float().contiguous(), 24)]
    else:
        uv = torch.stack([(p[:, 0] + 1.0) * 0.5, (p[:, 2] + 1.0) * 0.5], 1)
        streams = [(torch.cat([q, p], 1).float().contiguous(), 24), (uv.float().contiguous(), 8)]
    edge = SHADERS[case["shader"]][2]
    tex = torch.from_numpy(_checker(rng, edge).view(np.int32)).cuda() if edge else None
    return streams, f.reshape(-1).contiguous(), mvp, tex


def _edges(f):
    """Undirected edges of a triangle list, each once, in order of first use."""
    e = torch.stack([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]], 1).reshape(-1, 2)
    return e[e[:, 0] < e[:, 1]].contiguous()


def _line_inputs(case, seed):
    rng = np.random.default_rng([12, int(seed)])
    level = 0
    while 30 * 4 ** level < case["lines"]:
        level += 1
    p, f = _sphere(level)
    q = _bumps(p, rng.random(6) * 0.3 - 0.15)
    idx = _edges(f)[:case["lines"]]
    rgb = torch.rand(q.shape, generator=_generator(seed), device="cuda", dtype=torch.float64)
    # far enough for the whole object to be in the frustum, whichever side is shorter
    d = 2.9 + 0.8 * rng.random()
    aspect = case["width"] / case["height"]
    mvp = _camera(rng, aspect, d * max(1.0, 1.0 / aspect))
    return torch.cat([q, rgb], 1).float().contiguous(), idx.reshape(-1).contiguous(), mvp


def _point_inputs(case, seed):
    rng = np.random.default_rng([13, int(seed)])
    g, n = _generator(seed), case["points"]
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    v = _bumps(v / v.norm(dim=1, keepdim=True), rng.random(6) * 0.4 - 0.2)
    v = v * (0.9 + 0.2 * torch.rand((n, 1), generator=g, device="cuda", dtype=torch.float64))
    rgb = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    mvp = _camera(rng, case["width"] / case["height"], 2.6 + rng.random())
    return torch.cat([v, rgb], 1).float().contiguous(), torch.arange(n, dtype=torch.int32, device="cuda"), mvp


def _list_inputs(case, seed):
    """RasterizerVertex records: triangles of log-uniform area in [0.5, 1000] px^2, either
    winding, depths in [0, 1]; one in 64 skipped by a first index of -1."""
    g, n, w, h = _generator(seed), case["tris"], case["width"], case["height"]

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    area = 0.5 * torch.exp(rand(n) * math.log(2000.0))
    pts = rand(n, 3, 2) * 2.0 - 1.0
    a, b = pts[:, 1] - pts[:, 0], pts[:, 2] - pts[:, 0]
    a0 = (0.5 * (a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]).abs()).clamp(min=0.1)
    centre = rand(n, 1, 2) * torch.tensor([w, h], device="cuda")
    rv = torch.zeros((n, 3, 36), dtype=torch.float64, device="cuda")
    rv[:, :, 0:2] = centre + pts * torch.sqrt(area / a0)[:, None, None]
    rv[:, :, 2] = (rand(n, 1) * 0.9 + 0.1 * rand(n, 3)).clamp(0.0, 0.999)
    rv[:, :, 3] = 0.5 + 1.5 * rand(n, 3)
    rv[:, :, 20:23] = rand(n, 3, 3)
    idx = torch.arange(3 * n, dtype=torch.int32, device="cuda").view(n, 3)
    idx[rand(n) < 1.0 / 64, 0] = -1
    return rv.view(-1, 36).float().contiguous(), idx.view(-1).contiguous()


def _soup_inputs(case, seed):
    """Independent triangles: centre uniform on the screen, area uniform inside an octave of
    [0.5, 10^4] px^2 chosen uniformly, depth uniform in [0.05, 200] (vertices at 0.5 to 1.5
    times it), random winding, colour per vertex."""
    g, n, w, h = _generator(seed), case["tris"], case["width"], case["height"]

    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)

    octave = torch.randint(0, 15, (n,), generator=g, device="cuda").double()
    area = 0.5 * torch.exp2(octave) * (1.0 + rand(n))
    area = torch.where(area > 1e4, 8192.0 + (1e4 - 8192.0) * rand(n), area)
    pts = rand(n, 3, 2) * 2.0 - 1.0
    a, b = pts[:, 1] - pts[:, 0], pts[:, 2] - pts[:, 0]
    a0 = (0.5 * (a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]).abs()).clamp(min=0.05)
    size = torch.tensor([w, h], device="cuda")
    s = rand(n, 1, 2) * size + pts * torch.sqrt(area / a0)[:, None, None]
    ndc = (s - size / 2) / (size / 2)
    z = (0.05 + 199.95 * rand(n, 1)) * (0.5 + rand(n, 3))
    v = torch.empty((n, 3, 6), dtype=torch.float64, device="cuda")
    v[:, :, 0] = ndc[:, :, 0] * z * (w / h) / math.sqrt(3.0)
    v[:, :, 1] = -ndc[:, :, 1] * z / math.sqrt(3.0)
    v[:, :, 2] = -z
    v[:, :, 3:] = rand(n, 3, 3)
    mvp = np.array(scenes.perspective(w / h, 0.1, 100.0), np.float32).reshape(16)
    return v.view(-1, 6).float().contiguous(), torch.arange(3 * n, dtype=torch.int32, device="cuda"), mvp


def _batch_scenes(case, seed):
    """Deformed icospheres with triangle counts log-uniform in [100, max_tris], targets of
    256, 512, 768 and 1024 pixels a side in turn, a camera and a 512 x 512 texture each."""
    rng = np.random.default_rng([14, int(seed)])
    out = []
    for i in range(case["meshes"]):
        n = int(100 * math.exp(rng.random() * math.log(case["max_tris"] / 100)))
        p, f = scenes.icosphere(_level(n))
        p = p.astype(np.float32)
        q = _bumps(p, (rng.random(6) * 0.4 - 0.2).astype(np.float32))
        uv = np.stack([(p[:, 0] + 1) * 0.5, (p[:, 2] + 1) * 0.5], 1).astype(np.float32)
        side = 256 * (1 + i % 4)
        light = rng.random(3) - (0.5, 0.5, 0.0)
        light = light / np.linalg.norm(light)
        out.append(scenes.Scene(
            name=f"mesh{i}", vs=VS.POS_NRM_UV, ps=PS.LAMBERT_TEX, width=side, height=side, cull=CullMode.CW,
            raster=RasterMode.Block, viewport=(0, 0, side, side), scissor=(0, 0, side, side),
            attribs=[(np.concatenate([q, p], 1), 24), (uv, 8)], indices=f[:n].reshape(-1).astype(np.int32),
            mvp=_camera(rng, 1.0, 2.4 + 1.6 * rng.random()), light=np.append(light, 0.2).astype(np.float32),
            texture=_checker(rng, 512)))
    return out


def _diff_inputs(case, seed):
    """(vertex records, triangles, texture, cameras, targets) of a differentiable case."""
    rng = np.random.default_rng([15, int(seed)])
    g = _generator(seed)
    p, f = _sphere(case["level"])
    # vertex colours that vary smoothly over the object, a few seeded waves per channel
    k = torch.from_numpy(rng.random((4, 3)) * 6.0).cuda()
    rgb = 0.5 + 0.3 * torch.sin(k[0] + p @ k[1:])
    uv = torch.stack([(p[:, 0] + 1.0) * 0.5, (p[:, 1] + 1.0) * 0.5], 1)
    verts = torch.cat([p, rgb, uv], 1).float().contiguous()
    t = torch.linspace(0.0, 1.0, case["texture"], device="cuda", dtype=torch.float64)
    k = torch.from_numpy(rng.random((4, 3)) * 6.0).cuda()
    tex = 0.5 + 0.4 * torch.sin(k[:, 0] + k[:, 1] * t[:, None, None] + k[:, 2] * t[None, :, None])
    mvps = [_camera(rng, 1.0, 2.5 + rng.random()) for _ in range(case["views"])]
    n = case["size"]
    target = torch.rand((case["views"], n, n, 4), generator=g, device="cuda")
    return verts, f.reshape(-1).contiguous(), tex.float().contiguous(), mvps, target


# ---------------------------------------------------------------------------------------
# the objects a program keeps, and its frame

class _Frame:
    """One target drawn through a VertexProcessor / Rasterizer pair."""

    def __init__(self, case, ps, raster, mvp=None, texture=None, tex_wh=(0, 0), records=False, light=(0.3, 0.5, 0.81, 0.15), max_aniso=0):
        w, h = case["width"], case["height"]
        shape = scenes.Scene(name="target", vs=VS.POS_UV, ps=ps, width=w, height=h)
        self.target = DeviceTarget(shape, aux=records, clear_depth=CLEAR_DEPTH)
        self.texture, self.records, self.depth_tested = texture, records, shape.has_depth
        self.rast = Rasterizer()
        self.rast.setRasterMode(raster)
        self.rast.setScissorRect(0, 0, w, h)
        t = self.target
        self.uniforms = make_uniforms(
            np.eye(4) if mvp is None else mvp, light, 16, w, h, tex_ptr=texture.data_ptr() if texture is not None else 0,
            tex_w=tex_wh[0], tex_h=tex_wh[1], color=t.color.data_ptr(), depth=t.depth.data_ptr(),
            frag_count=t.frag_count.data_ptr() if records else 0, winner=t.winner.data_ptr() if records else 0,
            max_aniso=max_aniso)
        self.rast.setPixelShader(ps, self.uniforms)

    def geometry(self, vs, streams, indices, mode=DrawMode.Triangle, cull=CullMode.CW, graph=False, sync=True):
        w, h = self.target.depth.shape[1], self.target.depth.shape[0]
        self.mode, self.indices, self.count, self.sync = mode, indices, indices.numel(), sync
        self.vp = VertexProcessor(self.rast)
        self.vp.setViewport(0, 0, w, h)
        self.vp.setCullMode(cull)
        self.vp.setVertexShader(vs)
        for i, (buf, stride) in enumerate(streams):
            self.vp.setVertexAttribPointer(i, stride, buf)
        if graph:
            self.rast.ctx.set_graph_mode(True)
        return self

    def run(self):
        self.target.clear()
        self.rast.setUniforms(self.uniforms)  # a frame's camera
        self.vp.drawElements(self.mode, self.count, self.indices, sync=self.sync)
        return self.buffers()

    def buffers(self):
        t = self.target
        out = {"color": t.color}
        if self.depth_tested:
            out["depth"] = t.depth
        if self.records:
            out["frag_count"], out["winner"] = t.frag_count, t.winner
        return out


class _ListFrame(_Frame):
    """Screen-space records drawn with Rasterizer::drawTriangleList."""

    def run(self):
        self.target.clear()
        self.rast.setUniforms(self.uniforms)
        self.rast.drawTriangleList(self.vertices, self.list_indices)
        return self.buffers()


class _Batch:
    def __init__(self, case, seed):
        self.renderer = BatchRenderer(_batch_scenes(case, seed), graph=True, pooled=True)
        self.renderer.pool.clear_depth = CLEAR_DEPTH

    def run(self):
        self.renderer.clear()
        self.renderer.draw()
        return {"color": self.renderer.pool.color, "depth": self.renderer.pool.depth}


class _Diff:
    def __init__(self, case, seed):
        self.verts, idx, self.tex, mvps, self.target = _diff_inputs(case, seed)
        n, t = case["size"], case["texture"]
        self.renderer = DiffRenderer(idx, self.verts.shape[0], t, t, mvps, n, n)
        self.autograd = case["autograd"]

    def run(self):
        if self.autograd:
            v, t = self.verts.detach().requires_grad_(), self.tex.detach().requires_grad_()
            img = render(v, t, self.renderer)
            loss = (img - self.target).square().sum()
            loss.backward()
            return {"image": img.detach(), "grad_vertices": v.grad, "grad_texture": t.grad, "loss": loss.detach()}
        img = self.renderer.forward(self.verts, self.tex)
        gv, gt, loss = self.renderer.backward(self.verts, self.tex, target=self.target)
        return {"image": img, "grad_vertices": gv, "grad_texture": gt, "loss": loss}


def _cube(case, seed):
    rng = np.random.default_rng([16, int(seed)])
    v, idx = scenes.cube_mesh()
    mvp = _camera(rng, case["width"] / case["height"], 3.0 + (4.0 * rng.random() if case["mip"] else 0.0), far=10.0)
    if case["mip"]:
        tex = scenes.mip_chain(scenes.rgb_texture(256, 256, seed=int(seed) % 1000))
    else:
        tex = _checker(rng, 256)
    tex = torch.from_numpy(tex.view(np.int32)).cuda()
    f = _Frame(case, PS.TEX_MIP if case["mip"] else PS.TEX_NEAREST, RasterMode.Span, mvp, tex, (256, 256), max_aniso=8)
    return f.geometry(VS.POS_UV, [(torch.from_numpy(v).cuda(), 20)], torch.from_numpy(idx).cuda())


def prepare(case, seed):
    k = case["kind"]
    if k == "cube":
        return _cube(case, seed)
    if k == "mesh":
        vs, ps, edge, _ = SHADERS[case["shader"]]
        streams, idx, mvp, tex = _mesh_inputs(case, seed)
        f = _Frame(case, ps, RASTER[case["raster"]], mvp, tex, (edge, edge), case["records"])
        return f.geometry(vs, streams, idx, graph=case["graph"], sync=case["sync"])
    if k == "soup":
        v, idx, mvp = _soup_inputs(case, seed)
        return _Frame(case, PS.VCOLOR, RASTER[case["raster"]], mvp).geometry(VS.POS_RGB, [(v, 24)], idx)
    if k == "overdraw":
        v = torch.rand((3 * case["tris"], 6), generator=_generator(seed), device="cuda")
        idx = torch.arange(3 * case["tris"], dtype=torch.int32, device="cuda")
        f = _Frame(case, PS.VCOLOR_AFFINE, RASTER[case["raster"]])
        return f.geometry(VS.POS_RGB_AFFINE, [(v, 24)], idx, cull=CullMode.None_)
    if k == "batch":
        return _Batch(case, seed)
    if k == "diff":
        return _Diff(case, seed)
    if k == "lines":
        v, idx, mvp = _line_inputs(case, seed)
        return _Frame(case, PS.VCOLOR, RasterMode.Span, mvp).geometry(VS.POS_RGB, [(v, 24)], idx, mode=DrawMode.Line)
    if k == "points":
        v, idx, mvp = _point_inputs(case, seed)
        return _Frame(case, PS.VCOLOR, RasterMode.Span, mvp).geometry(VS.POS_RGB, [(v, 24)], idx, mode=DrawMode.Point)
    f = _ListFrame(case, PS.VCOLOR, RASTER[case["raster"]])
    f.vertices, f.list_indices = _list_inputs(case, seed)
    return f


def run(state):
    return state.run()


# ---------------------------------------------------------------------------------------
# the same in 64 bits

def _screen(pos, mvp, w, h):
    """Clip position and window x, y, z (depth range 0 to 1) of positions."""
    m = torch.from_numpy(np.asarray(mvp, np.float64).reshape(4, 4)).cuda()
    clip = torch.cat([pos.double(), torch.ones_like(pos[:, :1], dtype=torch.float64)], 1) @ m.T
    inv = 1.0 / clip[:, 3]
    return clip, torch.stack([w / 2 + w / 2 * clip[:, 0] * inv, h / 2 - h / 2 * clip[:, 1] * inv, 0.5 + 0.5 * clip[:, 2] * inv], 1)


def _cover(tri, mode, w, h):
    """Pixel centres inside screen triangles `tri` (n, 3, 3) of positive orientation: yields
    (triangle, pixel, z) in pieces.  In Block mode an 8 x 8 block whose four corners lie in
    no triangle and each satisfy an odd number of edges is skipped (Rasterizer.h:263-304)."""
    x, y, z = tri[..., 0], tri[..., 1], tri[..., 2]
    nx, ny = x.roll(-1, 1), y.roll(-1, 1)  # edge k: vertex k to k + 1
    ea, eb = y - ny, nx - x
    ec = -0.5 * (ea * (x + nx) + eb * (y + ny))
    area = ec.sum(1)
    # edge k opposes vertex k + 2
    zs = z.roll(-2, 1) / area[:, None]
    za, zb, zc = (ea * zs).sum(1), (eb * zs).sum(1), (ec * zs).sum(1)
    lo = torch.stack([x.amin(1), y.amin(1)], 1).sub(0.5).ceil().clamp(min=0).long()
    hi = torch.stack([x.amax(1).clamp(max=w), y.amax(1).clamp(max=h)], 1).sub(0.5).floor().long()
    ext = (hi - lo + 1).clamp(min=0)
    count = ext[:, 0] * ext[:, 1]
    count[~(area > 0)] = 0
    if mode == "adaptive":
        ratio = (x.amax(1) - x.amin(1)) / (y.amax(1) - y.amin(1))
        block = (ratio > 0.4) & (ratio < 1.6)
    else:
        block = torch.full_like(area, mode == "block", dtype=torch.bool)
    ends = count.cumsum(0)
    total, n = int(ends[-1]) if len(ends) else 0, 0
    first = 0
    while n < total:
        last = int(torch.searchsorted(ends, torch.tensor(n + (1 << 24), device="cuda")))
        last = max(first + 1, min(last, len(ends)))
        t = torch.repeat_interleave(torch.arange(first, last, device="cuda"), count[first:last])
        j = torch.arange(len(t), device="cuda") + n - (ends[t] - count[t])
        px, py = lo[t, 0] + j % ext[t, 0], lo[t, 1] + torch.div(j, ext[t, 0], rounding_mode="floor")

        def inside(cx, cy):
            return ea[t] * cx[:, None] + eb[t] * cy[:, None] + ec[t] > 0

        hit = inside(px + 0.5, py + 0.5).all(1)
        hit &= (px < w) & (py < h)
        t, px, py = t[hit], px[hit], py[hit]
        if bool(block.any()):
            bx, by = (px & ~7) + 0.5, (py & ~7) + 0.5
            corners = torch.stack([inside(bx + dx, by + dy).sum(1) for dx in (0.0, 7.0) for dy in (0.0, 7.0)], 1)
            keep = ~(block[t] & (corners % 2 == 1).all(1) & (corners < 3).all(1))
            t, px, py = t[keep], px[keep], py[keep]
        if len(t):
            yield t, py * w + px, za[t] * (px + 0.5) + zb[t] * (py + 0.5) + zc[t]
        n, first = int(ends[last - 1]), last


def _front(screen, faces, w, h):
    """Screen triangles of the faces that CullMode CW keeps, turned to positive orientation,
    and their face numbers."""
    tri = screen[faces.long()]
    a, b = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    keep = torch.nonzero(a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0] < 0).reshape(-1)
    return tri[keep][:, [2, 1, 0]], keep


def _depths(tri, mode, w, h):
    depth = torch.full((w * h,), CLEAR_DEPTH, dtype=torch.float64, device="cuda")
    for _, pix, z in _cover(tri, mode, w, h):
        depth.scatter_reduce_(0, pix, z, "amin")
    return depth.view(h, w)


def _exact_steps(case, a, b, steps):
    """Depths of stepped fragments: `steps` from each a towards b (n, 3), one per step."""
    w, h = case["width"], case["height"]
    depth = torch.full((w * h,), CLEAR_DEPTH, dtype=torch.float64, device="cuda")
    i = torch.repeat_interleave(torch.arange(len(steps), device="cuda"), steps)
    j = torch.arange(len(i), device="cuda") - (steps.cumsum(0) - steps)[i]
    p = a[i] + (b - a)[i] / steps[i].double()[:, None] * j[:, None]
    ok = (p[:, 0] >= 0) & (p[:, 0] < w) & (p[:, 1] >= 0) & (p[:, 1] < h)
    p = p[ok]
    depth.scatter_reduce_(0, p[:, 1].long() * w + p[:, 0].long(), p[:, 2].contiguous(), "amin")
    return depth.view(h, w)


def _exact_diff(case, seed):
    verts, idx, tex, mvps, target = _diff_inputs(case, seed)
    n, t = case["size"], case["texture"]
    faces = idx.view(-1, 3).long()
    v = verts.double().requires_grad_()
    tx = tex.double().requires_grad_()
    images = []
    for mvp in mvps:
        m = torch.from_numpy(np.asarray(mvp, np.float64).reshape(4, 4)).cuda()
        with torch.no_grad():
            _, s = _screen(v.detach()[:, :3], mvp, n, n)
            tri, face = _front(s, faces, n, n)
            depth = torch.full((n * n,), float("inf"), dtype=torch.float64, device="cuda")
            pieces = list(_cover(tri, "block", n, n))
            for _, pix, z in pieces:
                depth.scatter_reduce_(0, pix, z, "amin")
            winner = torch.full((n * n,), len(faces), dtype=torch.long, device="cuda")
            for k, pix, z in pieces:
                best = z == depth[pix]
                winner.scatter_reduce_(0, pix[best], face[k[best]], "amin")
            pix = torch.nonzero(winner < len(faces)).reshape(-1)
        vi = faces[winner[pix]]  # (p, 3)
        clip = torch.cat([v[:, :3], torch.ones_like(v[:, :1])], 1) @ m.T
        q = clip[vi]
        cx, cy = (pix % n + 0.5)[:, None], (torch.div(pix, n, rounding_mode="floor") + 0.5)[:, None]
        dx = n / 2 * q[..., 0] + (n / 2 - cx) * q[..., 3]
        dy = -n / 2 * q[..., 1] + (n / 2 - cy) * q[..., 3]
        e = dx.roll(-1, 1) * dy.roll(-2, 1) - dx.roll(-2, 1) * dy.roll(-1, 1)
        bary = e / e.sum(1, keepdim=True)
        a = (bary[..., None] * v[vi][..., 3:]).sum(1)  # r, g, b, u, v
        uv = a[:, 3:].clamp(0.0, 1.0) * (t - 1)
        i0 = uv.detach().floor().long().clamp(max=t - 1)
        i1 = (i0 + 1).clamp(max=t - 1)
        fr = uv - i0
        fx, fy = fr[:, :1], fr[:, 1:]
        c = (tx[i0[:, 1], i0[:, 0]] * (1 - fx) + tx[i0[:, 1], i1[:, 0]] * fx) * (1 - fy) + \
            (tx[i1[:, 1], i0[:, 0]] * (1 - fx) + tx[i1[:, 1], i1[:, 0]] * fx) * fy
        col = torch.cat([a[:, :3] * c[:, :3], c[:, 3:]], 1)
        images.append(torch.zeros((n * n, 4), dtype=torch.float64, device="cuda").index_put((pix,), col).view(n, n, 4))
    img = torch.stack(images)
    loss = (img - target.double()).square().sum()
    loss.backward()
    return {"image": img.detach(), "grad_vertices": v.grad, "grad_texture": tx.grad, "loss": loss.detach()}


def exact(case, seed):
    k = case["kind"]
    if k == "diff":
        return _exact_diff(case, seed)
    if k == "batch":
        depth = []
        for sc in _batch_scenes(case, seed):
            pos = torch.from_numpy(sc.attribs[0][0][:, :3]).cuda()
            _, s = _screen(pos, sc.mvp, sc.width, sc.height)
            tri, _ = _front(s, torch.from_numpy(sc.indices).cuda().view(-1, 3), sc.width, sc.height)
            depth.append(_depths(tri, "block", sc.width, sc.height).reshape(-1))
        return {"color": None, "depth": torch.cat(depth)}
    if k in ("soup", "overdraw") or (k == "cube" and case["mip"]):
        return None
    w, h = case["width"], case["height"]
    if k == "cube":
        rng = np.random.default_rng([16, int(seed)])
        v, idx = scenes.cube_mesh()
        mvp = _camera(rng, w / h, 3.0, far=10.0)
        _, s = _screen(torch.from_numpy(v[:, :3]).cuda(), mvp, w, h)
        depth = _depths(_front(s, torch.from_numpy(idx).cuda().view(-1, 3), w, h)[0], "span", w, h)
    elif k == "mesh":
        streams, idx, mvp, _ = _mesh_inputs(case, seed)
        _, s = _screen(streams[0][0][:, :3], mvp, w, h)
        depth = _depths(_front(s, idx.view(-1, 3), w, h)[0], case["raster"], w, h)
    elif k == "list":
        rv, idx = _list_inputs(case, seed)
        idx = idx.view(-1, 3)
        depth = _depths(rv.double()[:, :3][idx[idx[:, 0] >= 0].long()], case["raster"], w, h)
    elif k == "lines":
        v, idx, mvp = _line_inputs(case, seed)
        _, s = _screen(v[:, :3], mvp, w, h)
        a, b = s[idx.view(-1, 2).long()].unbind(1)
        d = (b[:, :2].long() - a[:, :2].long()).abs().amax(1)
        depth = _exact_steps(case, a[d > 0], b[d > 0], d[d > 0])
    else:
        v, idx, mvp = _point_inputs(case, seed)
        clip, s = _screen(v[:, :3], mvp, w, h)
        s = s[(clip[:, :3].abs() <= clip[:, 3:]).all(1)]
        depth = _exact_steps(case, s, s, torch.ones(len(s), dtype=torch.long, device="cuda"))
    out = {"color": None, "depth": depth}
    if case.get("records"):
        out["frag_count"] = out["winner"] = None
    return out
