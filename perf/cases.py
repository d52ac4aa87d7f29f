"""The calls a program makes to the strand rasteriser, as cases that can be timed.

Every case is one pass through the public entry points of
`bevy_strand_rasterizer_b200`: frame tables (`frame_begin`), then the frame's
nodes one by one, the fused frame, the host-buffer frame, the deep-shadow maps
alone, a multi-view frame, or a burst of requests to the request server.
Scenes are seeded hair: strands over the upper half of a 0.1 m head, drooping,
jittered, optionally curled, made on the GPU from the seed alone.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from bevy_strand_rasterizer_b200 import abi, batched, plugin as fiber
from bevy_strand_rasterizer_b200.scene import CameraSpec, LightSpec
from bevy_strand_rasterizer_b200.server import FiberServer

# What a case says when it does not say otherwise: the plugin's defaults on a
# 1080p camera with one light.
DEFAULTS = dict(mode="fused", strands=10_000, points=16, curly=False, instances=1, width=1920, height=1080,
                distance=0.6, lights=1, dom=1024, slices=8, refs=4, backend=0, pool=0, opaque=0, history=True,
                cull=True, scene32=False, radius=2.0, views=0, requests=0)


def case(name=None, **kw):
    unknown = set(kw) - set(DEFAULTS)
    assert not unknown, unknown
    c = dict(DEFAULTS, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # A thumbnail or a unit-test scene: launches and host work are all it costs.
        case("tiny_frame", strands=300, points=8, width=160, height=120, dom=128, slices=4),
        # A preview without lights of a few grooms, each with its own transform and material.
        case("preview_6_grooms", mode="nodes", strands=1_500, points=24, instances=6, width=510, height=382,
             lights=0, cull=False),
        # The small configuration: a character at mid distance, 720p.
        case("small_frame", strands=10_000, points=16, width=1280, height=720, dom=1024, slices=4),
        # The medium configuration: a hero character at 1080p, the frame an engine draws at 60 Hz or above.
        case("medium_frame", strands=100_000, points=32, dom=2048),
        # The same, for a host that keeps its images in host memory (pinned upload and download each frame).
        case("medium_host", mode="host", strands=100_000, points=32, dom=2048),
        # Node by node behind an opaque scene (4 samples), curly, odd sizes, two lights with the default 12 slices,
        # the scene in 32-bit floats.
        case("nodes_behind_opaque", mode="nodes", strands=40_000, points=25, curly=True, width=1366, height=766,
             lights=2, dom=1224, slices=12, refs=8, opaque=4, scene32=True),
        # The page-owned binning backend with deep-opacity pages resident on demand.
        case("page_csr_sparse", strands=50_000, points=24, width=1600, height=900, dom=2048, backend=1, pool=64),
        # Only the deep-shadow maps of two lights, for an engine that shades the rest of its scene with them.
        case("shadow_maps", mode="shadows", strands=80_000, points=20, width=1024, height=768, lights=2, dom=2048,
             slices=12, refs=8),
        # A close-up with wide strands: few segments, many pixels each.
        case("close_up", strands=30_000, points=32, distance=0.4, dom=1024, refs=16, radius=5.0),
        # Thumbnails and turntables: many independent views in one frame.
        case("views_16", mode="views", views=16, strands=200_000, dom=2048, history=False),
        # Requests of different scenes and sizes, submitted together to the request server.
        case("served_burst", mode="served", requests=12, strands=50_000, points=32, width=1280, height=720,
             dom=1024, history=False, refs=8),
        # The large configuration: half a million curly strands at 4K, two 4096^2 lights.
        case("large_frame", strands=500_000, points=32, curly=True, width=3840, height=2160, lights=2, dom=4096,
             refs=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    mode = rng.choice(["fused", "fused", "fused", "nodes", "host", "shadows", "views"])
    if mode == "views":
        return case(mode=mode, views=rng.randint(3, 24), strands=_log(rng, 3_000, 150_000),
                    dom=rng.choice([512, 1024, 2048]), history=False)
    curly = rng.random() < 0.4
    distance = rng.uniform(0.4, 1.0)
    lights = rng.choice([1, 1, 2]) if mode == "shadows" else rng.choice([0, 1, 1, 1, 2])
    width = _log(rng, 128, 2560)
    return case(mode=mode, strands=_log(rng, 300, 150_000), points=rng.randint(6, 40), curly=curly,
                instances=rng.choice([1, 1, 1, 2, 5]), width=width, height=max(64, int(width * rng.uniform(0.5, 1.0))),
                distance=distance, lights=lights, dom=8 * _log(rng, 16, 320), slices=rng.choice([4, 8, 12]),
                refs=16 if curly or distance < 0.5 else 8, backend=rng.choice([0, 0, 0, 1]),
                pool=rng.choice([0, 0, 0, 256]) if lights else 0, opaque=rng.choice([0, 0, 1, 4]) if mode == "nodes" else 0,
                history=rng.random() < 0.7, cull=rng.random() < 0.7, scene32=mode == "nodes" and rng.random() < 0.3,
                radius=rng.choice([2.0, 2.0, 4.0]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def hair(n: int, points: int, curly: bool, g: torch.Generator) -> fiber.PackedStrandBuffers:
    """Roots uniform by area on the upper half of a 0.1 m sphere, lengths
    U[0.15, 0.30] m along the normal with a 0.5 rad droop, 1 mm jitter; curls
    of radius U[2, 6] mm and pitch U[8, 20] mm."""
    dev = g.device

    def uniform(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device=dev)

    y, phi = uniform(0.0, 1.0), uniform(0.0, 2.0 * math.pi)
    r = (1.0 - y * y).clamp_min(0.0).sqrt()
    normal = torch.stack([r * phi.cos(), y, r * phi.sin()], 1)
    down = torch.tensor([0.0, -1.0, 0.0], device=dev)
    perp = down - (normal @ down)[:, None] * normal
    length = perp.norm(dim=1, keepdim=True)
    perp = torch.where(length > 1e-6, perp / length.clamp_min(1e-12), torch.tensor([1.0, 0.0, 0.0], device=dev))
    step = uniform(0.15, 0.30) / max(points - 1, 1)
    pos = torch.empty(n, points, 3, device=dev)
    p = 0.1 * normal
    pos[:, 0] = p
    for k in range(points - 1):
        a = 0.5 * (k + 0.5) / max(points - 1, 1)
        p = p + (math.cos(a) * normal + math.sin(a) * perp) * step[:, None]
        pos[:, k + 1] = p
    if curly:
        radius, pitch, phase = uniform(0.002, 0.006), uniform(0.008, 0.020), uniform(0.0, 2.0 * math.pi)
        side = torch.cross(normal, perp, dim=1)
        arc = torch.arange(points, device=dev)[None, :] * step[:, None]
        ph = 2.0 * math.pi * arc / pitch[:, None] + phase[:, None]
        ramp = (radius[:, None] * (arc / pitch[:, None]).clamp_max(1.0))[:, :, None]
        pos += ramp * (ph.cos()[:, :, None] * perp[:, None] + ph.sin()[:, :, None] * side[:, None])
    pos[:, 1:] += 0.001 * torch.randn(n, points - 1, 3, generator=g, device=dev)
    counts = np.full(n, points, np.uint32)
    offsets = (np.arange(n, dtype=np.uint64) * points).astype(np.uint32)
    return fiber.pack_indexed_strands(pos.reshape(-1, 3).cpu().numpy(), counts, offsets,
                                      np.arange(n * points, dtype=np.uint32))


def _on_sphere(rng, distance: float) -> tuple:
    """A point around the head, a little above or below it."""
    a, h = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(-0.1, 0.4)
    r = math.sqrt(1.0 - h * h)
    return (distance * r * math.sin(a), distance * h, distance * r * math.cos(a))


def _light(rng, dom: int) -> LightSpec:
    a = rng.uniform(0.0, 2.0 * math.pi)
    # 100 lux puts the shaded colours of the default material inside (0, 1).
    return LightSpec((math.cos(a), rng.uniform(0.6, 1.2), math.sin(a)), illuminance=100.0, size=dom)


def _material(k: int, radius: float) -> fiber.StrandMaterial:
    if k == 0:
        return fiber.StrandMaterial(max_radius_pixels=radius)
    return fiber.StrandMaterial(absorption_color=(0.3 + 0.1 * (k % 5), 0.6, 0.9 - 0.1 * (k % 4), 0.4 + 0.05 * (k % 3)),
                                beta=0.3 + 0.1 * (k % 4), alpha=0.2 + 0.05 * (k % 3), max_radius_pixels=radius)


def _placed(k: int) -> np.ndarray | None:
    """Instance k's column-major world_from_local: turned about y and moved aside."""
    if k == 0:
        return None
    m = np.eye(4, dtype=np.float32)
    a = 0.7 * k
    m[0, 0], m[0, 2], m[2, 0], m[2, 2] = math.cos(a), math.sin(a), -math.sin(a), math.cos(a)
    m[:3, 3] = (0.05 * math.cos(2.0 * k), 0.02 * (k % 3), 0.05 * math.sin(2.0 * k))
    return np.ascontiguousarray(m.T).reshape(16)


class _Device:
    """An array view of a device image that a plugin's context owns; the view keeps the plugin."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 2,
                                         "strides": None}


def _tensor(p: fiber.StrandRasterizerPlugin, what: int, shape, typestr: str) -> torch.Tensor:
    return torch.as_tensor(_Device(p, p.output_image(what).ptr, shape, typestr), device="cuda")


_STREAM = []


def _stream():
    """The program's render stream (a frame graph needs one of its own)."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


class _State:
    pass


def _frame_state(c, seed: int) -> _State:
    rng = np.random.default_rng(seed)
    g = torch.Generator("cuda").manual_seed(seed)
    s = _State()
    s.case = c
    s.plugin = fiber.StrandRasterizerPlugin(
        cull=fiber.StochasticCullSettings(enabled=c["cull"]), backend=fiber.FineBinningBackend(c["backend"]),
        dom_slices=c["slices"], history=c["history"], ref_capacity_factor=c["refs"], dom_page_pool=c["pool"])
    for k in range(c["instances"]):
        s.plugin.add_geometry(hair(max(1, c["strands"] // c["instances"]), c["points"], c["curly"], g),
                              _material(k, c["radius"]), _placed(k))
    w, h, d = c["width"], c["height"], c["dom"]
    s.config = fiber.FroxelConfig(w, h, 8, 8, 64)
    s.camera = CameraSpec(eye=_on_sphere(rng, c["distance"]), width=w, height=h)
    s.lights = [(fiber.FroxelConfig(d, d, 8, 8, 64), _light(rng, d)) for _ in range(c["lights"])]
    s.plugin.frame_begin(s.config, s.camera, s.lights, _stream())  # sizes the context's buffers
    s.scene_depth = s.opaque = None
    if c["mode"] == "host":
        s.scene = torch.rand(h, w, 4, generator=torch.Generator().manual_seed(seed)).half()
        s.scene[..., 3] = 1.0
        s.scene, s.out = s.scene.pin_memory(), torch.empty(h, w, 4, dtype=torch.float16).pin_memory()
        return s
    if c["mode"] == "shadows":
        n, k = c["lights"], c["slices"]
        s.results = {"map": _tensor(s.plugin, abi.DUMP_SHADOW_MAP, (n, d, d), "<f4")}
        if not c["pool"]:
            s.results["depth"] = _tensor(s.plugin, abi.DUMP_DOM_DEPTH, (n, d, d), "<f4")
            s.results["opacity"] = _tensor(s.plugin, abi.DUMP_DOM_OPACITY, (n, k, d, d), "<f4")
        return s
    kind, fmt = (torch.float32, abi.FMT_RGBA32F) if c["scene32"] else (torch.float16, abi.FMT_RGBA16F)
    s.scene = torch.rand(h, w, 4, generator=g, device="cuda").to(kind)
    s.scene[..., 3] = 1.0
    s.out = torch.zeros_like(s.scene)
    s.scene_image, s.out_image = fiber.image_from_tensor(s.scene, fmt), fiber.image_from_tensor(s.out, fmt)
    if c["opaque"]:
        # A wall through the head over part of the screen, a ramp below it.
        level = 0.1 / c["distance"]
        depth = torch.zeros(h, w, c["opaque"], device="cuda")
        depth[:, : int(0.55 * w)] = level
        depth[int(0.75 * h):] = torch.linspace(0.0, 2.0 * level, w, device="cuda")[None, :, None]
        s.opaque = depth.contiguous()
        s.opaque_image = fiber.image_from_tensor(s.opaque, abi.FMT_R32F)
    s.results = {"out": s.out,
                 "color": _tensor(s.plugin, abi.DUMP_COLOR, (h, w, 4), "<f2"),
                 "depth": _tensor(s.plugin, abi.DUMP_DEPTH, (h, w), "<f4")}
    torch.cuda.current_stream().synchronize()  # the scene image is drawn before the render stream reads it
    return s


_SHAPES = [(256, 256), (1280, 720), (512, 512), (1920, 1080), (640, 360), (330, 514)]


def _views_state(c, seed: int) -> _State:
    rng = np.random.default_rng(seed)
    g = torch.Generator("cuda").manual_seed(seed)
    s = _State()
    s.case = c
    specs, packed = [], []
    for strands, points, (w, h), dom in _view_sizes(c):
        specs.append(batched.ViewSpec(strands, points, 0, CameraSpec(eye=_on_sphere(rng, rng.uniform(0.5, 1.0)), width=w, height=h),
                                      fiber.FroxelConfig(w, h, 8, 8, 64), _light(rng, dom),
                                      fiber.FroxelConfig(dom, dom, 8, 8, 64)))
        packed.append(hair(strands, points, False, g))
    s.frame = batched.MultiViewFrame(specs, packed, dom_slices=c["slices"], ref_capacity_factor=c["refs"])
    s.frame.plugin.frame_begin_views(s.frame.views, _stream())  # sizes the context's buffers
    n = sum(x.camera_cfg.screen_width * x.camera_cfg.screen_height for x in specs)
    s.results = {"color": _tensor(s.frame.plugin, abi.DUMP_COLOR, (n, 4), "<f2"),
                 "depth": _tensor(s.frame.plugin, abi.DUMP_DEPTH, (n,), "<f4")}
    return s


def _view_sizes(c):
    """(strands, points, resolution, map) of each view: strands from 1,000 to
    the case's, evenly over their logarithm."""
    n = c["views"]
    for k in range(n):
        t = ((k * 7) % n) / max(1, n - 1)
        yield (int(1000 * (c["strands"] / 1000) ** t), (16, 32)[k % 2], _SHAPES[k % len(_SHAPES)],
               c["dom"] >> (k % 3))


def _request_sizes(c):
    """(scene, resolution, map) of each request."""
    for k in range(c["requests"]):
        w, h = [(256, 256), (512, 512), (c["width"], c["height"]), (250, 170)][k % 4]
        yield k % 3, (w, h), c["dom"] >> (k % 2)


def _served_state(c, seed: int) -> _State:
    rng = np.random.default_rng(seed)
    g = torch.Generator("cuda").manual_seed(seed)
    s = _State()
    s.case = c
    st = abi.default_settings()
    st.history_enabled = 0
    st.dom_slices = c["slices"]
    st.ref_capacity_factor = c["refs"]
    s.server = FiberServer(slots=3, max_width=c["width"], max_height=c["height"], max_dom=c["dom"], settings=st)
    packed = [hair(max(1, c["strands"] // d), c["points"], k == 1, g) for k, d in enumerate((10, 3, 1))]
    ids = [s.server.add_scene(p) for p in packed]
    s.server.start()
    s.requests, s.outs = [], []
    for k, (w, h), dom in _request_sizes(c):
        spec = CameraSpec(eye=_on_sphere(rng, rng.uniform(0.5, 1.0)), width=w, height=h)
        cam = abi.Camera()
        cam.clip_from_world[:] = [float(x) for x in spec.clip_from_world()]
        cam.world_position[:] = [float(x) for x in spec.eye]
        light = _light(rng, dom)
        lights = (abi.Light * 1)()
        lights[0].clip_from_world[:] = [float(x) for x in light.clip_from_world(packed[k].aabb_min, packed[k].aabb_max)]
        lights[0].direction_to_light[:] = [float(x) for x in light.direction()]
        lights[0].color[:] = [float(x) for x in light.color4()]
        scene = np.full((h, w, 4), 0.1, np.float16)
        scene[..., 3] = 1.0
        s.outs.append(np.zeros_like(scene))
        s.requests.append((ids[k], fiber.FroxelConfig(w, h, 8, 8, 64), cam, [fiber.FroxelConfig(dom, dom, 8, 8, 64)],
                           lights, s.outs[-1], scene))
    return s


def prepare(case, seed):
    c = dict(DEFAULTS, **case)
    if c["mode"] == "views":
        return _views_state(c, seed)
    if c["mode"] == "served":
        return _served_state(c, seed)
    return _frame_state(c, seed)


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    c = state.case
    if c["mode"] == "served":
        tickets = [state.server.submit(*r) for r in state.requests]
        for t in tickets:
            state.server.wait(t)
        return state.outs
    stream = _stream()
    if c["mode"] == "views":
        state.frame.launch(stream)
        return state.results
    p = state.plugin
    p.frame_begin(state.config, state.camera, state.lights, stream)
    if c["mode"] == "host":
        abi.check(p.lib.fiber_render_host(p.ctx, C.c_void_p(state.scene.data_ptr()), None,
                                          C.c_void_p(state.out.data_ptr()), C.c_void_p(stream.cuda_stream)),
                  "fiber_render_host")
        stream.synchronize()  # the image is in host memory
        return state.out
    if c["mode"] == "shadows":
        p.work_preparation_pass(stream)
        p.strand_shadow_rasterizer_pass(stream)
    elif c["mode"] == "nodes":
        p.render_nodes(state.scene_image, None, state.out_image, stream, opaque_samples=c["opaque"],
                       opaque_depth=state.opaque_image if c["opaque"] else None)
    else:
        p.frame_fused(state.scene_image, None, state.out_image, stream)
    return state.results


def exact(case, seed):
    """None: a frame's values rest on its discrete decisions (which 8x8 tile,
    depth slice and fine cell a segment enters, from 16-bit projected ends; the
    order by 17-bit depth keys; groups of four per cell; the 0.98 early out),
    which are defined in binary32 and fixed point, so there is no 64-bit value
    of the same image to compare with."""
    return None


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _frame_work(strands, points, width, height, lights, dom, slices, image_bytes):
    segments = strands * (points - 1)
    # Vertex, index and strand record read once; colour and depth written; the
    # scene read and the result written; the maps' depth and opacity written.
    nbytes = strands * (20 * points + 16) + width * height * (12 + image_bytes) + lights * 4 * (slices + 1) * dom * dom
    # Projection, clip and cell walk per segment and frustum; the quadrature of
    # the scattering lobes per camera segment and light.
    flops = segments * (1 + lights) * 150 + segments * max(lights, 1) * 800
    return nbytes, flops


def work(case):
    c = dict(DEFAULTS, **case)
    if c["mode"] == "views":
        parts = [_frame_work(n, p, w, h, 1, dom, c["slices"], 0) for n, p, (w, h), dom in _view_sizes(c)]
    elif c["mode"] == "served":
        parts = [_frame_work(c["strands"] // (10, 3, 1)[k], c["points"], w, h, 1, dom, c["slices"], 16)
                 for k, (w, h), dom in _request_sizes(c)]
    else:
        image = 0 if c["mode"] == "shadows" else 32 if c["scene32"] else 16
        parts = [_frame_work(c["strands"], c["points"], c["width"], c["height"], c["lights"], c["dom"], c["slices"], image)]
    return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(f for _, f in parts))}
