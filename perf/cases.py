"""The work that users of this renderer have it do, for measuring it.

Each case is one pass through the public entry points (`Graphics`, `Upsampler`,
`rz_bc7_decode`): a frame of a kind of scene, a batch of views, a frame read
back to the host, a reconstruction or a training step of the learned x2 path, or
the decoding of a compressed texture. Sizes are those of this repository's
tests, benchmark and configurations, or generic ones. The inputs are made from a
seed: geometry from `rosy_gb300.scene`, textures, images and block data here.

`exact` gives the training step's loss, gradients and parameters in 64 bits. The
other outputs have no 64-bit counterpart: colours, ids, decoded texels and
reconstructed images are whole numbers, and a depth is that of the triangle that
the 1/256-pixel grid of snapped fp32 vertices shows at a sample, so a 64-bit
transform shows other triangles there.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

from rosy_gb300 import _abi, _lib, bc7
from rosy_gb300 import scene as sc
from rosy_gb300.graphics import Graphics
from rosy_gb300.upsampler import LAYERS, OFFSETS, PARAM_COUNT, Upsampler, init_params

OVERFLOW = 14  # rz_result: the raster's work queue grows and the frame is rendered again


def listed():
    return [
        # the smallest call: the preview-sized frame of the smoke test; launches and latency count
        {"name": "frame_tiny", "kind": "soup", "triangles": 256, "width": 96, "height": 64, "shadow": 128,
         "texture": 64, "samples": 1},
        # the first configuration: a soup of overlapping triangles (deep overdraw), 5-tap shadows
        {"name": "frame_soup", "kind": "soup", "triangles": 4096, "width": 640, "height": 360, "shadow": 1024,
         "texture": 256, "samples": 1},
        # the benchmark's frame: many tessellated meshes, textured, shadowed, 1080p
        {"name": "frame_scene", "kind": "scene", "meshes": 64, "triangles": 4096, "materials": 8, "texture": 1024,
         "width": 1920, "height": 1080, "shadow": 4096, "cascades": 1, "samples": 1},
        # the same scene as the engine renders it by default, with 4x multisampling
        {"name": "frame_scene_msaa4", "kind": "scene", "meshes": 64, "triangles": 4096, "materials": 8, "texture": 1024,
         "width": 1920, "height": 1080, "shadow": 4096, "cascades": 1, "samples": 4},
        # a quarter of every mesh alpha-blended (glass, foliage) and the editor's debug lines on top; ragged extent
        {"name": "frame_blended", "kind": "blended", "meshes": 48, "triangles": 1024, "materials": 8, "texture": 512,
         "width": 1279, "height": 717, "shadow": 2048, "fraction": 0.25, "mask": False, "lines": 24, "samples": 1},
        # the largest frame: the stress workload's million triangles and four shadow cascades in one 4K view
        {"name": "frame_4k_cascades", "kind": "scene", "meshes": 256, "triangles": 4096, "materials": 8, "texture": 1024,
         "width": 3840, "height": 2160, "shadow": 4096, "cascades": 4, "samples": 1},
        # many views of uneven size over several scenes in one frame (thumbnails, probes, dataset rendering)
        {"name": "views_batch", "kind": "views", "views": 32, "scenes": 4, "max_tris": 100000, "max_size": 1024,
         "max_shadow": 2048},
        # a frame exported to the host: rendered, copied to pinned memory, waited for
        {"name": "frame_to_host", "kind": "host", "meshes": 32, "triangles": 2048, "materials": 4, "texture": 512,
         "width": 1280, "height": 720, "shadow": 2048, "samples": 1},
        # the learned path: half-resolution frame with its G-buffer, then the x2 network, 1080p out
        {"name": "learned_frame", "kind": "learned", "triangles": 4096, "width": 960, "height": 540, "shadow": 1024,
         "texture": 256},
        # the network alone on a G-buffer of odd extent, without sub-pixel sources (as multisampled frames give it)
        {"name": "upsample", "kind": "upsample", "width": 957, "height": 539, "sources": False},
        # its training step: two frames accumulated, the gradients read, an Adam update
        {"name": "upsample_train", "kind": "train", "width": 960, "height": 540, "batch": 2, "sources": True},
        # a texture of the engine's assets decoded on the device (loading a level decodes hundreds)
        {"name": "bc7_decode", "kind": "bc7", "width": 4096, "height": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["soup", "scene", "scene", "blended", "views", "host", "learned", "upsample", "train", "bc7"])
    w, h = _log(rng, 96, 2560), _log(rng, 64, 1440)
    if kind == "soup":
        return {"kind": kind, "triangles": _log(rng, 256, 4096), "width": w, "height": h, "shadow": _log(rng, 128, 2048),
                "texture": 2 ** rng.randint(5, 9), "samples": rng.choice([1, 1, 4])}
    if kind in ("scene", "host"):
        c = {"kind": kind, "meshes": _log(rng, 1, 128), "triangles": 128 * rng.randint(1, 32), "materials": rng.randint(1, 8),
             "texture": 2 ** rng.randint(6, 10), "width": w, "height": h, "shadow": _log(rng, 512, 4096),
             "samples": rng.choice([1, 1, 4])}
        return dict(c, cascades=rng.choice([1, 1, 2, 4])) if kind == "scene" else c
    if kind == "blended":
        return {"kind": kind, "meshes": _log(rng, 1, 48), "triangles": 128 * rng.randint(1, 12), "materials": rng.randint(1, 8),
                "texture": 2 ** rng.randint(6, 9), "width": min(w, 1279), "height": min(h, 719), "shadow": _log(rng, 512, 2048),
                "fraction": rng.choice([0.1, 0.25, 0.5]), "mask": rng.random() < 0.5, "lines": rng.choice([0, 0, 8, 24]),
                "samples": rng.choice([1, 1, 4])}
    if kind == "views":
        return {"kind": kind, "views": rng.randint(2, 32), "scenes": rng.randint(1, 4), "max_tris": _log(rng, 2000, 100000),
                "max_size": _log(rng, 128, 1024), "max_shadow": _log(rng, 512, 2048)}
    if kind == "learned":
        return {"kind": kind, "triangles": _log(rng, 256, 4096), "width": min(w, 960), "height": min(h, 540), "shadow": 1024,
                "texture": 256}
    if kind == "bc7":
        return {"kind": kind, "width": _log(rng, 4, 8192), "height": _log(rng, 4, 8192)}
    c = {"kind": kind, "width": _log(rng, 64, 1440), "height": _log(rng, 36, 810), "sources": rng.random() < 0.5}
    return dict(c, batch=rng.randint(1, 3)) if kind == "train" else c


# --- frames -----------------------------------------------------------------------------


class Context:
    """A renderer context, closed when neither the program nor a tensor of its buffers holds it any more."""

    def __init__(self):
        self.g = Graphics()

    def __del__(self):
        self.g.deinit()


class View:
    """A device buffer of a context, which it keeps alive, for torch to see as a tensor."""

    def __init__(self, context, ptr, shape, typestr):
        self.context = context
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


class Renderer:
    """What a program that renders keeps: its context, its path of scene constants and its object transforms."""

    def __init__(self):
        self.context = Context()
        self.g, self.cams, self.objects, self.at, self.tensors = self.context.g, [], None, 0, {}

    def tensor(self, ptr, shape, typestr):
        key = (int(ptr), shape, typestr)
        if key not in self.tensors:
            self.tensors[key] = torch.as_tensor(View(self.context, *key), device="cuda")
        return self.tensors[key]

    def next_frame(self):
        """The next camera of the path, all transforms (the engine uploads its mobs each frame), a frame."""
        self.g.update_objects(0, self.objects)
        self.g.update(self.cams[self.at % len(self.cams)])
        self.at += 1
        self.g.render()

    def warm_up(self, render):
        """The start-up frames of a program: every camera once, so that the work queues have their size."""
        for _ in range(len(self.cams)):
            render()
            while self.g.sync_code() == OVERFLOW:
                self.g.render()
        self.at = 0


def _texture(gen, size, kind, cells):
    """Value noise with a full mip chain, made on the GPU: sRGB colour, normal map or metallic-roughness."""
    n = torch.zeros(1, 3, size, size, device="cuda")
    for o in range(3):
        c = max(1, min(cells << o, size))
        lattice = torch.rand(1, 3, c, c, generator=gen, device="cuda")
        n += 0.5 ** o / 1.75 * F.interpolate(lattice, size=(size, size), mode="bilinear", align_corners=False)
    one = torch.ones_like(n[:, :1])
    if kind == sc.IMAGE_NORMAL_MAP:
        xy = n[:, :2] * 0.8 - 0.4
        img = torch.cat([torch.cat([xy, (1.0 - (xy * xy).sum(1, keepdim=True)).sqrt()], 1) * 0.5 + 0.5, one], 1)
    elif kind == sc.IMAGE_METALLIC_ROUGHNESS:
        img = torch.cat([one, 0.15 + 0.85 * n[:, :1], (n[:, 1:2] * 1.6 - 0.5).clamp(0, 1), one], 1)
    else:
        img = torch.cat([0.1 + 0.85 * n, one], 1)
    levels = []
    while True:
        levels.append((img * 255.0).round().to(torch.uint8)[0].permute(1, 2, 0).reshape(-1))
        if img.shape[-1] == 1:
            break
        img = F.avg_pool2d(img, 2)
    return sc.Texture(size, size, len(levels), kind, torch.cat(levels).cpu().numpy())


def _scene(case, seed):
    s = sc.scene_scale(seed=seed, meshes=case["meshes"], triangles_per_mesh=case["triangles"], materials=case["materials"],
                       texture_size=4, width=case["width"], height=case["height"], shadow_size=case["shadow"], frames=4)
    gen = torch.Generator("cuda").manual_seed(seed)
    kinds = [(sc.IMAGE_COLOR, 16), (sc.IMAGE_NORMAL_MAP, 32), (sc.IMAGE_METALLIC_ROUGHNESS, 8)]
    s.textures = [_texture(gen, case["texture"], *kinds[i % 3]) for i in range(3 * case["materials"])]
    s.samples = case["samples"]
    n = case.get("cascades", 1)
    if n > 1:  # the near cascade covers the light's extent / 2^(n - 2), the coarsest twice the extent
        s.draw_config["shadow_cascades"] = n
        for c in s.cameras:
            p = c["shadow_projection_near"][0].reshape(4, 4)
            p[:, 0:2] *= 2.0 ** (n - 2)
    if case["kind"] == "blended":
        s = sc.with_blended(s, fraction=case["fraction"], mask_cutoff=0.5 if case["mask"] else None, seed=seed)
        if case["lines"]:
            s.debug_objects = sc.random_debug_objects(seed, case["lines"], extent=12.0)
    return s


def _soup(case, seed):
    s = sc.random_triangles(seed=seed, triangles=case["triangles"], width=case["width"], height=case["height"],
                            shadow_size=case["shadow"], texture_size=case["texture"])
    s.samples = case.get("samples", 1)
    s.cameras = [sc.orbit_view(s, d, s.width, s.height) for d in sc.camera_dirs(4, seed)]
    return s


def _open(s):
    r = Renderer()
    r.g.init(s.width, s.height, s.shadow_size, samples=s.samples)
    r.g.set_asset(s)
    r.g.set_graphic_objects(s.objects, s.surfaces)
    r.g.set_draw_config(s.draw_config)
    if s.debug_objects is not None:
        r.g.set_debug_objects(s.debug_objects)
    r.cams = [np.ascontiguousarray(c) for c in s.cameras]
    r.objects = np.ascontiguousarray(s.objects, np.float32)
    r.samples, r.cascades = s.samples, max(1, int(s.draw_config["shadow_cascades"][0]))
    return r


def _frame_outputs(r):
    f = r.g.frame()
    h, w, n = f.height, f.width, f.shadow_map_size
    return {"color": r.tensor(f.color_rgba8, (h, w, 4), "|u1"), "depth": r.tensor(f.depth_f32, (h, w), "<f4"),
            "visibility": r.tensor(f.visibility_u64, (r.samples, h, w), "<i8"),
            "shadow": r.tensor(f.shadow_map_f32, (r.cascades, n, n), "<f4")}


def _prepare_frame(case, seed):
    r = _open(_soup(case, seed) if case["kind"] == "soup" else _scene(case, seed))
    r.warm_up(r.next_frame)
    if case["kind"] == "host":
        h, w = case["height"], case["width"]
        r.color = torch.empty(h, w, 4, dtype=torch.uint8, pin_memory=True).numpy()
        r.depth = torch.empty(h, w, dtype=torch.float32, pin_memory=True).numpy()
    return r


def _run_frame(r):
    r.next_frame()
    return _frame_outputs(r)


def _run_host(r):
    r.next_frame()
    r.g.read_frame(r.color, r.depth)
    r.g.read_sync()
    return {"color": r.color, "depth": r.depth}


def _layout(case):
    """The scenes' triangle counts and the views' (scene, width, height, shadow map): uneven, the case's own."""
    rng = random.Random(case["views"])
    tris = [_log(rng, 1000, case["max_tris"]) for _ in range(case["scenes"])]
    return tris, [(rng.randrange(len(tris)), _log(rng, 64, case["max_size"]), _log(rng, 64, case["max_size"]),
                   _log(rng, 512, case["max_shadow"])) for _ in range(case["views"])]


def _prepare_views(case, seed):
    tris, layout = _layout(case)
    r, scenes = Renderer(), []
    r.g.init(64, 64, 512)
    for k, n in enumerate(tris):
        meshes = max(1, min(64, n // 2048))
        scenes.append(_scene({"kind": "views", "meshes": meshes, "triangles": max(128, n // meshes // 128 * 128),
                              "materials": min(8, meshes), "texture": 256, "width": 512, "height": 512, "shadow": 512,
                              "samples": 1}, len(tris) * seed + k))
        r.g.add_scene(scenes[-1])
    views = [(k, sc.view_of(scenes[k], w, h, n, camera=i)) for i, (k, w, h, n) in enumerate(layout)]
    r.g.set_views([(k, v.width, v.height, v.shadow_size, v.draw_config) for k, v in views])
    r.cams = [[np.ascontiguousarray(v.scene) for _, v in views]]
    r.warm_up(lambda: _render_views(r))
    return r


def _render_views(r):
    for i, c in enumerate(r.cams[0]):
        r.g.update_view(i, c)
    r.g.render()


def _run_views(r):
    _render_views(r)
    out, f = [], _abi.RzFrameOut()
    for i in range(len(r.cams[0])):
        r.g._lib.rz_get_view_frame(r.g._ctx, i, ctypes.byref(f))
        out.append((r.tensor(f.color_rgba8, (f.height, f.width, 4), "|u1"),
                    r.tensor(f.visibility_u64, (f.height, f.width), "<i8")))
    return out


def _prepare_learned(case, seed):
    r = _open(_soup(case, seed))
    r.g.set_gbuffer(True)
    r.warm_up(r.next_frame)
    r.net = Upsampler(0, case["width"], case["height"])
    r.net.set_params(_params(seed))
    r.out = torch.zeros(2 * case["height"], 2 * case["width"], 4, dtype=torch.uint8, device="cuda")
    return r


def _run_learned(r):
    r.next_frame()
    gb = r.g.gbuffer()
    r.net.infer(gb, r.out.data_ptr(), r.g.stream)
    n = (gb.height, gb.width)
    return {"out": r.out, "color": r.tensor(gb.color_rgba8, (*n, 4), "|u1"), "albedo": r.tensor(gb.albedo_rgba8, (*n, 4), "|u1"),
            "normal": r.tensor(gb.normal_oct_f16x2, (*n, 2), "<f2"), "sources": r.tensor(gb.sources_u16, n, "<i2")}


# --- the learned x2 network ----------------------------------------------------------------


def _params(seed):
    """A network as after some training: the initial weights, biases, and a last layer of some size."""
    p = init_params(seed, last_scale=0.3)
    rng = np.random.default_rng(seed)
    for (_, bo), (_, cout) in zip(OFFSETS, LAYERS):
        n = 12 if cout == 16 else cout
        p[bo:bo + n] = rng.normal(0.0, 0.05, n).astype(np.float32)
    return p


def _labels(jitter, x, y, cell):
    """The nearest of a jittered grid of sites at points (x, y): a label per point (patches like a frame's triangles)."""
    gx, gy = (x / cell).floor().long(), (y / cell).floor().long()
    best, label = torch.full_like(x, 1e30), torch.zeros_like(gx)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            cx, cy = (gx + dx).clamp(0, jitter.shape[1] - 1), (gy + dy).clamp(0, jitter.shape[0] - 1)
            site = jitter[cy, cx]
            d = (x - (cx + site[..., 0]) * cell) ** 2 + (y - (cy + site[..., 1]) * cell) ** 2
            label = torch.where(d < best, cy * jitter.shape[1] + cx, label)
            best = torch.minimum(best, d)
    return label


def _images(w, h, seed, sources):
    """A half-resolution G-buffer of flat-shaded patches and the full-resolution frame it stands for."""
    gen = torch.Generator("cuda").manual_seed(seed)
    cell = 9.0
    jitter = torch.rand(int(h / cell) + 2, int(w / cell) + 2, 2, generator=gen, device="cuda")
    n = jitter.shape[0] * jitter.shape[1]
    tint = torch.rand(n, 3, generator=gen, device="cuda")
    light = 0.2 + 0.8 * torch.rand(n, 1, generator=gen, device="cuda")
    normal = torch.rand(n, 2, generator=gen, device="cuda") - 0.5
    depth = 0.3 * torch.rand(n, generator=gen, device="cuda") ** 3
    covered = torch.rand(n, generator=gen, device="cuda") < 0.9

    def grid(width, height, scale):
        y, x = torch.meshgrid((torch.arange(height, device="cuda") + 0.5) * scale,
                              (torch.arange(width, device="cuda") + 0.5) * scale, indexing="ij")
        return x, y

    def shade(label, x, y):
        c = tint[label] * light[label] * (0.75 + 0.25 * torch.sin(0.05 * x + 0.03 * y))[..., None]
        c = torch.where(covered[label][..., None], c, torch.tensor([0.0, 0.25, 0.35], device="cuda"))
        return (torch.cat([c, torch.ones_like(c[..., :1])], -1) * 255.0).round().to(torch.uint8).contiguous()

    x, y = grid(w, h, 1.0)
    lo = _labels(jitter, x, y, cell)
    xf, yf = grid(2 * w, 2 * h, 0.5)
    hi = _labels(jitter, xf, yf, cell)
    on = covered[lo]
    albedo = torch.where(on[..., None], tint[lo], torch.zeros((), device="cuda"))
    gb = {"color": shade(lo, x, y), "target": shade(hi, xf, yf),
          "albedo": (torch.cat([albedo, on[..., None].float()], -1) * 255.0).round().to(torch.uint8).contiguous(),
          "depth": torch.where(on, depth[lo], torch.zeros((), device="cuda")).contiguous(),
          "normal": torch.where(on[..., None], normal[lo], torch.zeros((), device="cuda")).half().contiguous()}
    if sources:
        mask = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        ix, iy = torch.arange(w, device="cuda"), torch.arange(h, device="cuda")
        for k in range(4):
            nx, ny = (ix + (1 if k & 1 else -1)).clamp(0, w - 1), (iy + (1 if k >> 1 else -1)).clamp(0, h - 1)
            point = hi[k >> 1::2, k & 1::2]
            for s, src in enumerate((lo, lo[:, nx], lo[ny], lo[ny][:, nx])):
                mask |= (src == point).int() << (4 * k + s)
        gb["sources"] = mask.to(torch.int16).contiguous()
    return gb


def _gbuffer(im):
    g = _abi.RzGbuffer()
    g.color_rgba8, g.depth_f32 = im["color"].data_ptr(), im["depth"].data_ptr()
    g.albedo_rgba8, g.normal_oct_f16x2 = im["albedo"].data_ptr(), im["normal"].data_ptr()
    g.sources_u16 = im["sources"].data_ptr() if "sources" in im else None
    g.height, g.width = im["depth"].shape
    return g


class Network:
    def __init__(self, case, seed, batch):
        w, h = case["width"], case["height"]
        self.images = [_images(w, h, 1000 * seed + i, case["sources"]) for i in range(batch)]
        self.gb = [_gbuffer(im) for im in self.images]
        self.net = Upsampler(0, w, h)
        self.net.set_params(_params(seed))
        self.out = torch.zeros(2 * h, 2 * w, 4, dtype=torch.uint8, device="cuda")


def _run_upsample(st):
    st.net.infer(st.gb[0], st.out.data_ptr())
    return st.out


LEARNING_RATE = 1e-7  # as near the end of the cosine schedule, where passes of one state stay alike


def _run_train(st):
    for g, im in zip(st.gb, st.images):
        st.net.accumulate(g, im["target"].data_ptr())
    grads, loss, values = st.net.grads()
    st.net.adam_step(LEARNING_RATE, grad_scale=1.0 / values)
    return {"grads": grads, "loss": loss, "params": st.net.params()}


def _exact_train(case, seed):
    """The same step in 64 bits: torch convolutions and their gradients, no 16-bit storage."""
    p0 = torch.from_numpy(_params(seed)).cuda().double().requires_grad_(True)
    total, values = 0.0, 0
    for i in range(case["batch"]):
        im = _images(case["width"], case["height"], 1000 * seed + i, case["sources"])
        c = im["color"].double() / 255.0
        h, w = im["depth"].shape
        feats = [c[..., :3], im["albedo"].double()[..., :3] / 255.0, im["normal"].double(),
                 im["albedo"].double()[..., 3:] / 255.0, (im["depth"].double() * 16.0).clamp(max=4.0)[..., None]]
        bilinear = (0.5625, 0.1875, 0.1875, 0.0625)
        mask = im["sources"].int() if "sources" in im else torch.full((h, w), 0xFFFF, dtype=torch.int32, device="cuda")
        kept = [[((mask >> (4 * k + s)) & 1).double() * bilinear[s] for s in range(4)] for k in range(4)]
        matched = torch.stack([sum(k) for k in kept], -1) if "sources" in im else torch.zeros(h, w, 4, device="cuda").double()
        x = torch.cat(feats + [matched, torch.zeros(h, w, 2, device="cuda").double()], -1).permute(2, 0, 1)[None]
        for l, ((wo, bo), (cin, cout)) in enumerate(zip(OFFSETS, LAYERS)):
            weight = p0[wo:bo].reshape(cout, 9, cin)
            xp = F.pad(x, (1, 1, 1, 1))
            y = sum(torch.einsum("oc,chw->ohw", weight[:, t], xp[0, :, t // 3:t // 3 + h, t % 3:t % 3 + w]) for t in range(9))
            x = (y + p0[bo:bo + cout, None, None])[None]
            x = F.relu(x) if l < 3 else x
        ix, iy = torch.arange(w, device="cuda"), torch.arange(h, device="cuda")
        rgb = c[..., :3]
        for k in range(4):
            nx, ny = (ix + (1 if k & 1 else -1)).clamp(0, w - 1), (iy + (1 if k >> 1 else -1)).clamp(0, h - 1)
            sums = sum(kept[k])
            ws = [torch.where(sums > 0, a / sums.clamp(min=1e-30), torch.full_like(a, b)) for a, b in zip(kept[k], bilinear)]
            base = sum(a[..., None] * b for a, b in zip(ws, (rgb, rgb[:, nx], rgb[ny], rgb[ny][:, nx])))
            v = base.permute(2, 0, 1) + x[0, 3 * k:3 * k + 3]
            t = im["target"][k >> 1::2, k & 1::2, :3].double().permute(2, 0, 1) / 255.0
            total = total + ((v - t) ** 2).sum()
        values += 12 * h * w
    total.backward()
    g = p0.grad
    step = g / values
    new = p0.detach() - LEARNING_RATE * step / (step.abs() + 1e-8)
    return {"grads": g.cpu().numpy(), "loss": float(total.detach()), "params": new.cpu().numpy()}


# --- compressed textures ----------------------------------------------------------------------


def _prepare_bc7(case, seed):
    """Blocks of every mode in the proportions of a shuffled pool (a texture's blocks mix modes)."""
    w, h = case["width"], case["height"]
    pool = torch.from_numpy(bc7.mixed_blocks(np.random.default_rng(seed), 1024)).cuda()
    gen = torch.Generator("cuda").manual_seed(seed)
    n = ((w + 3) // 4) * ((h + 3) // 4)
    blocks = pool[torch.randint(0, len(pool), (n,), generator=gen, device="cuda")].contiguous()
    return {"lib": _lib.load(), "blocks": blocks, "w": w, "h": h,
            "out": torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")}


def _run_bc7(st):
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = st["lib"].rz_bc7_decode(ctypes.c_void_p(st["blocks"].data_ptr()), st["w"], st["h"],
                                 ctypes.c_void_p(st["out"].data_ptr()), stream)
    if rc != 0:
        raise RuntimeError("rz_bc7_decode: %d" % rc)
    return st["out"]


# --- the contract -------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "views":
        st = _prepare_views(case, seed)
    elif kind == "learned":
        st = _prepare_learned(case, seed)
    elif kind in ("upsample", "train"):
        st = Network(case, seed, case.get("batch", 1))
    elif kind == "bc7":
        st = _prepare_bc7(case, seed)
    else:
        st = _prepare_frame(case, seed)
    torch.cuda.synchronize()  # the renderer's streams do not wait for torch's
    return {"kind": kind, "state": st}


RUN = {"soup": _run_frame, "scene": _run_frame, "blended": _run_frame, "host": _run_host, "views": _run_views,
       "learned": _run_learned, "upsample": _run_upsample, "train": _run_train, "bc7": _run_bc7}


def run(state):
    return RUN[state["kind"]](state["state"])


def exact(case, seed):
    return _exact_train(case, seed) if case["kind"] == "train" else None


def _frame_work(pixels, samples, shadow_texels, tris, verts, textures):
    """Compulsory traffic of a frame: vertices and indices once per pass, the shadow map and the visibility
    written and read once, colour and depth out, every texture read at most once; about 600 operations a pixel
    (three trilinear samples, nine shadow taps, the lighting) and 150 a triangle and pass."""
    texel_bytes = min(textures, 3 * 8 * pixels) * 4
    return {"bytes": 2 * (64 * verts + 12 * tris) + 8 * shadow_texels + (16 * samples + 8) * pixels + texel_bytes,
            "flops": 600 * pixels + 300 * tris}


def work(case):
    kind = case["kind"]
    px = case.get("width", 0) * case.get("height", 0)
    macs = 9 * (14 * 32 + 32 * 32 + 32 * 32 + 32 * 12) * px  # the network's real channels
    if kind == "bc7":
        return {"bytes": ((case["width"] + 3) // 4) * ((case["height"] + 3) // 4) * 16 + 4 * px, "flops": 0}
    if kind == "upsample":
        return {"bytes": 4 * 4 * px + 16 * px + 4 * PARAM_COUNT, "flops": 2 * macs}
    if kind == "train":
        return {"bytes": case["batch"] * (18 * px + 16 * px) + 24 * PARAM_COUNT, "flops": case["batch"] * 6 * macs}
    if kind == "views":
        counts, views = _layout(case)
        tris = sum(counts[k] for k, _, _, _ in views)
        return _frame_work(sum(w * h for _, w, h, _ in views), 1, sum(n * n for *_, n in views), tris, sum(counts) / 1.9,
                           case["scenes"] * 24 * 87381)
    tris = case["triangles"] * case.get("meshes", 1)
    verts = 3 * tris if kind in ("soup", "learned") else tris / 1.9
    tex = (1 if kind in ("soup", "learned") else 3 * case["materials"]) * case["texture"] ** 2 * 4 // 3
    w = _frame_work(px, case.get("samples", 1), case.get("cascades", 1) * case["shadow"] ** 2, tris, verts, tex)
    if kind == "learned":
        w = {"bytes": w["bytes"] + 34 * px, "flops": w["flops"] + 2 * macs}
    return w
