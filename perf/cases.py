"""The work that users of this library have it do, as measurable cases.

Each case is one pass through the public entry points (the Python mirror `sqwheel` of the C ABI in include/swgpu.h
and include/swlearn.h): whole frames as a game's frame loop asks for them, the per-call API, the batched
surface build, the HDR postprocessor alone, the frame upscalers, and the learned upscaler's training step.

A case's "kind" names the calls that `run` makes; its other fields are sizes and options:

  frame     HostRenderer.render_frame: visibility and preparation, then the whole frame into device memory
  draw      GpuRenderer.draw_frame: a whole frame from descriptors that the host program prepared itself
  calls     frame_begin, submit_surfaces, submit_draws, render (and postprocess) one after another
  surfaces  frame_begin, rebuild_surfaces, submit_draws, render: a batch of surfaces, every texel of it shown
  post      postprocess of the HDR frame in the context
  noalloc   sw_postprocess_noalloc: the postprocessor of callers that own their device memory
  upscale   the non-learned frame upscalers (nearest, 2x average)
  infer     Upscaler.infer: the learned 2x upscale
  train     Upscaler.train_step, then the updated parameters (params), as a loop that keeps checkpoints does
  grads     Upscaler.gradients: loss and gradients without an update
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "square-wheel_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from sqwheel import abi, gpu, host, learned, synth  # noqa: E402

DEV = "cuda:0"

# The maps that frames are drawn of: the small colour32 map, the full-size HDR map, the same with four shadowed
# lights (one of them a projector), scrolling, framed, turbulent, layered, water and fire materials, and the
# 128-room map with portals, models, sprites and decals. Effects move with time alone, so their map's camera path
# is a long one, walked slowly; on the others a frame loop repeats eight consecutive frames.
MAPS = {
    "small": host.SMALL_MAP,
    "sky": host.SKY_MAP,
    "full": host.FULL_MAP,
    "effects": dict(host.FULL_MAP, num_frames=16384, shadowed_lights=4, projector_lights=1, scrolling_materials=2,
                    animated_materials=2, turb_materials=2, layered_materials=2, water_materials=2, fire_materials=1),
    "stress": host.STRESS_MAP,
}
_scenes = {}


def scene_of(name):
    """A map is loaded once by a program and drawn from many poses: the seed of a case picks the pose."""
    if name not in _scenes:
        _scenes[name] = host.Scene(**MAPS[name])
    return _scenes[name]


def listed():
    return [
        # the CPU-runnable configuration's frame: colour32, no postprocess; launches and latency decide
        {"name": "frame_small_640x480", "kind": "draw", "map": "small", "width": 640, "height": 480, "hdr": False},
        # the headline frame: HDR, directional lightmaps, normal maps, specular, 8 moving lights, bloom and tonemap
        {"name": "frame_hdr_1920x1080", "kind": "frame", "map": "full", "width": 1920, "height": 1080, "hdr": True},
        # the drop-in's per-call API on a laptop panel's size (odd tiles on both sides)
        {"name": "calls_hdr_1366x768", "kind": "calls", "map": "full", "width": 1366, "height": 768, "hdr": True},
        # shadow maps, simulated and generated textures ahead of every frame
        {"name": "frame_effects_1920x1080", "kind": "frame", "map": "effects", "width": 1920, "height": 1080, "hdr": True},
        # the stress map at 4K: portal views, model, sprite and decal triangles
        {"name": "frame_stress_3840x2160", "kind": "frame", "map": "stress", "width": 3840, "height": 2160, "hdr": True},
        # the batched surface build's configuration: 4,096 surfaces of 4x4 to 512x512 texels, directional lightmaps
        {"name": "surfaces_4096_hdr", "kind": "surfaces", "count": 4096, "max_side": 512, "hdr": True, "directional": True,
         "lights": 0},
        # simple lightmaps, colour32, dynamic lights: what a small map's surface rebuild is made of
        {"name": "surfaces_512_c32", "kind": "surfaces", "count": 512, "max_side": 256, "hdr": False, "directional": False,
         "lights": 6},
        # an HDR frame rendered elsewhere, wide linear bloom, a common desktop size
        {"name": "post_2560x1440", "kind": "post", "width": 2560, "height": 1440, "scale_log2": 2, "sigma": 2.0, "linear": 1},
        # the learned upscale of a thumbnail or an inset view: a handful of tiles, odd sides
        {"name": "infer_161x91", "kind": "infer", "width": 161, "height": 91},
        # half of 1080p: the learned upscaler's own configuration
        {"name": "infer_960x540", "kind": "infer", "width": 960, "height": 540},
        # half of 4K: the stress configuration's upscale
        {"name": "infer_1920x1080", "kind": "infer", "width": 1920, "height": 1080},
        # one training step at the batch the training loop uses
        {"name": "train_16", "kind": "train", "crops": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "draw", "calls", "surfaces", "surfaces", "post", "noalloc", "upscale", "infer", "infer",
                       "train", "grads"])
    if kind in ("frame", "draw", "calls"):
        m = rng.choice({"frame": ["small", "sky", "full", "effects", "stress"], "draw": ["small", "full"],
                        "calls": ["small", "full"]}[kind])
        w = _log_int(rng, 320, 3840)
        return {"kind": kind, "map": m, "width": w, "height": max(180, w * rng.choice([9, 10, 12]) // 16),
                "hdr": m != "small" and (m != "sky" or rng.random() < 0.5)}
    if kind == "surfaces":
        return {"kind": kind, "count": _log_int(rng, 32, 3000), "max_side": rng.choice([64, 200, 256, 512]),
                "hdr": rng.random() < 0.6, "directional": rng.random() < 0.6, "lights": rng.choice([0, 0, 3, 6])}
    if kind in ("post", "noalloc"):
        w = _log_int(rng, 320, 3840 if kind == "post" else 1920)
        return {"kind": kind, "width": w, "height": max(180, min(2160 if kind == "post" else 1080, w * 9 // 16 + rng.randrange(8))),
                "scale_log2": rng.choice([1, 1, 2, 3]), "sigma": rng.choice([0.0, 1.0, 1.0, 2.5]), "linear": rng.randrange(2)}
    if kind == "upscale":
        w = 2 * _log_int(rng, 640, 1920)
        return {"kind": kind, "width": w, "height": 2 * (w * 9 // 32), "average": rng.random() < 0.5}
    if kind == "infer":
        w = _log_int(rng, 100, 1920)
        return {"kind": kind, "width": w, "height": max(60, w * 9 // 16 + rng.randrange(5))}
    return {"kind": kind, "crops": _log_int(rng, 1, 16 if kind == "train" else 12)}


# ---- inputs ----


def _pack(b):
    return ((b[0] | (b[1] << 8) | (b[2] << 16) | (255 << 24)) - (1 << 32)).to(torch.int32).contiguous()  # alpha 255: the sign bit


def _image(gen, height, width):
    """A rendered-looking Color32 frame: smooth shading, flat blocks with hard edges, fine texture."""
    def noise(n):
        c = torch.rand((1, 3, max(2, height // n), max(2, width // n)), generator=gen, device=DEV)
        return torch.nn.functional.interpolate(c, size=(height, width), mode="bilinear", align_corners=False)[0]
    blocks = torch.rand((1, 3, height // 24 + 1, width // 24 + 1), generator=gen, device=DEV)
    blocks = torch.nn.functional.interpolate(blocks, size=(height, width), mode="nearest")[0]
    v = (0.5 * noise(64) + 0.3 * blocks + 0.2 * noise(3)).clamp(0, 1)
    b = (v * 255.0).round().to(torch.int64)
    return _pack(b)


def _hdr(gen, height, width):
    """Color64 as the renderer leaves it: 256 is white, most pixels below it, a few lamps far above."""
    c = torch.rand((1, 3, max(2, height // 48), max(2, width // 48)), generator=gen, device=DEV)
    v = torch.nn.functional.interpolate(c, size=(height, width), mode="bilinear", align_corners=False)[0] * 400.0
    v = v * (0.6 + 0.8 * torch.rand((3, height, width), generator=gen, device=DEV))
    lamp = torch.rand((1, 1, height // 40 + 1, width // 40 + 1), generator=gen, device=DEV) < 0.01
    lamp = torch.nn.functional.interpolate(lamp.float(), size=(height, width), mode="nearest")[0]
    b = (v + lamp * 12000.0).clamp(0, 65535).to(torch.int64)
    return (b[0] | (b[1] << 16) | (b[2] << 32) | (255 << 48)).contiguous()


def _post_config(case):
    c = abi.PostConfig.default()
    if "sigma" in case:
        c.bloom_sigma, c.bloom_buffer_scale_log2, c.linear_bloom_filter = case["sigma"], case["scale_log2"], case["linear"]
        if case["sigma"] == 0.0:
            c.bloom_scale = 0.0
    return c


def _he_params(seed):
    """He-normal weights, zero biases, a small last layer: the canonical parameter layout of swlearn.h."""
    rng = np.random.default_rng(seed)
    p = []
    for ci, co, k in ((3, 32, 1.0), (32, 32, 1.0), (32, 32, 1.0), (32, 12, 0.1)):
        p.append(rng.normal(0, k * math.sqrt(2.0 / (9 * ci)), co * 9 * ci))
        p.append(np.zeros(co))
    return np.concatenate(p).astype(np.float32)


def _train_inputs(case, seed):
    """Frame pairs and the crops a training step takes of them."""
    gen = torch.Generator(DEV).manual_seed(seed)
    rng = np.random.default_rng(seed)
    hi = [_image(gen, 540, 960) for _ in range(4)]
    lo = []
    for h in hi:
        u = torch.stack([(h >> s) & 255 for s in (0, 8, 16)]).float()
        m = torch.nn.functional.avg_pool2d(u[None], 2)[0].round().to(torch.int64)
        lo.append(_pack(m))
    spots = [(int(rng.integers(4)), int(rng.integers(480 - 128 + 1)), int(rng.integers(270 - 64 + 1)))
             for _ in range(case["crops"])]
    return lo, hi, spots


def _surface_batch(case, seed):
    """Surfaces with log-uniform sides, mips 0..3 and random lightmaps, and a sheet that shows them 1:1."""
    rng = np.random.default_rng(seed)
    n = case["count"]
    texels, mips = synth.make_material_set(seed, 8, 256)
    sizes = np.random.default_rng((n, case["max_side"])).uniform(np.log(4), np.log(case["max_side"] + 1), (n, 2))
    sides = np.clip(np.exp(sizes).astype(np.int64), 4, case["max_side"])  # a case's sheet has one size, whatever the seed
    mip = rng.integers(0, 4, n)
    log2 = 4 - mip
    shift = rng.integers(0, 1 << 16, (n, 2)) & ((1 << log2[:, None]) - 1)
    lm = ((sides - 1 + shift) >> log2[:, None]) + 2
    lm_count = lm[:, 0] * lm[:, 1]
    total_lm = int(1 + lm_count.sum())
    if case["directional"]:  # 64k random elements, repeated: drawing every one of millions takes seconds
        dirl, simple = np.resize(synth.random_directional_lightmap(rng, min(total_lm, 65521)), total_lm), None
    else:
        dirl, simple = None, np.resize(rng.uniform(0, 4, (min(total_lm, 65521), 3)).astype(np.float32), (total_lm, 3))
    q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q = q.astype(np.float32)
    d = np.zeros(n, abi.SURFACE_DESC)
    scale = (1 << mip).astype(np.float32)[:, None]
    d["basis_u"], d["basis_v"], d["basis_normal"] = q[:, 0] * scale, q[:, 1] * scale, q[:, 2]
    d["basis_start"] = rng.uniform(-256, 256, (n, 3))
    d["size"], d["tc_start"] = sides, rng.integers(-2048, 2048, (n, 2))
    d["texture_mip"] = rng.integers(0, 8, n) * synth.NUM_MIPS + mip
    d["emissive_mip"] = abi.SW_NO_EMISSIVE
    d["lightmap_offset"] = 1 + np.concatenate([[0], np.cumsum(lm_count)[:-1]])
    d["lightmap_size"], d["lightmap_scale_log2"], d["lightmap_tc_shift"] = lm, log2, shift
    d["flags"] = abi.SW_SURF_DIFFUSE_LAYER
    lights = synth.random_lights(rng, case["lights"])
    if case["lights"]:
        d["num_lights"] = rng.integers(0, min(case["lights"], abi.SW_MAX_POLYGON_LIGHTS) + 1, n)
        d["lights"][:, :case["lights"]] = np.argsort(rng.random((n, case["lights"])), axis=1)
    area = sides[:, 0] * sides[:, 1]
    d["out_offset"] = np.concatenate([[0], np.cumsum(area)[:-1]])
    # shelves of surfaces sorted by height, as an atlas packs them
    width = int(min(16384, max(case["max_side"], 1.02 * math.sqrt(float(area.sum())) + 64)))
    draws, verts = np.zeros(n, abi.DRAW_CMD), np.zeros((n, 4), abi.VERTEX16)
    x = y = shelf = 0
    for k, i in enumerate(np.argsort(-sides[:, 1], kind="stable")):
        w, h = int(sides[i, 0]), int(sides[i, 1])
        if x + w > width:
            x, y, shelf = 0, y + shelf, 0
        shelf = max(shelf, h)
        verts[k]["x"] = np.array([x, x + w, x + w, x]) << 16
        verts[k]["y"] = np.array([y, y, y + h, y + h]) << 16
        c = draws[k]
        c["first_vertex"], c["vertex_count"], c["mode"] = 4 * k, 4, abi.SW_RASTER_AFFINE
        c["depth_eq"], c["tc_eq"] = (0, 0, 1), (1, 0, 0, 1, -x, -y)
        c["tex_size"], c["tex_offset"] = (w, h), d["out_offset"][i]
        x += w
    static = gpu.StaticData(texels, mips, lightmaps=simple, directional_lightmaps=dirl)
    fmt = abi.SW_PIXEL_C64 if case["hdr"] else abi.SW_PIXEL_C32
    cam = rng.uniform(-512, 512, 3).astype(np.float32)
    params = gpu.frame_params(width, y + shelf, fmt, cam, directional=case["directional"], clear_background=True)
    return static, params, lights, d, int(area.sum()), draws, verts.reshape(-1)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, kind = case, case["kind"]
    gen = torch.Generator(DEV).manual_seed(seed)
    if kind in ("frame", "draw", "calls"):
        w, h, hdr = case["width"], case["height"], case["hdr"]
        scene = scene_of(case["map"])
        s.options = host.frame_options(w, h, abi.SW_PIXEL_C64 if hdr else abi.SW_PIXEL_C32, directional=case["map"] not in ("small", "sky"))
        s.index, s.passes = int(np.random.default_rng(seed).integers(scene.info().frames)), 0
        s.post = abi.PostConfig.default() if hdr else None
        s.out = torch.zeros((h, w), dtype=torch.int32, device=DEV)
        if kind == "frame":
            s.renderer = host.HostRenderer(scene)
        else:
            s.renderer = gpu.GpuRenderer(scene.static_data())
            s.frame = host.Frame(scene)
            f = s.frame.prepare(s.index, s.options)
            s.arrays = f.params, f.lights, f.surfaces, f.total_texels, f.draws, f.vertices
            if kind == "draw":
                s.input = s.renderer.frame_input(*s.arrays, post_config=s.post, dst_device_ptr=s.out.data_ptr(), pitch=w)
    elif kind == "surfaces":
        static, s.params, s.lights, descs, total, s.draws, s.verts = _surface_batch(case, seed)
        s.renderer = gpu.GpuRenderer(static)
        s.out = torch.zeros((s.params.height, s.params.width), dtype=torch.int64 if case["hdr"] else torch.int32, device=DEV)
        s.renderer.frame_begin(s.params, s.lights)
        s.renderer.submit_surfaces(descs, total)
        s.renderer.sync()
    elif kind in ("post", "noalloc"):
        w, h = case["width"], case["height"]
        hdr = _hdr(gen, h, w)
        s.post = _post_config(case)
        s.out = torch.zeros((h, w), dtype=torch.int32, device=DEV)
        if kind == "post":
            s.renderer = gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))
            s.renderer.set_framebuffer(hdr.cpu().numpy().view(np.uint64), abi.SW_PIXEL_C64)
            s.renderer.sync()
        else:
            s.hdr, s.average = hdr, torch.zeros(4, device=DEV)
            s.modulate = (ctypes.c_float * 3)(1.0, 1.0, 1.0)
            s.call = gpu.load_library().sw_postprocess_noalloc
    elif kind == "upscale":
        w, h = case["width"], case["height"]
        s.renderer = gpu.GpuRenderer(gpu.StaticData(np.zeros(1, np.uint64), np.zeros(0, abi.TEXTURE_MIP)))
        s.lo = _image(gen, h // 2, w // 2)
        s.out = torch.zeros((h, w), dtype=torch.int32, device=DEV)
    elif kind == "infer":
        s.upscaler = learned.Upscaler(0, seed=1)
        s.upscaler.set_params(_he_params(seed))
        s.lo = _image(gen, case["height"], case["width"])
        s.out = torch.zeros((2 * case["height"], 2 * case["width"]), dtype=torch.int32, device=DEV)
    else:
        s.upscaler = learned.Upscaler(0, seed=1)
        s.upscaler.set_params(_he_params(seed))
        s.lo, s.hi, spots = _train_inputs(case, seed)
        s.items = [(s.lo[k], s.hi[k], x, y) for k, x, y in spots]
    torch.cuda.synchronize()
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "frame":
        index = s.index + (s.passes if case["map"] == "effects" else s.passes % 8)
        s.passes += 1
        s.renderer.render_frame(index, s.options, device_ptr=s.out.data_ptr(), pitch=s.out.stride(0), post=s.post)
        return s.out
    if kind == "draw":
        s.renderer.draw_frame(s.input)
        return s.out
    if kind == "calls":
        params, lights, surfaces, total, draws, vertices = s.arrays
        r = s.renderer
        r.frame_begin(params, lights)
        r.submit_surfaces(surfaces, total)
        r.submit_draws(draws, vertices)
        if s.post is None:
            r.render(device_ptr=s.out.data_ptr(), pitch=s.out.stride(0))
        else:
            r.render()
            r.postprocess(s.post, 1.0 / 60.0, (1.0, 1.0, 1.0), device_ptr=s.out.data_ptr(), pitch=s.out.stride(0))
        return s.out
    if kind == "surfaces":
        r = s.renderer
        r.frame_begin(s.params, s.lights)
        r.rebuild_surfaces()
        r.submit_draws(s.draws, s.verts)
        r.render(device_ptr=s.out.data_ptr(), pitch=s.out.stride(0))
        return s.out
    if kind == "post":
        s.renderer.postprocess(s.post, 1.0 / 60.0, (1.0, 1.0, 1.0), device_ptr=s.out.data_ptr(), pitch=s.out.stride(0))
        return s.out
    if kind == "noalloc":
        status = s.call(ctypes.c_void_p(s.hdr.data_ptr()), case["width"], case["height"], ctypes.byref(s.post), 1.0, s.modulate,
                        ctypes.c_void_p(s.out.data_ptr()), s.out.stride(0), ctypes.c_void_p(s.average.data_ptr()), None)
        if status != 0:
            raise gpu.SwError(f"sw_postprocess_noalloc failed ({status})")
        return {"frame": s.out, "average": s.average}
    if kind == "upscale":
        mode = abi.SW_UPSCALE_AVG2X if case["average"] else abi.SW_UPSCALE_NEAREST
        s.renderer.upscale_device(mode, 2, s.lo.data_ptr(), s.out.data_ptr(), s.out.shape[1], s.out.shape[0], s.out.stride(0))
        return s.out
    if kind == "infer":
        s.upscaler.infer(s.lo, s.out)
        return s.out
    if kind == "train":
        s.upscaler.train_step(s.items, 1e-3)
        return {"params": s.upscaler.params()}
    grads, loss = s.upscaler.gradients(s.items)
    return {"grads": grads, "loss": loss}


def work(case):
    kind = case["kind"]
    if kind in ("frame", "draw", "calls"):
        # about one surface texel for every two pixels is read and lit, every pixel is drawn, tonemapped and written
        n = case["width"] * case["height"]
        return {"bytes": n * (4 + 4 + 4 + 4), "flops": n * (300 if case["hdr"] else 60)}
    if kind == "surfaces":
        # E[side]^2 of log-uniform sides; textures, lightmaps (by mip, 1/16^2 .. 1/2^2 elements a texel) in, the sheet out
        side = (case["max_side"] - 4) / math.log(case["max_side"] / 4)
        n = case["count"] * side * side
        lm = 0.083 * (40 if case["directional"] else 12)
        return {"bytes": n * (lm + (8 if case["hdr"] else 4)) + 8 * 256 * 256 * 8 * 4 / 3,
                "flops": n * ((250 if case["directional"] else 100) + 25 * case["lights"])}
    if kind in ("post", "noalloc"):
        n = case["width"] * case["height"]
        return {"bytes": 12 * n, "flops": 40 * n}
    if kind == "upscale":
        return {"bytes": 5 * case["width"] * case["height"], "flops": 0}
    macs = 9 * (3 * 32 + 32 * 32 + 32 * 32 + 32 * 12)
    if kind == "infer":
        n = case["width"] * case["height"]
        return {"bytes": 20 * n, "flops": 2 * macs * n}
    n = case["crops"] * 128 * 64
    # forward, input gradients (but the first layer's) and weight gradients
    return {"bytes": 20 * n + 4 * 22860 * 7, "flops": 2 * (3 * macs - 9 * 3 * 32) * n}


def exact(case, seed):
    """The training kinds in 64 bits (every other kind returns pixels): the network, its loss, autograd, Adam's first step."""
    if case["kind"] not in ("train", "grads"):
        return None
    lo, hi, spots = _train_inputs(case, seed)
    p0 = torch.from_numpy(_he_params(seed)).to(DEV).double()
    p = p0.clone().requires_grad_(True)

    def lanes(t):
        return torch.stack([(t >> s) & 255 for s in (0, 8, 16)]).double() / 255.0

    loss, count = 0.0, case["crops"] * (128 - 8) * (64 - 8) * 12
    for k, x, y in spots:
        full = lanes(lo[k])
        pad = torch.nn.functional.pad(full[None], (1, 1, 1, 1), mode="replicate")[0]
        a = full[None, :, y:y + 64, x:x + 128]
        off = 0
        for layer, (ci, co) in enumerate(((3, 32), (32, 32), (32, 32), (32, 12))):
            wt = p[off:off + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)
            off += co * 9 * ci
            a = torch.nn.functional.conv2d(a, wt, p[off:off + co], padding=1)
            off += co
            if layer < 3:
                a = torch.relu(a)
        net = torch.nn.functional.pixel_shuffle(a, 2)[0]
        base = torch.zeros((3, 128, 256), dtype=torch.float64, device=DEV)
        for sy in range(2):
            for sx in range(2):
                ys, xs = slice(y + 1, y + 65), slice(x + 1, x + 129)
                yn, xn = slice(y + 2 * sy, y + 2 * sy + 64), slice(x + 2 * sx, x + 2 * sx + 128)
                base[:, sy::2, sx::2] = (0.75 * (0.75 * pad[:, ys, xs] + 0.25 * pad[:, ys, xn]) +
                                         0.25 * (0.75 * pad[:, yn, xs] + 0.25 * pad[:, yn, xn]))
        target = lanes(hi[k])[:, 2 * y:2 * y + 128, 2 * x:2 * x + 256]
        diff = (net + base - target)[:, 8:-8, 8:-8]
        loss = loss + 0.5 * (diff * diff).sum() / count
    g, = torch.autograd.grad(loss, p)
    if case["kind"] == "grads":
        return {"grads": g.cpu().numpy(), "loss": float(loss)}
    return {"params": (p0 - 1e-3 * g / (g.abs() + 1e-8)).cpu().numpy()}
