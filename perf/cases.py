"""The work this renderer is run for, as cases that can be timed one by one.

Every case goes through the public entry points: render sessions and the
render server (path tracing, sparse distance volumes, previews), the learned
denoiser (`UNet`: inference, the gradient of one training step, Adam), one
convolution layer of it through the C ABI, and the temporal and spatial image
filters.

`listed()` names the cases, `draw(rng)` gives another one of the same ranges,
`prepare(case, seed)` what a program holds before the call, `run(state)` one
pass, `work(case)` the bytes and operations the pass cannot do without and
`exact(case, seed)` the result in 64 bits where plain tensor code gives it.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from denrimrendererkit_gb300 import (Camera, DenrimRenderer, RenderOutput, RenderQuality, RenderSettings,
                                     compile_scene, library, scenes)
from denrimrendererkit_gb300.denoiser import LEVELS, SvgfDenoiser, UNet, flops_per_pixel, layer_plan, spatial_denoise
from denrimrendererkit_gb300.presets import FAMILIES, PRESETS
from denrimrendererkit_gb300.serving import RenderServer, ServerConfig

AOVS = (RenderOutput.BEAUTY, RenderOutput.DEPTH, RenderOutput.NORMAL, RenderOutput.ALBEDO, RenderOutput.MATERIAL_ID,
        RenderOutput.OBJECT_ID)


def listed():
    return [
        # A small interactive still: the Cornell-style box of the small
        # configuration, all its samples in one wave.  Launches and latency.
        {"name": "cornell_320x180_16spp", "kind": "render", "scene": "cornell", "width": 320, "height": 180, "spp": 16},
        # The final-quality frame of the large configuration (1.31 M triangles,
        # HDRI with a sun, four material families), a quarter of its samples.
        {"name": "spheres_1920x1080_16spp", "kind": "render", "scene": "spheres", "detail": 5, "width": 1920,
         "height": 1080, "spp": 16},
        # Every feature of the layered material: textures, normal map, cut-outs,
        # subsurface, rough transmission, interior media.
        {"name": "materials_512x512_16spp", "kind": "render", "scene": "materials", "width": 512, "height": 512,
         "spp": 16},
        # The sparse distance-volume configuration: 768^3 virtual grid, FP16 bricks.
        {"name": "volume_1024x1024_16spp", "kind": "render", "scene": "volume", "detail": 768, "width": 1024,
         "height": 1024, "spp": 16},
        # One frame of a viewport while the camera moves, encoded for display.
        {"name": "viewport_1280x720", "kind": "viewport", "quality": "interactive", "width": 1280, "height": 720},
        # Serving: material-preview requests of mixed sizes and sample counts
        # packed into shared waves (the serving configuration's size mix).
        {"name": "serve_20_jobs", "kind": "serve", "jobs": 20, "spp_max": 64},
        # Learned denoising of a full-HD frame, and of the three 256^2 images
        # one served request needs (two half renders and their average).
        {"name": "denoise_1920x1080", "kind": "denoise", "width": 1920, "height": 1080, "batch": 0},
        {"name": "denoise_256x256_batch3", "kind": "denoise", "width": 256, "height": 256, "batch": 3},
        # The gradient of one training step of the learned denoiser: 16 crops of 256^2.
        {"name": "train_16x256x256", "kind": "train", "crop": 256, "batch": 16},
        # Backward of one convolution layer (activation, weight, bias and input
        # gradients): the half-resolution level's layer at the training crops.
        {"name": "conv_backward_16x128x128_64_64", "kind": "conv", "direction": "backward", "batch": 16,
         "height": 128, "width": 128, "cin": 64, "cout": 64},
        # Temporal filter of a full-HD frame with its history.
        {"name": "svgf_1920x1080", "kind": "filter", "filter": "svgf", "width": 1920, "height": 1080, "radius": 2,
         "iterations": 5},
        # The optimiser's part of a training step: every layer's weights and biases.
        {"name": "adam", "kind": "adam", "step": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("render", "render", "render", "viewport", "serve", "denoise", "denoise", "train", "conv",
                       "conv", "filter", "adam"))
    if kind == "render":
        scene = rng.choice(("cornell", "spheres", "materials", "volume"))
        case = {"kind": kind, "scene": scene}
        if scene == "spheres":
            case["detail"] = rng.choice((3, 4, 5))
        if scene == "volume":
            case["detail"] = rng.choice((192, 256, 384, 512, 768))
        case["width"] = _log_int(rng, 96, 1920)
        case["height"] = _log_int(rng, 96, 1080)
        pixels = case["width"] * case["height"]
        top = {"cornell": 24e6, "spheres": 30e6, "materials": 6e6, "volume": 16e6}[scene]
        case["spp"] = max(1, min(_log_int(rng, 1, 64), int(top / pixels)))
        return case
    if kind == "viewport":
        return {"kind": kind, "quality": rng.choice(("preview", "interactive")), "width": _log_int(rng, 128, 1920),
                "height": _log_int(rng, 96, 1080)}
    if kind == "serve":
        return {"kind": kind, "jobs": rng.randint(2, 20), "spp_max": rng.choice((16, 64))}
    if kind == "denoise":
        if rng.random() < 0.5:
            return {"kind": kind, "width": _log_int(rng, 96, 1920), "height": _log_int(rng, 96, 1080), "batch": 0}
        size = rng.choice((96, 128, 250, 256, 512))
        return {"kind": kind, "width": size, "height": size - rng.choice((0, 0, 6)),
                "batch": rng.randint(1, 24 if size <= 256 else 6)}
    if kind == "train":
        crop = rng.choice((64, 96, 112, 128, 192, 256))
        return {"kind": kind, "crop": crop, "batch": rng.randint(1, 16)}
    if kind == "conv":
        cin = 16 * rng.randint(1, 18)
        cout = 16 * rng.randint(1, 10)
        height, width = _log_int(rng, 8, 272), _log_int(rng, 8, 480)
        batch = max(1, min(rng.choice((1, 2, 4, 8, 16)), int(6e9 / (cin * cout * height * width))))
        return {"kind": kind, "direction": rng.choice(("forward", "backward")), "batch": batch, "height": height,
                "width": width, "cin": cin, "cout": cout}
    if kind == "filter":
        return {"kind": kind, "filter": rng.choice(("svgf", "spatial")), "width": _log_int(rng, 96, 1920),
                "height": _log_int(rng, 96, 1080), "radius": rng.randint(1, 3), "iterations": rng.randint(1, 5)}
    return {"kind": "adam", "step": rng.randint(1, 20000)}


# ------------------------------------------------------------ path tracing --
@functools.lru_cache(maxsize=None)
def _open_scene(name, detail):
    """The compiled scene of a render case (host arrays), opened once as a
    program opens a scene file; views of it differ by camera and seed."""
    if name == "spheres":
        wl = scenes.spheres_large(subdivisions=detail)
    elif name == "volume":
        wl = scenes.sdf_spheres(resolution=detail)
    elif name == "materials":
        wl = scenes.material_zoo()
    else:
        wl = scenes.cornell_small()
    return wl, compile_scene(wl.scene)


def _view(camera, rng):
    """The scene's camera, moved a little."""
    jitter = rng.uniform(-1.0, 1.0, 3)
    distance = float(np.linalg.norm(np.asarray(camera.origin, np.float64) - np.asarray(camera.target, np.float64)))
    origin = tuple(float(p + 0.06 * distance * j) for p, j in zip(camera.origin, jitter))
    return dataclasses.replace(camera, origin=origin)


class _Render:
    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        wl, build = _open_scene(case["scene"], case.get("detail", 0))
        if wl.scene.environment.texture is not None:
            build = dataclasses.replace(build, environment_rotation_y=float(rng.uniform(0.0, 2.0 * math.pi)))
        settings = dataclasses.replace(wl.settings, width=case["width"], height=case["height"],
                                       frame_seed=int(rng.integers(1, 2 ** 31)))
        renderer = DenrimRenderer(0)
        scene = dataclasses.replace(wl.scene, camera=_view(wl.scene.camera, rng))
        self.session = renderer.make_session(scene, settings, build=build)
        self.spp = case["spp"]
        self.planes = [torch.empty(case["height"], case["width"], 4, device="cuda") for _ in AOVS]

    def run(self):
        self.session.reset_accumulation()
        self.session.render(self.spp)
        return {kind.name.lower(): self.session.copy_output(kind, plane) for kind, plane in zip(AOVS, self.planes)}


class _Viewport:
    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        wl, build = _open_scene("materials", 0)
        quality = RenderQuality.PREVIEW if case["quality"] == "preview" else RenderQuality.INTERACTIVE
        settings = RenderSettings(width=case["width"], height=case["height"], max_bounces=wl.settings.max_bounces,
                                  quality=quality)
        self.cameras = [_view(wl.scene.camera, rng) for _ in range(2)]
        scene = dataclasses.replace(wl.scene, camera=self.cameras[0])
        self.session = DenrimRenderer(0).make_session(scene, settings, build=build)

    def run(self):
        self.session.update_camera(self.cameras[1], previous_camera=self.cameras[0])
        self.session.render(1)
        return self.session.rgba8()


class _Serve:
    SIZES = ((96, 10), (256, 6), (512, 3), (1024, 1))  # of every 20 jobs

    @classmethod
    def plan(cls, case):
        """(size, samples) of every job: the serving configuration's shares of
        sizes, sample counts 16 / 64 in turn."""
        sizes = [size for size, share in cls.SIZES for _ in range(share)]
        order = [sizes[(7 * i) % len(sizes)] for i in range(case["jobs"])]
        return [(size, 16 if size == 1024 or i % 2 else case["spp_max"]) for i, size in enumerate(order)]

    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        scene, build = _preview_scene()
        self.server = RenderServer(build, ServerConfig(max_resident_jobs=256))
        families = list(FAMILIES)
        self.jobs = []
        for size, samples in self.plan(case):
            names = FAMILIES[families[int(rng.integers(0, len(families)))]]
            table = build.materials.copy()
            table[1] = PRESETS[names[int(rng.integers(0, len(names)))]].gpu_material()
            settings = RenderSettings(width=size, height=size, max_bounces=8, quality=RenderQuality.FINAL,
                                      frame_seed=int(rng.integers(1, 2 ** 31)))
            self.jobs.append((settings, _view(scene.camera, rng), samples, table))

    def run(self):
        ids = [self.server.submit(*job) for job in self.jobs]
        while self.server.step():
            pass
        images = {}
        for size in sorted({job[0].width for job in self.jobs}):
            same = [i for i, job in zip(ids, self.jobs) if job[0].width == size]
            out = torch.empty(len(same), size, size, 4, device="cuda")
            images[str(size)] = self.server.copy_outputs(same, RenderOutput.BEAUTY, out)
        for i in ids:
            self.server.release(i)
        return images


@functools.lru_cache(maxsize=None)
def _preview_scene():
    scene = scenes.material_preview()
    return scene, compile_scene(scene)


# --------------------------------------------------------------- denoising --
def _planes(batch, height, width, seed):
    """Beauty (noisy, long-tailed), albedo, encoded normal, depth and target
    planes of smooth seeded surfaces with edges, (batch, height, width, 4)."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    y = torch.arange(height, device="cuda").view(1, -1, 1) / height
    x = torch.arange(width, device="cuda").view(1, 1, -1) / width
    k = rand(batch, 1, 1, 8) * 12.0
    wave = torch.sin(k[..., 0] * x + k[..., 1] * y) + torch.cos(k[..., 2] * x - k[..., 3] * y)
    surface = torch.floor(wave * 1.5)  # which surface a pixel sees: constant regions with edges
    ones = torch.ones(batch, height, width, device="cuda")
    depth = torch.stack([2.0 + surface + 0.3 * wave, ones, ones, ones], -1).abs()
    nx, ny = 0.4 * torch.sin(surface * 2.1), 0.4 * torch.cos(surface * 1.7)
    nz = torch.sqrt((1.0 - nx * nx - ny * ny).clamp(min=0.0))
    normal = torch.stack([nx * 0.5 + 0.5, ny * 0.5 + 0.5, nz * 0.5 + 0.5, ones], -1)
    albedo = torch.stack([0.5 + 0.4 * torch.sin(surface + c) for c in (0.0, 2.0, 4.0)] + [ones], -1)
    clean = albedo * (0.6 + 0.4 * torch.cos(4.0 * x + 3.0 * y))[..., None]
    noise = -torch.log(rand(batch, height, width, 1).clamp(min=1e-6))
    beauty = clean * noise
    beauty[..., 3] = 1.0
    clean[..., 3] = 1.0
    return [t.contiguous() for t in (beauty, albedo, normal, depth, clean)]


class _Denoise:
    def __init__(self, case, seed):
        self.net = UNet(seed=seed)
        self.case = case
        n = max(1, case["batch"])
        planes = _planes(n, case["height"], case["width"], seed)[:4]
        self.planes = planes if case["batch"] else [p[0] for p in planes]
        self.out = torch.empty_like(self.planes[0])

    def run(self):
        call = self.net.denoise_batch if self.case["batch"] else self.net.denoise
        call(*self.planes, self.case["width"], self.case["height"], self.out)
        return self.out


class _Train:
    def __init__(self, case, seed):
        self.net = UNet(seed=seed)
        self.n, self.crop = case["batch"], case["crop"]
        self.planes = _planes(self.n, self.crop, self.crop, seed)
        self.net.grad_buffers(self.n, self.crop, self.crop)

    def run(self):
        net, n, s = self.net, self.n, self.crop
        beauty, albedo, normal, depth, target = self.planes
        buffers = net.grad_buffers(n, s, s)
        for j in range(n):
            net.pack(beauty[j], albedo[j], normal[j], depth[j], s, s, 0, 0, n, s, s, j)
        net.zero_grad()
        buffers["loss"].zero_()
        net.forward(n, s, s)
        net.loss(target, n, s, s)
        net.backward(n, s, s)
        return {"loss": buffers["loss"], "weights": {l.name: l.gw for l in net.layers},
                "biases": {l.name: l.gb for l in net.layers}}


class _Adam:
    def __init__(self, case, seed):
        self.net = UNet(seed=seed)
        self.net.step_count = case["step"] - 1
        g = torch.Generator(device="cuda").manual_seed(seed)
        for l in self.net.layers:
            for grad, mean, square in ((l.gw, l.mw, l.vw), (l.gb, l.mb, l.vb)):
                grad.copy_(torch.randn(grad.shape, generator=g, device="cuda") * 1e-3)
                if case["step"] > 1:
                    mean.copy_(torch.randn(grad.shape, generator=g, device="cuda") * 3e-4)
                    square.copy_(torch.rand(grad.shape, generator=g, device="cuda") * 1e-6)

    def run(self):
        self.net.adam()
        return {l.name: [l.w, l.b, l.vw] for l in self.net.layers}


class _Conv:
    def __init__(self, case, seed):
        self.lib = library.load()
        self.case = case
        n, h, w, cin, cout = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
        self.pixels = n * h * w
        self.x, self.act, self.gout, master, self.bias = _conv_inputs(case, seed)
        bf = dict(dtype=torch.bfloat16, device="cuda")
        self.weight, self.flipped = torch.empty(cout, 9, cin, **bf), torch.empty(cin, 9, cout, **bf)
        library.check(self.lib.dk_unet_weights_to_bf16(master.data_ptr(), master.numel(), self.weight.data_ptr(),
                                                       self.flipped.data_ptr(), cout, cin, None))
        self.out = torch.empty(n, h, w, cout, **bf)
        self.dpre = torch.empty(n, h, w, cout, **bf)
        self.gin = torch.empty(n, h, w, cin, **bf)
        self.gw, self.gb = torch.zeros(cout, 9, cin, device="cuda"), torch.zeros(cout, device="cuda")

    def run(self):
        c, lib = self.case, self.lib
        n, h, w, cin, cout = (c[k] for k in ("batch", "height", "width", "cin", "cout"))
        if c["direction"] == "forward":
            library.check(lib.dk_unet_conv3x3(self.x.data_ptr(), n, h, w, cin, cin, self.weight.data_ptr(),
                                              self.bias.data_ptr(), cout, self.out.data_ptr(), cout, 0, 1, 0, None))
            return self.out
        self.gw.zero_()
        self.gb.zero_()
        library.check(lib.dk_unet_relu_backward(self.act.data_ptr(), cout, self.gout.data_ptr(), cout,
                                                self.dpre.data_ptr(), cout, cout, self.pixels, None))
        library.check(lib.dk_unet_conv3x3_wgrad(self.x.data_ptr(), cin, self.dpre.data_ptr(), cout, n, h, w, cin,
                                                cout, self.gw.data_ptr(), None))
        library.check(lib.dk_unet_bias_grad(self.dpre.data_ptr(), cout, cout, self.pixels, self.gb.data_ptr(), None))
        library.check(lib.dk_unet_conv3x3(self.dpre.data_ptr(), n, h, w, cout, cout, self.flipped.data_ptr(), None,
                                          cin, self.gin.data_ptr(), cin, 0, 0, 0, None))
        return {"weight": self.gw, "bias": self.gb, "input": self.gin}


def _conv_inputs(case, seed):
    """Input activations, the layer's own output (its ReLU mask), the output's
    gradient, FP32 weights and bias."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, h, w, cin, cout = (case[k] for k in ("batch", "height", "width", "cin", "cout"))

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    x = randn(n, h, w, cin).relu().to(torch.bfloat16)
    act = randn(n, h, w, cout).relu().to(torch.bfloat16)
    gout = (randn(n, h, w, cout) * 1e-4).to(torch.bfloat16)
    master = randn(cout, 9, cin) * math.sqrt(2.0 / (9 * cin))
    bias = randn(cout) * 0.1
    return x, act, gout, master, bias


# ----------------------------------------------------------------- filters --
class _Filter:
    def __init__(self, case, seed):
        self.case = case
        w, h = case["width"], case["height"]
        self.beauty, self.albedo, self.normal, self.depth, _ = (p[0] for p in _planes(1, h, w, seed))
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        pan = torch.rand(2, generator=g, device="cuda") * 3.0 - 1.5  # pixels since the previous frame
        self.motion = torch.zeros(h, w, 4, device="cuda")
        self.motion[..., :2] = pan
        self.motion[..., 3] = 1.0
        self.out = torch.empty(h, w, 4, device="cuda")
        if case["filter"] == "svgf":
            self.svgf = SvgfDenoiser(w, h)
            for _ in range(5):  # a running history
                self._svgf()

    def _svgf(self):
        self.svgf.denoise(self.beauty, self.depth, self.normal, self.motion, self.out, radius=self.case["radius"],
                          iterations=self.case["iterations"])

    def run(self):
        if self.case["filter"] == "svgf":
            self._svgf()
        else:
            spatial_denoise(self.beauty, self.depth, self.normal, self.albedo, self.out, self.case["width"],
                            self.case["height"], radius=self.case["radius"], iterations=self.case["iterations"])
        return self.out


KINDS = {"render": _Render, "viewport": _Viewport, "serve": _Serve, "denoise": _Denoise, "train": _Train,
         "adam": _Adam, "conv": _Conv, "filter": _Filter}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work --
# Lower bounds: every input read once, every output written once; for a path
# the arithmetic of its camera ray, one traversal to a leaf and one surface
# evaluation.
PATH_FLOPS = 1000.0


def _parameters():
    return sum(l.count + l.cout for l in layer_plan())


def work(case):
    kind = case["kind"]
    if kind == "render":
        pixels = case["width"] * case["height"]
        data = 0.0
        if case["scene"] == "spheres":
            data = 64 * 20 * 4 ** case["detail"] * 48.0 + 2048 * 1024 * 16.0
        elif case["scene"] == "volume":
            data = 0.03 * case["detail"] ** 3 * 2.0  # the 3 % of samples in occupied bricks
        return {"bytes": pixels * 16.0 * len(AOVS) + data, "flops": pixels * case["spp"] * PATH_FLOPS}
    if kind == "viewport":
        pixels = case["width"] * case["height"]
        return {"bytes": pixels * 4.0, "flops": pixels * PATH_FLOPS}
    if kind == "serve":
        jobs = _Serve.plan(case)
        return {"bytes": sum(s * s * 16.0 for s, _ in jobs), "flops": sum(s * s * n * PATH_FLOPS for s, n in jobs)}
    if kind in ("denoise", "train"):
        n = max(1, case["batch"])
        w, h = (case["crop"], case["crop"]) if kind == "train" else (case["width"], case["height"])
        pixels, weights = n * w * h, 2.0 * _parameters()
        if kind == "denoise":
            return {"bytes": pixels * 5 * 16.0 + weights, "flops": pixels * flops_per_pixel()}
        first = 2.0 * 9 * layer_plan()[0].cin * LEVELS[0]  # the first layer has no input gradient
        return {"bytes": pixels * 5 * 16.0 + 3 * weights, "flops": pixels * (3.0 * flops_per_pixel() - first)}
    if kind == "adam":
        n = _parameters()
        return {"bytes": n * (4 * 4 + 3 * 4.0) + (n * 4.0), "flops": n * 15.0}
    if kind == "conv":
        pixels = case["batch"] * case["height"] * case["width"]
        one = 2.0 * 9 * case["cin"] * case["cout"] * pixels
        if case["direction"] == "forward":
            return {"bytes": pixels * 2.0 * (case["cin"] + case["cout"]) + 18.0 * case["cin"] * case["cout"],
                    "flops": one}
        return {"bytes": pixels * 2.0 * (2 * case["cin"] + 2 * case["cout"]) + 54.0 * case["cin"] * case["cout"],
                "flops": 2.0 * one}
    pixels = case["width"] * case["height"]
    taps = (2 * case["radius"] + 1) ** 2
    history = 6 * 16.0 if case["filter"] == "svgf" else 0.0
    return {"bytes": pixels * (5 * 16.0 + history), "flops": pixels * taps * case["iterations"] * 30.0}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    if case["kind"] == "adam":
        net = _Adam(case, seed).net
        b1, b2, lr, eps, step = 0.9, 0.999, 1e-3, 1e-8, case["step"]
        result = {}
        for l in net.layers:
            new = []
            for value, grad, mean, square in ((l.w, l.gw, l.mw, l.vw), (l.b, l.gb, l.mb, l.vb)):
                g = grad.double()
                m = b1 * mean.double() + (1.0 - b1) * g
                v = b2 * square.double() + (1.0 - b2) * g * g
                new.append((value.double() - lr * (m / (1.0 - b1 ** step)) / (torch.sqrt(v / (1.0 - b2 ** step)) + eps),
                            v))
            result[l.name] = [new[0][0], new[1][0], new[0][1]]
        return result
    if case["kind"] == "conv":
        x, act, gout, master, bias = _conv_inputs(case, seed)
        n, h, w, cin, cout = (case[k] for k in ("batch", "height", "width", "cin", "cout"))
        weight = master.to(torch.bfloat16).double().view(cout, 3, 3, cin)

        def padded(t):
            return torch.nn.functional.pad(t, (0, 0, 1, 1, 1, 1))

        if case["direction"] == "forward":
            p, out = padded(x), torch.zeros(n, h, w, cout, dtype=torch.float64, device="cuda")
            for dy in range(3):
                for dx in range(3):
                    out += p[:, dy:dy + h, dx:dx + w].double() @ weight[:, dy, dx].T
            return (out + bias.double()).clamp(min=0.0)
        g = torch.where(act > 0, gout, torch.zeros_like(gout))
        flat = g.double().reshape(-1, cout)
        p, q = padded(x), padded(g)
        gw = torch.empty(cout, 3, 3, cin, dtype=torch.float64, device="cuda")
        gin = torch.zeros(n, h, w, cin, dtype=torch.float64, device="cuda")
        for dy in range(3):
            for dx in range(3):
                gw[:, dy, dx] = flat.T @ p[:, dy:dy + h, dx:dx + w].double().reshape(-1, cin)
                gin += q[:, 2 - dy:2 - dy + h, 2 - dx:2 - dx + w].double() @ weight[:, dy, dx]
        return {"weight": gw.view(cout, 9, cin), "bias": flat.sum(0), "input": gin}
    return None
