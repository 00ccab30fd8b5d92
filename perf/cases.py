"""The workloads by which this framework's speed is followed.

Each case is a call that a user's program makes, through the public entry points, at the
sizes of this repository's configurations, tests and benchmark or at generic ones:

* ``frame``   one ``doVisualization``: buffer update, draw and (where asked for) readback;
* ``batch``   many views over several timesteps in one launch (``IsaacBatch``);
* ``infer``   the learned reconstructor on one half-size frame;
* ``train``   training steps of the reconstructor, then a read of its parameters;
* ``minmax``  the "minmax" request over every source;
* ``encode``  a rendered frame as the server's payload message.

``prepare`` makes what the program holds before the call (device fields, particles, the
visualization with its settings, the network), from the seed alone; ``run`` is one pass.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from isaac_b200 import IsaacVisualization, ParticleSource, VolumeSource, scenes
from isaac_b200.batch import IsaacBatch
from isaac_b200.protocol import FrameEncoder
from isaac_b200.recon import LAYER_SHAPES, WEIGHTS_COMBINED, Reconstructor, inference_flops

SLOPES = (-5.0 / 3.0, -2.0, -3.0, -11.0 / 3.0)
FINE_TUNING = 1.0e-5  # learning rate: trained weights on a new scene's pairs

# every setting of a frame case; a case names those that differ
FRAME = {
    "kind": "frame",
    "scene": "spectral",  # spectral: scalar fields; gaussian: scalar + curl; full: density, gradient, iso scalar
    "x": 128, "y": 128, "z": 128,
    "sources": 1,
    "w": 512, "h": 512,
    "step": 0.5,
    "interpolation": True,
    "renderer": "combined",
    "storage": 0,  # per-source bricks: 0 FP32, 1 BF16, 2 FP16
    "chain": "idem",  # functor chain of the scalar sources
    "guard": 0,  # ghost cells around every source
    "dither": 1,
    "particles": 0,
    "iso": False,
    "clips": 0,
    "ao": False,
    "advect": False,  # the curl field as an advected field source
    "readback": False,  # the frame as a host array, as the reference hands it out
}


def _frame(name: str, **settings) -> dict:
    return {"name": name, **FRAME, **settings}


def listed() -> list[dict]:
    return [
        # the smallest call: a coarse field shown as it is stepped, the frame on the host
        _frame("frame_tiny", x=32, y=32, z=32, w=200, h=150, interpolation=False, readback=True),
        # the first benchmark configuration: a scalar and a vector field, an ordinary window
        _frame("frame_small", scene="gaussian", x=128, y=128, z=128, w=512, h=512),
        # odd sizes with ghost cells, a functor chain, blue-noise dither and a clip plane:
        # a simulation's own local domain rather than a power of two
        _frame("frame_ragged", x=201, y=157, z=133, sources=3, w=1001, h=563, chain="mul(1.5)|add(-0.1)", guard=2, dither=3,
               clips=1, step=0.75),
        # the full-feature configuration: particles, iso surface, clip planes, SSAO
        _frame("frame_full_feature", scene="full", x=256, y=256, z=256, sources=3, w=1920, h=1080, particles=1_000_000,
               iso=True, clips=2, ao=True),
        # the headline configuration: four 512^3 sources to a full HD frame every timestep
        _frame("frame_headline", x=512, y=512, z=512, sources=4, w=1920, h=1080),
        # the same from BF16 bricks with the transfer functions applied per sample
        _frame("frame_per_source", x=512, y=512, z=512, sources=4, w=1920, h=1080, renderer="per_source", storage=1),
        # a vector field drawn by line integral convolution
        _frame("frame_advection", scene="gaussian", x=256, y=256, z=256, w=1280, h=720, advect=True),
        # several cameras and timesteps served together: every resolution of the batching
        # configuration once, over two timesteps
        {"name": "batch_views", "kind": "batch", "x": 512, "sources": 4, "timesteps": 2, "views": 8, "scale": 1.0},
        # the learned path: a half-size frame to full HD, and its training
        {"name": "recon_infer", "kind": "infer", "h": 540, "w": 960},
        {"name": "recon_train", "kind": "train", "h": 128, "w": 128, "batch": 16, "steps": 4, "pairs": 256},
        # the value ranges a user asks for before setting transfer functions
        {"name": "minmax_fields", "kind": "minmax", "x": 512, "y": 512, "z": 512, "sources": 2, "vector": True},
        # a frame for the streaming server
        {"name": "encode_frame", "kind": "encode", "w": 1920, "h": 1080, "quality": 90, "jpeg": True},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choices(["frame", "batch", "infer", "train", "minmax", "encode"], [10, 1, 2, 2, 2, 1])[0]
    if kind == "batch":
        return {"kind": kind, "x": _log(rng, 64, 400), "sources": rng.randint(1, 4), "timesteps": rng.randint(1, 3),
                "views": rng.randint(2, 8), "scale": rng.uniform(0.3, 1.0)}
    if kind == "infer":
        return {"kind": kind, "h": _log(rng, 60, 720), "w": _log(rng, 80, 1024)}
    if kind == "train":
        c = rng.choice([32, 48, 64, 96, 128])
        return {"kind": kind, "h": c, "w": c, "batch": rng.randint(2, 16), "steps": rng.randint(1, 4), "pairs": rng.randint(32, 256)}
    if kind == "minmax":
        x, y, z = (_log(rng, 16, 400) for _ in range(3))
        return {"kind": kind, "x": x, "y": y, "z": z, "sources": rng.randint(1, 3), "vector": rng.random() < 0.5}
    if kind == "encode":
        return {"kind": kind, "w": _log(rng, 64, 1920), "h": _log(rng, 48, 1080), "quality": rng.randint(50, 95),
                "jpeg": rng.random() < 0.8}
    n, w = _log(rng, 32, 320), _log(rng, 120, 1920)
    x, y, z = (int(n * rng.uniform(0.6, 1.4)) for _ in range(3))
    c = dict(FRAME, x=x, y=y, z=z, w=w, h=int(w / rng.uniform(1.0, 1.9)), step=rng.choice([0.5, 0.75, 1.0]),
             interpolation=rng.random() < 0.8, dither=rng.randint(0, 4), clips=rng.choice([0, 0, 1, 2]), readback=rng.random() < 0.3)
    what = rng.choice(["spectral", "spectral", "guarded", "per_source", "gaussian", "full", "advect"])
    if what in ("spectral", "guarded", "per_source"):
        c.update(sources=rng.randint(1, 4), chain=rng.choice(["idem", "idem", "mul(1.5)|add(-0.1)"]))
    if what == "guarded":
        c.update(guard=rng.randint(1, 4))
    if what == "per_source":
        c.update(renderer="per_source", storage=rng.randint(0, 2), chain="idem")
    if what == "gaussian":
        c.update(scene="gaussian")
    if what == "advect":
        c.update(scene="gaussian", advect=True)
    if what == "full":
        c.update(scene="full", sources=3, particles=_log(rng, 1000, 1_000_000), iso=True, ao=rng.random() < 0.5)
        c.update({a: min(c[a], 256) for a in "xyz"})
    return c


# ---------------------------------------------------------------------------- inputs
def _crop(field: torch.Tensor, c: dict) -> torch.Tensor:
    return field[: c["z"], : c["y"], : c["x"]].contiguous()


def _stretch(field: torch.Tensor, c: dict) -> torch.Tensor:
    """The whole cube's field on the case's box (the Gaussians may lie in any corner)."""
    for dim, a in enumerate("zyx"):
        n = field.shape[dim]
        if c[a] != n:
            field = field.index_select(dim, torch.arange(c[a], device=field.device) * n // c[a])
    return field.contiguous()


def _guarded(field: torch.Tensor, g: int) -> torch.Tensor:
    """The field with ``g`` ghost cells on every side, periodic as a simulation fills them."""
    if g == 0:
        return field
    dims = [torch.arange(-g, n + g, device=field.device) % n for n in field.shape[:3]]
    return field[dims[0][:, None, None], dims[1][None, :, None], dims[2][None, None, :]].contiguous()


def _spectral(c: dict, seed: int, count: int, shift: float = 0.0) -> list[torch.Tensor]:
    n = max(c["x"], c.get("y", 1), c.get("z", 1))
    seeds = [1000 * seed + 6 + i for i in range(count)]
    return scenes.precision_scene(n, seeds=seeds, slopes=SLOPES[:count], device="cuda", shift=shift)


def _image(h: int, w: int, count: int, seed: int) -> torch.Tensor:
    """Smooth RGBA8 images with soft edges, as a volume frame shows them: (count, h, w, 4)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.zeros((count, 4, h, w), device="cuda")
    for cells, amp in ((6, 0.5), (24, 0.3), (96, 0.12)):
        coarse = torch.rand((count, 4, cells, cells), generator=g, device="cuda")
        out += amp * torch.nn.functional.interpolate(coarse, size=(h, w), mode="bicubic", align_corners=False)
    out += 0.08 * torch.rand((count, 4, 1, 1), generator=g, device="cuda")
    alpha = ((out[:, 3:] - 0.25) * 2.0).clamp(0, 1)
    out[:, :3] *= alpha
    out[:, 3:] = alpha
    return (out.clamp(0, 1) * 255.0).to(torch.uint8).permute(0, 2, 3, 1).contiguous()


def _frame_state(c: dict, seed: int) -> dict:
    n = max(c["x"], c["y"], c["z"])
    functions, iso, transfer = [], [], []
    if c["scene"] == "gaussian":
        scalar, curl = scenes.gaussian_scene(n, seed=seed + 1, device="cuda")
        fields = [(scalar, 1), (curl, 3)]
        functions, iso = ["idem", "length"], [0.0, 0.0]
        transfer = [scenes.transfer_4point(0.3)] * 2
    elif c["scene"] == "full":
        dens, grad, s, p90 = scenes.density_gradient_scene(n, seeds=(3 * seed + 2, 3 * seed + 3, 3 * seed + 4), device="cuda")
        fields = [(dens, 1), (grad, 3), (s, 1)]
        functions = ["mul(2),add(1)", "length", "idem"]
        iso = [0.0, 0.0, 0.5 if c["iso"] else 0.0]
        k = min(max(int(round(p90 * 1024)), 2), 1022)
        transfer = [
            scenes.transfer_4point(0.2),
            scenes.transfer_4point(1.4),
            {0: (0.2, 0.6, 0.9, 0.0), k - 1: (0.2, 0.6, 0.9, 0.0), k: (0.9, 0.8, 0.2, 1.0), 1024: (0.9, 0.8, 0.2, 1.0)},
        ]
    else:
        fields = [(f, 1) for f in _spectral(c, seed, c["sources"])]
        functions = [c["chain"]] * len(fields)
        iso = [0.0] * len(fields)
        transfer = [scenes.transfer_4point(0.7 * i) for i in range(len(fields))]
    size = (c["x"], c["y"], c["z"])
    fit = _stretch if c["scene"] == "gaussian" else _crop
    volumes = [VolumeSource(f"src{i}", _guarded(fit(f, c), c["guard"]), feature_dim=fd, guard_size=c["guard"])
               for i, (f, fd) in enumerate(fields)]
    parts = []
    if c["particles"]:
        off, pos, attr = scenes.particles_uniform(c["particles"], size, seed=seed + 5, device="cuda")
        parts = [ParticleSource("particles", off, pos, attr, radius=0.25)]
        functions.append("length")
        transfer.append({0: (0.1, 0.3, 1.0, 1.0), 1024: (1.0, 0.2, 0.1, 1.0)})
    viz = IsaacVisualization("case", (c["w"], c["h"]), size, size, size if parts else (1, 1, 1), (0, 0, 0), volumes, parts)
    viz.functions = functions
    viz.updateFunctions()
    for i, points in enumerate(transfer):
        viz.setTransferPoints(i, points)
    for i, v in enumerate(iso):
        viz.setIsoThreshold(i, v)
    for i in range(c["clips"]):
        viz.addClipping(*((0.3, 0.0, 0.0, -1.0, 0.1, 0.0), (0.0, 0.0, -0.4, 0.2, 0.1, 1.0))[i])
    if c["ao"]:
        viz.setAmbientOcclusion(True, 0.5)
    if c["renderer"] == "per_source":
        viz.setRenderOptimization(False)
        for i in range(len(volumes)):
            viz.setStorage(i, c["storage"])
    if c["advect"]:
        viz.setFieldSource(1)
        viz.setAdvection(seed_points=1000)
    viz.setInterpolation(c["interpolation"])
    viz.setStep(c["step"])
    viz.setDitherMode(c["dither"])
    viz.setCamera(*scenes.camera(c["w"], c["h"], seed=seed + 3, distance=2.5))
    out = None if c["readback"] else torch.empty((c["h"], c["w"], 4), dtype=torch.uint8, device="cuda")
    return {"viz": viz, "out": out}


def _batch_state(c: dict, seed: int) -> dict:
    n = (c["x"],) * 3
    vis = []
    for t in range(c["timesteps"]):
        fields = _spectral(c, seed, c["sources"], shift=0.05 * t)
        viz = IsaacVisualization("step", (256, 256), n, n, (1, 1, 1), (0, 0, 0),
                                 [VolumeSource(f"src{i}", f) for i, f in enumerate(fields)])
        for i in range(len(fields)):
            viz.setTransferPoints(i, scenes.transfer_4point(0.7 * i))
        viz.setInterpolation(True)
        vis.append(viz)
    sizes = scenes.BATCH_RESOLUTIONS[::2][: c["views"]]
    sizes = [(max(8, int(w * c["scale"])), max(8, int(h * c["scale"]))) for w, h in sizes]
    views = scenes.batch_views(sizes, timesteps=c["timesteps"], seed0=100 + 31 * seed)
    return {"batch": IsaacBatch(vis, views)}


def _train_data(c: dict, seed: int) -> dict:
    high = _image(2 * c["h"], 2 * c["w"], c["pairs"], seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    low = high[:, ::2, ::2].to(torch.int16)
    low = (low + torch.randint(-2, 3, low.shape, generator=g, device="cuda", dtype=torch.int16)).clamp(0, 255).to(torch.uint8)
    index = torch.randint(0, c["pairs"], (c["steps"], c["batch"]), generator=g, device="cuda", dtype=torch.int32)
    return {"low": low.contiguous(), "high": high, "index": index}


def _minmax_fields(c: dict, seed: int) -> list[torch.Tensor]:
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (c["z"], c["y"], c["x"])
    fields = [torch.randn(shape, generator=g, device="cuda") * (1.0 + i) for i in range(c["sources"])]
    if c["vector"]:
        fields[-1] = torch.randn(shape + (3,), generator=g, device="cuda")
    return fields


def _minmax_state(c: dict, seed: int) -> dict:
    size = (c["x"], c["y"], c["z"])
    volumes = [VolumeSource(f"src{i}", f) for i, f in enumerate(_minmax_fields(c, seed))]
    viz = IsaacVisualization("case", (64, 64), size, size, (1, 1, 1), (0, 0, 0), volumes)
    viz.functions = ["length" if v.featureDim == 3 else "idem" for v in volumes]
    viz.updateFunctions()
    return {"viz": viz}


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    seed = seed % 1_000_003
    if kind == "frame":
        state = _frame_state(case, seed)
    elif kind == "batch":
        state = _batch_state(case, seed)
    elif kind == "infer":
        net = Reconstructor(1, case["h"], case["w"], seed=1)
        net.load(WEIGHTS_COMBINED)
        state = {"net": net, "low": _image(case["h"], case["w"], 1, seed)[0],
                 "out": torch.empty((2 * case["h"], 2 * case["w"], 4), dtype=torch.uint8, device="cuda")}
    elif kind == "train":
        net = Reconstructor(case["batch"], case["h"], case["w"], seed=1)
        net.load(WEIGHTS_COMBINED)
        state = {"net": net, **_train_data(case, seed)}
    elif kind == "minmax":
        state = _minmax_state(case, seed)
    else:
        # the message goes into the buffer that the program sends from
        state = {"encoder": FrameEncoder(case["quality"]), "frame": _image(case["h"], case["w"], 1, seed)[0], "jpeg": case["jpeg"],
                 "send": np.zeros(6 * case["h"] * case["w"] + 4096, dtype=np.uint8)}
    return {"kind": kind, **state}


def run(state: dict):
    kind = state["kind"]
    if kind == "frame":
        if state["out"] is None:
            return state["viz"].doVisualization()
        return state["viz"].doVisualization(host=False, out=state["out"])
    if kind == "batch":
        state["batch"].render(update=True)
        return state["batch"].frames
    if kind == "infer":
        return state["net"].infer(state["low"], state["out"])
    if kind == "train":
        for step in range(state["index"].shape[0]):
            loss = state["net"].train_step(state["low"], state["high"], state["index"][step], FINE_TUNING)
        return {"loss": loss, "params": state["net"].params()}
    if kind == "minmax":
        return list(state["viz"].minMax())
    message = state["encoder"].message(state["frame"], state["jpeg"])
    state["send"][: len(message)] = np.frombuffer(message, dtype=np.uint8)
    return {"bytes": len(message), "message": state["send"]}


# ---------------------------------------------------------------------------- work and exact results
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "frame":
        voxels = case["x"] * case["y"] * case["z"]
        floats = {"gaussian": 4, "full": 5}.get(case["scene"], case["sources"])
        pixels = case["w"] * case["h"]
        # about 0.6 of a frame's rays times the volume's depth in steps are samples; a
        # sample is 8 taps of 4 channels (of each source in the per-source renderer)
        samples = 0.6 * pixels * (voxels ** (1.0 / 3.0)) / case["step"]
        per = case["sources"] if case["renderer"] == "per_source" else 1
        channels = 1 if case["renderer"] == "per_source" else 4
        return {"bytes": 4 * floats * voxels + 16 * case["particles"] + 4 * pixels, "flops": samples * per * (16 * channels + 8)}
    if kind == "batch":
        sizes = scenes.BATCH_RESOLUTIONS[::2][: case["views"]]
        pixels = sum(int(w * case["scale"]) * int(h * case["scale"]) for w, h in sizes)
        return {"bytes": 4 * case["sources"] * case["timesteps"] * case["x"] ** 3 + 4 * pixels,
                "flops": 0.6 * pixels * case["x"] / 0.5 * 72}
    if kind == "infer":
        return {"bytes": 20 * case["h"] * case["w"], "flops": inference_flops(case["h"], case["w"])}
    if kind == "train":
        pixels = case["h"] * case["w"] * case["batch"] * case["steps"]
        return {"bytes": 20 * pixels + 28 * 216_464 * case["steps"],
                "flops": 3 * inference_flops(case["h"], case["w"]) * case["batch"] * case["steps"]}
    if kind == "minmax":
        floats = case["sources"] + (2 if case["vector"] else 0)
        return {"bytes": 4 * floats * case["x"] * case["y"] * case["z"], "flops": 0}
    return {"bytes": 5 * case["w"] * case["h"], "flops": 0}


def _unet_loss(params: torch.Tensor, low: torch.Tensor, high: torch.Tensor) -> torch.Tensor:
    """The reconstructor's loss in the parameters' precision: NCHW, plain torch."""
    F = torch.nn.functional
    layers, at = [], 0
    for k, _, _, ci, co, _ in LAYER_SHAPES:
        w = params[at : at + co * k * k * ci].reshape(co, k, k, ci).permute(0, 3, 1, 2)
        at += co * k * k * ci
        layers.append((w, params[at : at + co]))
        at += co

    def conv(i, x, relu=True):
        y = F.conv2d(x, *layers[i], stride=LAYER_SHAPES[i][1], padding=LAYER_SHAPES[i][2])
        return F.relu(y) if relu else y

    def cat(coarse, fine):
        iy = (torch.arange(fine.shape[2], device=fine.device) // 2).clamp(max=coarse.shape[2] - 1)
        ix = (torch.arange(fine.shape[3], device=fine.device) // 2).clamp(max=coarse.shape[3] - 1)
        return torch.cat([coarse[:, :, iy][:, :, :, ix], fine], 1)

    rgba = low.permute(0, 3, 1, 2).to(params.dtype) / 255.0
    e1b = conv(1, conv(0, torch.cat([rgba, torch.zeros_like(rgba)], 1)))
    e2 = conv(3, conv(2, e1b))
    d23 = conv(4, e2)
    u21 = conv(8, cat(conv(7, cat(conv(6, cat(conv(5, d23), d23)), e2)), e1b))
    r = conv(10, conv(9, u21), relu=False)
    b, _, h, w = r.shape
    residual = r.reshape(b, 2, 2, 4, h, w).permute(0, 3, 4, 1, 5, 2).reshape(b, 4, 2 * h, 2 * w)

    def double(x, dim):  # even pixels copy, odd ones average their neighbours
        n = x.shape[dim]
        nxt = x.index_select(dim, (torch.arange(n, device=x.device) + 1).clamp(max=n - 1))
        return torch.stack([x, 0.5 * (x + nxt)], dim + 1).flatten(dim, dim + 1)

    pred = double(double(rgba, 2), 3) + residual
    return ((pred - high.permute(0, 3, 1, 2).to(params.dtype) / 255.0) ** 2).mean()


def exact(case: dict, seed: int):
    """What ``run`` returns, in 64 bits, where it returns computed numbers (frames and
    messages are bytes)."""
    if case["kind"] == "minmax":
        fields = _minmax_fields(case, seed % 1_000_003)
        values = [torch.linalg.vector_norm(f.double(), dim=-1) if f.dim() == 4 else f.double() for f in fields]
        return [np.array([float(v.min()) for v in values]), np.array([float(v.max()) for v in values])]
    if case["kind"] == "train":
        s = _train_data(case, seed % 1_000_003)
        p = torch.from_numpy(np.fromfile(WEIGHTS_COMBINED, dtype=np.float32)).cuda().double().requires_grad_(True)
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        for t in range(case["steps"]):
            pick = s["index"][t].long()
            loss = _unet_loss(p, s["low"][pick], s["high"][pick])
            (g,) = torch.autograd.grad(loss, p)
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            step = (m / (1 - 0.9 ** (t + 1))) / ((v / (1 - 0.999 ** (t + 1))).sqrt() + 1e-8)
            p = (p - FINE_TUNING * step).detach().requires_grad_(True)
        return {"loss": loss.detach().reshape(1), "params": p.detach()}
    return None
