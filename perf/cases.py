"""Performance cases of the renderer: what a program has it do, through its public entry points.

A case is a dict of plain values.  `prepare` makes what the program holds
before the call (the scene, a renderer or batch, a film buffer), `run` is one
pass, `work` what the pass cannot do without and `exact` its value in 64 bits
where that can be computed.

  frame    one progressive frame from the reference's Uniforms and its
           normalised RGBA image on the host (the interactive viewer)
  render   `spp` samples of every pixel (the film to the host, left on the
           device, or in double precision)
  noalloc  samples added to a caller-owned device film without allocating
  open     a scene built from host arrays and its first frame
  batch    many scenes and views in one launch
  train    a render that trains the path guide from scratch
  guided   a render that samples from a trained guide
  readout  the film normalised and tonemapped to host memory
"""
from __future__ import annotations

import math

import numpy as np
import torch

from raymond_b200 import _abi, api, scenes
from raymond_b200._abi import SceneDesc

MODES = {"bsdf": _abi.SAMPLING_BSDF, "nee": _abi.SAMPLING_NEE, "mis": _abi.SAMPLING_MIS}
RNGS = {"pcg": _abi.RNG_PCG32, "tea": _abi.RNG_TEA}
TONEMAPS = {"linear": _abi.TONEMAP_LINEAR, "hable": _abi.TONEMAP_HABLE, "aces": _abi.TONEMAP_ACES}

_contexts: dict[str, api.Context] = {}


def _context(builder: str) -> api.Context:
    """One context per BVH builder for the whole program."""
    if builder not in _contexts:
        _contexts[builder] = api.Context(torch.cuda.current_device(), bvh_builder=builder)
    return _contexts[builder]


def listed() -> list[dict]:
    return [
        # the interactive viewer's frame after a change: one sample, cleared film, tonemapped to the window;
        # the smallest call, every light type in the scene
        {"name": "frame_lights_192x108", "kind": "frame", "scene": "lights", "width": 192, "height": 108, "depth": 8,
         "mode": "mis", "tonemap": "hable"},
        # a plug-in whose host owns all device memory: a real-time preview into its film
        {"name": "noalloc_terrain_640x360", "kind": "noalloc", "scene": "terrain", "subdivisions": 3, "cells": 128,
         "width": 640, "height": 360, "spp": 1, "depth": 8},
        # the reference's Cornell configuration: 256 x 256, 16 spp, read back normalised
        {"name": "cornell_256_16spp", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "mode": "mis", "rng": "pcg", "film": "host"},
        # an odd-sized accumulation in double precision with light sampling only and the reference's generator
        {"name": "lights_401x233_nee_fp64", "kind": "render", "scene": "lights", "width": 401, "height": 233, "spp": 5,
         "depth": 6, "mode": "nee", "rng": "tea", "film": "fp64"},
        # one full-HD progressive frame of the large scene, kept on the device (a denoiser reads it there)
        {"name": "terrain_1080p_1spp", "kind": "render", "scene": "terrain", "subdivisions": 5, "cells": 512,
         "width": 1920, "height": 1080, "spp": 1, "depth": 12, "mode": "mis", "rng": "pcg", "film": "device"},
        # the throughput benchmark: 64 spp of the same frame with saved launch choices, read back
        {"name": "terrain_1080p_64spp_tuned", "kind": "render", "scene": "terrain", "subdivisions": 5, "cells": 512,
         "width": 1920, "height": 1080, "spp": 64, "depth": 12, "mode": "mis", "rng": "pcg", "film": "host",
         "tuned": True},
        # a chunk of the glossy room (deep paths, no direct light but a window), launch choices as created
        {"name": "room_720p_32spp", "kind": "render", "scene": "room", "width": 1280, "height": 720, "spp": 32,
         "depth": 16, "mode": "mis", "rng": "pcg", "film": "device"},
        # the guide's training: its network from scratch on the room's light and path records
        {"name": "room_640x360_train", "kind": "train", "scene": "room", "width": 640, "height": 360, "spp": 16,
         "depth": 16},
        # sampling from a trained guide
        {"name": "cornell_192_guided", "kind": "guided", "scene": "cornell", "width": 192, "height": 192, "spp": 512,
         "depth": 8},
        # several scenes and views of different sizes as one launch
        {"name": "batch_12_views", "kind": "batch", "views": 12, "width": 480, "height": 270, "spp": 4, "depth": 10,
         "graph": True},
        # opening the large scene (geometry, BVH on the device, materials, lights) to its first image
        {"name": "open_terrain_first_frame", "kind": "open", "scene": "terrain", "subdivisions": 5, "cells": 512,
         "width": 1280, "height": 720, "spp": 1, "depth": 8, "builder": "gpu"},
        # the finished 4K film, tonemapped to host memory
        {"name": "readout_4k_aces", "kind": "readout", "width": 3840, "height": 2160, "tonemap": "aces"},
    ]


def _log_uniform(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["frame", "noalloc", "render", "render", "render", "open", "batch", "train", "guided", "readout"])
    width = _log_uniform(rng, 97, 1920)
    height = max(64, min(1080, int(width * rng.uniform(0.5, 1.0))))
    pixels = width * height
    depth = rng.randint(2, 16)
    scene = rng.choice(["lights", "cornell", "terrain", "terrain", "room"])
    case: dict = {"kind": kind, "scene": scene, "width": width, "height": height, "depth": depth}
    if kind in ("noalloc", "open") and scene == "room":
        case["scene"] = scene = "terrain"
    if scene == "terrain":
        case.update(subdivisions=rng.randint(2, 5), cells=_log_uniform(rng, 24, 512))
    if kind == "frame":
        case.update(mode=rng.choice(["bsdf", "nee", "mis"]), tonemap=rng.choice(["linear", "hable", "aces"]))
    elif kind == "noalloc":
        case.update(spp=rng.randint(1, max(1, min(8, 400_000 // pixels))))
    elif kind == "render":
        case.update(spp=_log_uniform(rng, 1, max(1.01, min(64, 40_000_000 / pixels))), mode=rng.choice(["bsdf", "nee", "mis", "mis"]),
                    rng=rng.choice(["pcg", "pcg", "tea"]), film=rng.choice(["host", "device", "fp64"]))
    elif kind == "open":
        case.update(spp=1, builder=rng.choice(["gpu", "gpu", "host"]))
    elif kind == "batch":
        case = {"kind": "batch", "views": rng.randint(2, 16), "width": min(width, 640), "height": min(height, 400),
                "spp": rng.randint(1, 6), "depth": depth, "graph": rng.random() < 0.8}
    elif kind == "train":
        case.update(scene="room", width=rng.randint(320, 800), height=rng.randint(200, 450), spp=rng.randint(8, 16),
                    depth=rng.randint(6, 16))
        case.pop("subdivisions", None), case.pop("cells", None)
    elif kind == "guided":
        case.update(scene="cornell", width=rng.randint(128, 256), height=rng.randint(128, 256),
                    spp=rng.randint(384, 640), depth=rng.randint(4, 8))
        case.pop("subdivisions", None), case.pop("cells", None)
    else:
        case = {"kind": "readout", "width": _log_uniform(rng, 97, 3840), "height": _log_uniform(rng, 64, 2160),
                "tonemap": rng.choice(["linear", "hable", "aces"])}
    return case


def _scene(case: dict, seed: int) -> dict:
    s = seed % (1 << 20)
    if case["scene"] == "cornell":
        return scenes.cornell(seed=s)
    if case["scene"] == "lights":
        return scenes.cornell_all_lights(seed=s)
    if case["scene"] == "room":
        return scenes.glossy_room(seed=s)
    return scenes.spheres_terrain(seed=s, subdivisions=case["subdivisions"], terrain_cells=case["cells"])


def _batch(case: dict, seed: int) -> tuple[list, list]:
    """Half the views on small terrains of different sizes, half on Cornell boxes."""
    s = seed % (1 << 20)
    n = case["views"]
    descs, views = [], []
    for i in range(n):
        if i % 2 == 0:
            descs.append(scenes.spheres_terrain(seed=s + i, subdivisions=2 + i % 3, terrain_cells=48 + 40 * (i % 4),
                                                envmap_exponent=4))
        else:
            descs.append(scenes.cornell(seed=s + i, envmap_exponent=4))
        scale = 0.5 + 0.25 * (i % 4)  # views from half to 1.25 times the case's size
        views.append({"scene": i, "width": max(32, int(case["width"] * scale)),
                      "height": max(32, int(case["height"] * scale))})
    return descs, views


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state: dict = {"case": case, "seed": seed}
    if kind == "readout":
        # a film in linear radiance as a render leaves it: RGB sums of 16 samples, most values below 1, a few bright
        scene = api.Scene(_context("host"), scenes.cornell(seed=1, envmap_exponent=4))
        r = api.Renderer(scene, case["width"], case["height"], pool_size=1 << 16)
        r.film_tensor().copy_(_film_values(case, seed).to("cuda", torch.float32))
        r.set_samples(16)
        torch.cuda.synchronize()
        state.update(renderer=r, out=_pinned(case))
        return state
    if kind == "batch":
        descs, views = _batch(case, seed)
        state["batch"] = api.Batch(_context("host"), descs, views, graph=case["graph"])
        state["views"] = len(views)
        return state
    desc = SceneDesc(_scene(case, seed))
    state["desc"] = desc
    if kind == "open":
        return state
    scene = api.Scene(_context("host"), desc)
    if kind == "noalloc":
        state.update(scene=scene, film=torch.zeros(case["height"], case["width"], 4, device="cuda"))
        torch.cuda.synchronize()
        return state
    r = api.Renderer(scene, case["width"], case["height"])
    if case.get("tuned"):  # what the autotuner chose for this workload, saved
        r.set_tuning({"shade_min_blocks": 16, "trace_blocks_per_sm": 12, "pool_size": 1 << 23})
    if kind == "guided":  # train online, then keep the network
        r.set_guide(sampling=True, training=True, reset=True, seed=seed & 0xFFFF, batch_size=1 << 19)
        r.render(spp=128, max_depth=case["depth"], seed=seed)
        r.set_guide(sampling=True, training=False)
    state.update(renderer=r)
    if case.get("film") == "host":
        state["out"] = _pinned(case)
    return state


def _pinned(case: dict) -> np.ndarray:
    return torch.empty(case["height"], case["width"], 3, pin_memory=True).numpy()


def _film_values(case: dict, seed: int) -> torch.Tensor:
    g = torch.Generator().manual_seed(seed)
    film = torch.rand(case["height"], case["width"], 4, generator=g)
    return (16.0 * film ** 4 * 8.0).to(torch.float32)


def run(state: dict):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "frame":
        r = state["renderer"]
        u = _abi.default_uniforms(accumulate=0, exposure=1.2, sampling_mode=MODES[case["mode"]],
                                  tonemapping=TONEMAPS[case["tonemap"]])
        r.render_frame(u, max_depth=case["depth"])
        return r.film_normalize(u)
    if kind == "noalloc":
        state["film"].zero_()
        torch.cuda.current_stream().synchronize()  # the library renders on its own stream
        api.render_noalloc(state["scene"], state["desc"].scene["camera"], case["width"], case["height"],
                           state["film"].data_ptr(), spp=case["spp"], first_sample=0, max_depth=case["depth"])
        return state["film"]
    if kind == "batch":
        b = state["batch"]
        b.reset()
        b.render(spp=case["spp"], max_depth=case["depth"], first_sample=0)
        return [b.film(v, normalize=True) for v in range(state["views"])]
    if kind == "open":
        scene = api.Scene(_context(case["builder"]), state["desc"])
        r = api.Renderer(scene, case["width"], case["height"])
        r.render(spp=case["spp"], max_depth=case["depth"])
        return r.film(normalize=True)
    r = state["renderer"]
    if kind == "readout":
        return r.film(normalize=True, tonemapping=TONEMAPS[case["tonemap"]], exposure=1.2, out=state["out"])
    r.reset()
    if kind == "train":
        # a small learning rate and training batch, as fine tuning uses
        r.set_guide(sampling=False, training=True, reset=True, seed=1, batch_size=1 << 17, learning_rate=1e-4)
        r.render(spp=case["spp"], max_depth=case["depth"], first_sample=0)
        return {"film": _copy(r), "params": r.guide_params()}
    if kind == "guided":
        r.render(spp=case["spp"], max_depth=case["depth"], first_sample=0)
        return _copy(r)
    r.render(spp=case["spp"], max_depth=case["depth"], sampling_mode=MODES[case["mode"]], rng=RNGS[case["rng"]],
             first_sample=0, film_fp64=case["film"] == "fp64")
    if case["film"] == "fp64":
        return r.film64()
    if case["film"] == "host":
        return r.film(normalize=True, out=state["out"])
    return _copy(r)


def _copy(renderer: api.Renderer) -> torch.Tensor:
    """The film for later work on the device: film_tensor() aliases the renderer's own memory, which goes with it."""
    return renderer.film_tensor().clone()


def _triangles(case: dict) -> int:
    if case["scene"] == "terrain":
        return 64 * 5 * 4 ** case["subdivisions"] + 2 * case["cells"] ** 2
    return 197_490 if case["scene"] == "room" else 36


def work(case: dict) -> dict:
    """Bytes: the scene read once (vertices, normals, texcoords and indices of
    its triangles, about 60 B each) and the images written once.  Operations:
    per ray 11 nodes of 8 boxes (12 operations each) and 4 triangle tests of
    50; per shaded vertex 1,500 for material, light and BSDF sampling; rays
    and vertices per path from the scenes' mean path lengths."""
    pixels = case["width"] * case["height"]
    if case["kind"] == "readout":
        return {"bytes": pixels * (16 + 12), "flops": pixels * 40}
    if case["kind"] == "batch":
        n = case["views"]
        pixels = sum(max(32, int(case["width"] * (0.5 + 0.25 * (i % 4)))) * max(32, int(case["height"] * (0.5 + 0.25 * (i % 4))))
                     for i in range(n))
        triangles, vertices = 10_000 * n, 2.0
    else:
        triangles = _triangles(case)
        vertices = {"terrain": 0.75, "room": 5.0}.get(case["scene"], 2.5)
    vertices = min(vertices, case["depth"])
    rays = 1.0 + 2.0 * vertices
    paths = pixels * case.get("spp", 1)
    flops = paths * (rays * (11 * 8 * 12 + 4 * 50) + vertices * 1500)
    image = 24 if case.get("film") == "fp64" else 16
    if case["kind"] == "guided":
        flops += paths * vertices * 43_008
    if case["kind"] == "train":
        flops += 8 * (paths / (1 << 17)) * (1 << 13) * 129_000
    return {"bytes": triangles * 60 + pixels * image, "flops": flops}


def exact(case: dict, seed: int):
    """The read-out's arithmetic in 64 bits; a path-traced image has no such
    value that could be computed here (its paths follow the FP32 rounding)."""
    if case["kind"] != "readout":
        return None
    c = _film_values(case, seed).to(torch.float64).numpy()[..., :3] * 1.2 / 16.0
    if case["tonemap"] == "hable":
        def partial(x):
            return ((x * (0.15 * x + 0.05) + 0.004) / (x * (0.15 * x + 0.5) + 0.06)) - 0.02 / 0.3
        c = partial(2.0 * c) / partial(11.2)
    elif case["tonemap"] == "aces":
        c = np.clip((c * (2.51 * c + 0.03)) / (c * (2.43 * c + 0.59) + 0.14), 0.0, 1.0)
    return c
