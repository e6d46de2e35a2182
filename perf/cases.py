"""What is timed of this framework: renders through its public entry points.

A case is one call (or one small burst of calls) that a program using the renderer makes on a
scene it has loaded: a pass of a progressive render into its film, a region of one, a tile for a
host that may not allocate, a denoiser's inputs beside the beauty film, a guided pass, a burst of
requests to the server.  The scenes are the repository's own workloads (``scenes.py``): the
Cornell box, the torus knot under a sky (Disney materials), the many-light scene with media and
subsurface, the instanced grid and the indirect-lit room.

``prepare`` hands over what such a program holds before the call: the scene on a device of its
own, a camera and a sampler seed (both from the case's seed) and an empty film.  Built scenes are
kept per process, as a program that loads a scene once and renders many views of it does.

A pass adds the next ``spp`` samples of each pixel to the state's film, so no two passes on a
state trace the same samples.

``exact`` gives nothing: a film is a sum over paths whose branches (light picked, lobe sampled,
roulette, surface hit) are decided by 32-bit comparisons, so evaluating the same samples in 64
bits follows other paths and is not the same quantity held more precisely.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

import pe_pkg

pe = pe_pkg.load()
scenes = importlib.import_module("photon_engine_b200.scenes")

# Per scene: depth of its workload, the largest camera orbit (degrees) that keeps the view on it,
# and per camera path its closest-hit rays, shadow rays, boxes and triangles tested per ray.
_KINDS = {
    "cornell": {"depth": 8, "orbit": 8.0, "closest": 3.5, "shadow": 2.5, "boxes": 20, "tris": 6},
    "knot": {"depth": 12, "orbit": 20.0, "closest": 2.1, "shadow": 1.0, "boxes": 32, "tris": 4},
    "media": {"depth": 24, "orbit": 10.0, "closest": 8.0, "shadow": 2.0, "boxes": 32, "tris": 5},
    "grid": {"depth": 12, "orbit": 8.0, "closest": 2.5, "shadow": 1.0, "boxes": 48, "tris": 5},
    "room": {"depth": 12, "orbit": 4.0, "closest": 5.0, "shadow": 4.0, "boxes": 36, "tris": 5},
}
_BOX_FLOPS, _TRI_FLOPS, _VERTEX_FLOPS = 21, 46, 900
_BYTES_PER_TRIANGLE, _BYTES_PER_TEXEL = 96, 20  # geometry, tree and shading data; image and its sampling tables

_loaded: dict = {}


def listed():
    return [
        # the smallest call: one 64×64 bucket of a host application's frame, in the host's own buffers
        {"name": "tile_knot_64x64", "call": "tile", "scene": "knot", "width": 1920, "height": 1080, "x0": 928, "y0": 508,
         "w": 64, "h": 64, "spp": 1},
        # interactive viewport: one sample per pixel of a small frame
        {"name": "cornell_256_1spp", "call": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 1},
        # the whole plain Cornell render
        {"name": "cornell_256_64spp", "call": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 64},
        # a preview request
        {"name": "knot_512_16spp", "call": "render", "scene": "knot", "width": 512, "height": 512, "spp": 16},
        # one batch of the full-HD knot frame, the headline workload
        {"name": "knot_1080p_4spp", "call": "render", "scene": "knot", "width": 1920, "height": 1080, "spp": 4},
        # a crop of a frame being looked at, odd in both sizes
        {"name": "knot_crop_333x217", "call": "region", "scene": "knot", "width": 1920, "height": 1080, "x0": 701, "y0": 433,
         "w": 333, "h": 217, "spp": 5},
        # full-HD batch of 5.2M instanced triangles (a top-level tree over shared meshes)
        {"name": "grid_1080p_2spp", "call": "render", "scene": "grid", "width": 1920, "height": 1080, "spp": 2},
        # many lights, glass, media and subsurface walks at the workload's depth of 24
        {"name": "media_720p_4spp", "call": "render", "scene": "media", "width": 1280, "height": 720, "spp": 4},
        # an interior lit through one window: long indirect paths
        {"name": "room_1080p_2spp", "call": "render", "scene": "room", "width": 1920, "height": 1080, "spp": 2},
        # beauty with the denoiser's albedo, normal and coverage films
        {"name": "knot_720p_aovs", "call": "render", "scene": "knot", "width": 1280, "height": 720, "spp": 2, "aovs": True},
        # guided sampling with a network the program holds (no further training)
        {"name": "room_guided_320x180", "call": "guided", "scene": "room", "width": 320, "height": 180, "spp": 16},
        # previews of two resident scenes arriving together at the request server
        {"name": "served_8_previews", "call": "served", "scene": "cornell", "second": "knot", "width": 512, "height": 512,
         "spp": 16, "requests": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Frame sizes from 40 to 1920 columns with any aspect between tall and wide, 1 to 64 samples,
    every call and scene of the list; never more camera paths than the listed case of its scene."""
    call = rng.choice(["tile", "render", "render", "render", "render", "region", "aovs", "adaptive", "guided", "served"])
    scene = rng.choice(["cornell", "knot", "knot", "media", "grid", "room"])
    most = {"cornell": 4_000_000, "knot": 8_000_000, "media": 3_600_000, "grid": 4_000_000, "room": 4_000_000}[scene]
    width = _log_int(rng, 40, 1920)
    height = max(24, min(1080, int(width * rng.uniform(0.4, 1.2))))
    spp = max(1, min(_log_int(rng, 1, 64), most // (width * height)))
    c = {"call": call, "scene": scene, "width": width, "height": height, "spp": spp}
    if call in ("tile", "region"):
        c["width"], c["height"] = 1920, 1080
        c["w"], c["h"] = (_log_int(rng, 16, 181), _log_int(rng, 16, 181)) if call == "tile" else \
            (_log_int(rng, 32, 1200), _log_int(rng, 32, 900))
        c["x0"], c["y0"] = rng.randint(0, 1920 - c["w"]), rng.randint(0, 1080 - c["h"])
        c["spp"] = max(1, min(_log_int(rng, 1, 32), most // (c["w"] * c["h"])))
    elif call == "aovs":
        c.update(call="render", aovs=True, spp=max(1, min(spp, 1_800_000 // (width * height))))
    elif call == "adaptive":
        c.update(call="render", adaptive=True, spp=max(1, min(rng.randint(17, 40), most // (width * height))))
    elif call == "guided":
        c.update(scene="room", spp=max(1, min(spp, 900_000 // (width * height))))
    elif call == "served":
        c.update(scene=rng.choice(["cornell", "grid"]), second="knot", width=min(width, 640), height=min(height, 640),
                 spp=rng.randint(1, 16), requests=rng.randint(2, 8))
    elif rng.random() < 0.3:
        c["lens"] = round(rng.uniform(0.01, 0.1), 3)  # a thin-lens camera
    return c


def _scene(kind: str):
    if kind not in _loaded:
        make = {"cornell": scenes.cornell_box, "knot": scenes.torus_knot_scene, "media": scenes.media_scene,
                "grid": scenes.instanced_grid_scene, "room": scenes.room_scene}[kind]
        scene, _, settings = make()
        scene.build_accelerator()
        _loaded[kind] = scene, settings
    return _loaded[kind]


def _view(kind: str, width: int, height: int, rng: random.Random, lens: float = 0.0):
    """The workload's camera orbited about its target by the seed's angle."""
    pos, target, up, fov = scenes.CAMERAS[kind]
    a = math.radians(rng.uniform(-1.0, 1.0) * _KINDS[kind]["orbit"])
    dx, dz = pos[0] - target[0], pos[2] - target[2]
    at = (target[0] + math.cos(a) * dx + math.sin(a) * dz, pos[1], target[2] - math.sin(a) * dx + math.cos(a) * dz)
    if lens > 0.0:
        return pe.ThinLensCamera(at, target, up, fov, width / height, lens, math.dist(at, target))
    return pe.PerspectiveCamera(at, target, up, fov, width / height)


def _settings(kind: str, case: dict, seed: int):
    base = _scene(kind)[1]
    return pe.RenderSettings(width=case["width"], height=case["height"], max_bounces=_KINDS[kind]["depth"],
                             filter_type=base.filter_type, filter_width=base.filter_width, seed=seed,
                             adaptive_sampling=bool(case.get("adaptive")), noise_threshold=0.05, min_adaptive_samples=16)


class _State(dict):
    """What the program holds; its server ends before its device does."""

    def __del__(self):
        for key in ("server", "device"):
            if key in self:
                self.pop(key).close()


def prepare(case: dict, seed: int):
    rng = random.Random(seed)
    kind = case["scene"]
    device = pe.create_device("cuda:0")
    state = _State(device=device, case=case, next=0)
    scene, _ = _scene(kind)
    if case["call"] == "served":
        server = pe.RenderServer(device, 32 << 30)
        state["server"] = server
        ids = [server.add_scene(scene), server.add_scene(_scene(case["second"])[0])]
        kinds = [kind, case["second"]]
        state["requests"] = [(ids[k % 2], _view(kinds[k % 2], case["width"], case["height"], rng),
                              _settings(kinds[k % 2], case, rng.randrange(1 << 31))) for k in range(case["requests"])]
        return state
    device.set_scene(scene)
    state["camera"] = _view(kind, case["width"], case["height"], rng, case.get("lens", 0.0))
    state["settings"] = _settings(kind, case, rng.randrange(1 << 31))
    if case["call"] == "tile":
        n = case["width"] * case["height"]
        state["tile"] = (torch.zeros(n, 3, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"),
                         torch.zeros(n, device="cuda"))
        return state
    state["film"] = pe.Film(case["width"], case["height"])
    if case.get("aovs"):
        state["aovs"] = pe.AovFilms(case["width"], case["height"])
    if case["call"] == "guided":
        pe._capi.check(pe._capi.load().pe_device_guide_reset(device.handle, rng.randrange(1 << 31), None, None))
        device.set_guiding(1, 0, 0.0)
    return state


def _arrays(film):
    return {"sum": film.sum, "count": film.count.view(np.int32), "sum_sq": film.sum_sq}


def run(state):
    case, device = state["case"], state["device"]
    spp = case["spp"]
    if case["call"] == "served":
        server = state["server"]
        ids = [server.submit(sid, camera, settings, spp) for sid, camera, settings in state["requests"]]
        films = []
        for rid in ids:
            server.wait(rid)
            films.append(_arrays(server.take(rid)))
        return films
    first = state["next"]
    state["next"] = first + spp
    if case["call"] == "tile":
        total, count, squares = state["tile"]
        device.render_tile_noalloc(state["camera"], state["settings"], case["x0"], case["y0"], case["w"], case["h"], first, spp,
                                   total.data_ptr(), count.data_ptr(), squares.data_ptr())
        return {"sum": total, "count": count, "sum_sq": squares}
    film = state["film"]
    if case["call"] == "region":
        device.render_region(state["camera"], state["settings"], film, (case["x0"], case["y0"], case["w"], case["h"]), first,
                             spp)
        return _arrays(film)
    aovs = state.get("aovs")
    device.render(state["camera"], state["settings"], pe.RenderTargets(beauty=film, aovs=aovs), first, spp)
    out = _arrays(film)
    if aovs is not None:
        out["albedo"], out["normal"], out["alpha"] = (_arrays(f) for f in (aovs.albedo, aovs.normal, aovs.alpha))
    return out


def _triangles(kind: str):
    return {"cornell": 36, "knot": 1_048_580, "media": 200_000, "grid": 262_146, "room": 545_000}[kind]


def work(case: dict):
    """Bytes: the scene's data read once, the film's pixels written on the device and added to the
    caller's (20 B each, read and written).  Flops: box, triangle and vertex arithmetic of the rays."""
    pixels = case.get("w", case["width"]) * case.get("h", case["height"])
    kinds = [case["scene"]] + ([case["second"]] if "second" in case else [])
    total_bytes, flops = 0.0, 0.0
    for kind in kinds:
        k = _KINDS[kind]
        texels = 0 if kind in ("cornell", "media") else 2048 * 1024
        total_bytes += _triangles(kind) * _BYTES_PER_TRIANGLE + texels * _BYTES_PER_TEXEL
        share = case.get("requests", 1) / len(kinds)
        rays = k["closest"] + k["shadow"]
        per_path = rays * (k["boxes"] * _BOX_FLOPS + k["tris"] * _TRI_FLOPS) + k["closest"] * _VERTEX_FLOPS
        flops += pixels * case["spp"] * share * per_path
        total_bytes += pixels * 20 * share * (3 if case["call"] != "served" else 1) * (4 if case.get("aovs") else 1)
    return {"bytes": total_bytes, "flops": flops}


def exact(case: dict, seed: int):
    return None
