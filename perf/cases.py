"""The renderer's work as its users call it, for timing: one pass per case.

Scenes are the repository's seeded puff recipes (fresh noise, camera azimuth
and sample streams for every seed), the phase table and the sky state are the
ones the tests and the benchmark use.  What a program keeps between calls (the
context with its uploaded scene and settings, output buffers, a batch) is made
by prepare(); a pass is one call of the public entry points.

Kinds of pass:
  frame          Renderer.render_tile_async into device buffers
  host           Renderer.render_tile into host buffers (the Blender addon's
                 call: the whole blocking call with its copies)
  shadow         Renderer.shadow_tile_async (the shadow pass)
  batch          Batch.launch, one CUDA graph over several fields and views
  adjoint        adjoint.render of several views, an L2 image loss, backward
  transmittance  dr_transmittance_noalloc on device rays
"""
import ctypes
import json
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "droplet-render_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "droplet-render_b200"))

from droplet_b200 import _native as N  # noqa: E402
from droplet_b200 import adjoint as AD  # noqa: E402
from droplet_b200 import camera as cam  # noqa: E402
from droplet_b200 import workloads as W  # noqa: E402
from droplet_b200.renderer import Batch, BatchView, PhaseTable, Renderer, RenderSettings, stream_handle  # noqa: E402
from droplet_b200.scene import build_from_dense, build_octree  # noqa: E402
from droplet_b200.sky import SkyState  # noqa: E402

# Launch shapes the autotuner chooses for the two large frames (kernel, blocks
# per SM, event batch, traversal, tile, visits, steps); "" is a context whose
# program never tunes, as the Blender module and the adjoint's do.
SHAPES = {"": None, "cumulus": (0, 8, 24, 2, 0, 3, 4), "slab": (0, 8, 16, 2, 0, 2, 4)}


def listed():
    base = {"scene": "puff", "n": 64, "w": 256, "h": 256, "x0": 0, "y0": 0, "tw": 256, "th": 256, "spp": 16,
            "sigma_t": 20.0, "albedo": 0.99, "events": 8, "phase": "mie", "env": "hosek", "depth": False,
            "occluders": False, "shape": ""}

    def c(name, kind, **k):
        return dict(base, name=name, kind=kind, **k)

    return [
        # one 64 x 64 tile of the addon's tiled render: the smallest blocking call
        c("addon tile", "host", n=128, w=640, h=360, x0=288, y0=148, tw=64, th=64),
        # the addon's viewport preview of a small cloud (config 0)
        c("preview", "frame"),
        # an odd region of a composited frame: depth texture, exact phase sampler, ragged sizes
        c("depth region", "frame", n=96, w=513, h=389, x0=41, y0=35, tw=333, th=217, spp=37, phase="exact",
          depth=True, events=32),
        # the reference's default build with its options on: HG phase, environment map, occluder meshes
        c("hg env occluders", "frame", n=128, w=640, h=360, tw=640, th=360, spp=32, sigma_t=40.0, events=64,
          phase="hg", env="map", occluders=True),
        # the headline frame (config 1), tuned
        c("cumulus frame", "frame", scene="cumulus", n=512, w=1920, h=1080, tw=1920, th=1080, spp=64, sigma_t=60.0,
          albedo=0.999, events=64, shape="cumulus"),
        # a final frame through the blocking host call of a program that never tunes
        c("cumulus host", "host", scene="cumulus", n=256, w=1280, h=720, tw=1280, th=720, spp=32, sigma_t=60.0,
          albedo=0.999, events=64),
        # the large sparse scene (config 4's slab): deep octree, mostly empty frame, many samples, tuned
        c("sparse slab", "frame", scene="slab", n=1024, w=1920, h=1080, tw=1920, th=1080, spp=256, sigma_t=100.0,
          events=128, shape="slab"),
        # the shadow pass over a frame's depth texture
        c("shadow pass", "shadow", scene="cumulus", n=256, w=960, h=540, tw=960, th=540, spp=16, depth=True,
          sigma_t=60.0, events=64),
        # many fields and views in one launch (config 2's ranges: fields to 256^3, sides 128-768, 16-256 spp)
        c("batch", "batch", fields=4, views=3, n=256, side=768, spp=64, sigma_t=45.0, events=500),
        # a contact sheet: many small views of small fields
        c("contact sheet", "batch", fields=4, views=8, n=64, side=128, spp=16, sigma_t=30.0, events=500),
        # one step of inverse rendering (config 3): forward and backward of 8 views
        c("inverse step", "adjoint", n=128, views=8, w=256, h=256, spp=32),
        # transmittance estimates along light rays for a host renderer that owns the memory
        c("transmittance", "transmittance", n=128, rays=4096, spp=2048, sigma_t=30.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "host", "host", "shadow", "batch", "adjoint", "transmittance"])
    scene = rng.choice(["puff", "puff", "cumulus", "slab"]) if kind in ("frame", "host", "shadow") else "puff"
    n = {"puff": lambda: rng.choice([64, 72, 96, 128, 200, 256]), "cumulus": lambda: rng.choice([128, 256, 384]),
         "slab": lambda: 1024}[scene]()
    w, h = int(_log(rng, 96, 1920)), int(_log(rng, 64, 1080))
    c = {"kind": kind, "scene": scene, "n": n, "w": w, "h": h, "x0": 0, "y0": 0, "tw": w, "th": h,
         "sigma_t": round(rng.uniform(10.0, 80.0), 1), "albedo": rng.choice([0.9, 0.99, 0.999]),
         "events": int(_log(rng, 4, 500)), "phase": "mie", "env": "hosek", "depth": False, "occluders": False,
         "shape": ""}
    # at most 2^25 path samples
    most = max(1, (1 << 25) // (w * h))
    c["spp"] = max(1, min(int(_log(rng, 1, 256)), most))
    if kind in ("frame", "host"):
        c["phase"] = rng.choice(["mie", "mie", "mie", "exact", "hg"])
        c["env"] = rng.choice(["hosek", "hosek", "hosek", "map", "none"])
        c["depth"] = rng.random() < 0.2
        c["occluders"] = rng.random() < 0.2
        c["shape"] = rng.choice(["", "", "cumulus", "slab"])
        if rng.random() < 0.3:  # a tile of the frame
            c["tw"], c["th"] = max(2, int(w * rng.uniform(0.1, 0.9))), max(2, int(h * rng.uniform(0.1, 0.9)))
            c["x0"], c["y0"] = rng.randrange(w - c["tw"] + 1), rng.randrange(h - c["th"] + 1)
    elif kind == "shadow":
        c["depth"] = True
    elif kind == "batch":
        c["fields"], c["views"] = rng.randint(1, 4), rng.randint(1, 8)
        c["side"] = int(_log(rng, 64, 512))
        c["spp"] = max(1, min(int(_log(rng, 4, 64)), (1 << 25) // (c["fields"] * c["views"] * c["side"] ** 2)))
    elif kind == "adjoint":
        c["n"], c["views"] = rng.choice([64, 96, 128]), rng.randint(1, 8)
        c["w"], c["h"] = int(_log(rng, 64, 384)), int(_log(rng, 64, 384))
        c["sigma_t"], c["albedo"], c["events"] = round(rng.uniform(10.0, 40.0), 1), 0.99, rng.randint(4, 16)
        c["spp"] = max(1, min(int(_log(rng, 4, 64)), (1 << 22) // (c["w"] * c["h"])))
    elif kind == "transmittance":
        c["rays"] = int(_log(rng, 16, 65536))
        c["spp"] = max(1, min(int(_log(rng, 64, 16384)), (1 << 24) // c["rays"]))
    return c


# ---- inputs --------------------------------------------------------------------
def _tables():
    golden = os.path.join(ROOT, "tests", "golden")
    z = np.load(os.path.join(golden, "mie_reference_table.npz"))
    with open(os.path.join(golden, "sky_states.json")) as f:
        sky = next(s for s in json.load(f) if s["note"] == "c0/c1 sun")
    return (PhaseTable(np.ascontiguousarray(z["pdf"], np.float32), np.ascontiguousarray(z["cdf"], np.float32)),
            SkyState(np.asarray(sky["configs"]), np.asarray(sky["radiances"])))


def _octree(scene, n, rng):
    """One of the repository's recipes with noise of its own for every seed."""
    s = int(rng.integers(1, 1 << 20))
    if scene == "puff":
        rec = W.config0_recipe(n, s)
    elif scene == "cumulus":
        rec = W.cumulus_recipe(n)
        for i, p in enumerate(rec.puffs):
            p.seed = s + i
    else:
        rec = W.slab_recipe(n)
        for i, p in enumerate(rec.puffs):
            p.seed = s + i
    org, vals = W.sparse_field_puffwise(rec)
    return build_octree(org, vals, rec.voxel_size, 12)


def _settings(case, rng, phase, sky, w, h, azimuth=None, **more):
    ss, sa, ev = W.medium_of(case["sigma_t"], case["albedo"], case["events"])
    az = float(rng.uniform(0.0, 360.0)) if azimuth is None else azimuth
    eye = cam.orbit_eye(W.CENTER, W.CAMERA["distance"], az, 25.0 if case["scene"] == "slab" else W.CAMERA["elevation"])
    viewi, proji = cam.camera_matrices(eye, W.CENTER, W.CAMERA["fov"], w, h)
    return RenderSettings(sigma_s=ss, sigma_a=sa, scattevs=ev,
                          sun_dir=cam.sun_direction(W.SUN["elevation"], W.SUN["azimuth"]),
                          sun_color=np.asarray(W.SUN["color"], np.float32), sun_angle=W.SUN["angle"], sky=sky,
                          phase=phase, viewi=viewi, proji=proji, w=w, h=h, **more)


def _options(case, rng):
    more = {}
    if case["phase"] == "exact":
        more["phase_mode"] = N.DR_PHASE_MIE_EXACT
    elif case["phase"] == "hg":
        more.update(phase_mode=N.DR_PHASE_HG, hg_g=0.8)
    if case["env"] == "map":
        # a smooth sky gradient with a bright blob, as an environment texture has
        y, x = np.mgrid[0:128, 0:256].astype(np.float32)
        g = 0.4 + 0.6 * (1.0 - y / 127.0)
        u = float(rng.uniform(40, 200))
        blob = np.exp(-((x - u) ** 2 + (y - 40.0) ** 2) / 200.0)
        more.update(env_mode=N.DR_ENV_MAP,
                    env_map=np.stack([g * 0.6 + blob, g * 0.7 + blob, g + blob, np.ones_like(g)], -1).astype(np.float32))
    elif case["env"] == "none":
        more["env_mode"] = N.DR_ENV_NONE
    if case["depth"]:
        # geometry in front of, inside and behind the cloud; a third of the pixels see none
        d = rng.uniform(2.0, 3.2, (case["h"], case["w"])).astype(np.float32)
        d[rng.random(d.shape) < 0.33] = np.float32(1e30)
        more.update(depth=d, depthcomp=case["kind"] != "shadow")
    if case["occluders"]:
        more["embree"] = True
    return more


def _occluders(rng):
    """A ground quad below the cloud and a scatter of small holdout triangles beside it."""
    ground = (np.array([[-20, -20, 0.02], [20, -20, 0.02], [20, 20, 0.02], [-20, 20, 0.02]], np.float32),
              np.array([[0, 1, 2], [0, 2, 3]], np.uint32), 0)
    base = rng.uniform([0.6, 0.4, 0.6], [1.6, 1.4, 1.4], (400, 3))
    v = (base[:, None, :] + rng.normal(scale=0.05, size=(400, 3, 3))).reshape(-1, 3).astype(np.float32)
    return [ground, (v, np.arange(1200, dtype=np.uint32).reshape(-1, 3), 2)]


class _DeviceTile:
    """A device buffer of the library as __cuda_array_interface__ (no copy); it
    keeps the owner of the memory alive for as long as a tensor uses it."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 2}


def _rays(case, rng):
    """Rays from around the cloud towards points inside it."""
    n = case["rays"]
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    target = 0.5 + rng.uniform(-0.3, 0.3, (n, 3))
    ro = target - 1.5 * d
    return np.ascontiguousarray(ro, np.float32), np.ascontiguousarray(d, np.float32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    phase, sky = _tables()
    stream = int(rng.integers(1, 1 << 31))
    r = Renderer(0)
    st = {"kind": case["kind"], "case": case, "r": r, "seed": stream}
    if case["kind"] == "batch":
        scenes = [_octree("puff", max(64, case["n"] >> (i % 3)), rng) for i in range(case["fields"])]
        views = []
        for f in range(case["fields"]):
            for k in range(case["views"]):
                # sides from a sixth of the largest upwards, a quarter of the samples for every other view
                side = max(2, int(case["side"] * (1.0, 0.3, 0.7, 0.17, 0.5)[(3 * f + k) % 5])) & ~1
                s = _settings(case, rng, phase, sky, side, side)
                views.append(BatchView(f, s, max(1, case["spp"] // (1 + 3 * (k & 1))), stream + 16 * f + k))
        st["batch"] = Batch(r, scenes, views)
        st["out"] = []
        for i, v in enumerate(views):
            shape = (v.settings.h, v.settings.w, 4)
            st["out"].append([torch.as_tensor(_DeviceTile(st["batch"], p, shape), device="cuda")
                              for p in st["batch"].output_ptrs(i)])
        return st
    if case["kind"] == "adjoint":
        n = case["n"]
        grid = np.full((n, n, n), 0.3, np.float32)
        oc = build_from_dense(grid, 1.0 / n, 12)
        r.upload(oc)
        g = torch.Generator(device="cuda").manual_seed(stream)
        b = torch.tensor(oc.bricks, device="cuda")
        st["bricks"] = (b * (0.5 + torch.rand(b.shape, generator=g, device="cuda"))).requires_grad_()
        st["albedo"] = torch.tensor(case["albedo"], device="cuda", requires_grad=True)
        st["views"] = [AD.DiffView(_settings(case, rng, phase, sky, case["w"], case["h"],
                                             azimuth=360.0 * k / case["views"]), case["spp"], stream + k)
                       for k in range(case["views"])]
        st["target"] = 0.2 * torch.rand((case["views"], case["h"], case["w"], 3), generator=g, device="cuda")
        return st
    oc = _octree(case["scene"], case["n"], rng)
    r.upload(oc)
    if case["kind"] == "transmittance":
        r.set_params(_settings(case, rng, phase, sky, 64, 64))
        ro, rd = _rays(case, rng)
        st["ro"], st["rd"] = torch.as_tensor(ro, device="cuda"), torch.as_tensor(rd, device="cuda")
        st["out"] = torch.zeros(case["rays"], dtype=torch.float64, device="cuda")
        st["octree"] = oc
        return st
    if case["occluders"]:
        r.set_occluders(_occluders(rng))
    r.set_params(_settings(case, rng, phase, sky, case["w"], case["h"], **_options(case, rng)))
    if SHAPES[case["shape"]]:
        r.set_tuning(*SHAPES[case["shape"]])
    shape = (case["th"], case["tw"], 4)
    if case["kind"] == "host":
        st["out"] = (np.zeros(shape, np.float32), np.zeros(shape, np.float32))
    else:
        st["out"] = tuple(torch.zeros(shape, device="cuda") for _ in range(1 if case["kind"] == "shadow" else 2))
    return st


def run(st):
    case, r, kind = st["case"], st["r"], st["kind"]
    if kind == "host":
        return r.render_tile(case["x0"], case["y0"], case["tw"], case["th"], case["spp"], seed=st["seed"],
                             sample_base=0, out=st["out"])
    sh = stream_handle(torch.cuda.current_stream())
    if kind == "frame":
        sun, sky = st["out"]
        r.render_tile_async(case["x0"], case["y0"], case["tw"], case["th"], case["spp"], st["seed"], 0,
                            sun.data_ptr(), sky.data_ptr(), sh)
    elif kind == "shadow":
        r.shadow_tile_async(case["x0"], case["y0"], case["tw"], case["th"], case["spp"], st["seed"], 0,
                            st["out"][0].data_ptr(), sh)
    elif kind == "batch":
        st["batch"].launch(sh)
    elif kind == "adjoint":
        st["bricks"].grad = st["albedo"].grad = None
        sun, sky = AD.render(st["bricks"], st["albedo"], r, st["views"], majorant_scale=1.05)
        loss = (((sun + sky)[..., :3] - st["target"]) ** 2).sum()
        loss.backward()
        return [sun.detach(), sky.detach(), st["bricks"].grad, st["albedo"].grad]
    elif kind == "transmittance":
        N.check(N.lib().dr_transmittance_noalloc(
            r.handle, ctypes.c_void_p(st["ro"].data_ptr()), ctypes.c_void_p(st["rd"].data_ptr()), case["rays"],
            case["spp"], st["seed"], ctypes.c_void_p(st["out"].data_ptr()), ctypes.c_void_p(sh)))
    return st["out"]


# ---- what a pass cannot do without ------------------------------------------------
def _scene_bytes(scene, n):
    """Bricks of the occupied part of the unit cube (8^3 floats per 7^3 cells), each read once."""
    part = {"puff": 0.17, "cumulus": 0.15, "slab": 0.023}[scene]
    return part * n ** 3 * (8 / 7) ** 3 * 4


def work(case):
    """bytes: the scene's bricks read once, the outputs (16 bytes a pixel and
    buffer) and further inputs once.  flops: 60 for a path sample's stream and
    root test, 300 for each segment in the medium and 400 for each scattering
    event (phase sampling and evaluation, sun sampling, MIS), with the
    segments and events a sample makes on average in these scenes."""
    kind, spp = case["kind"], case["spp"]
    per_path = {"puff": (1.2, 0.35), "cumulus": (0.8, 0.25), "slab": (0.3, 0.05)}[case["scene"]]
    if kind == "transmittance":
        return {"bytes": _scene_bytes("puff", case["n"]) + case["rays"] * 32, "flops": case["rays"] * spp * 360.0}
    if kind == "batch":
        px = 0.4 * case["fields"] * case["views"] * case["side"] ** 2
        scene = sum(_scene_bytes("puff", max(64, case["n"] >> (i % 3))) for i in range(case["fields"]))
        spp *= 0.7
    elif kind == "adjoint":
        px = case["views"] * case["w"] * case["h"]
        # a full grid: read by both directions, its gradient written once
        scene = 3.0 * case["n"] ** 3 * (8 / 7) ** 3 * 4
        per_path = (6.0, 1.8)
    else:
        px = case["tw"] * case["th"]
        scene = _scene_bytes(case["scene"], case["n"])
    out = 16 * px * (1 if kind == "shadow" else 2) * (2 if kind == "adjoint" else 1)
    depth = 4 * px if case["depth"] else 0
    seg, ev = (0.6, 0.0) if kind == "shadow" else per_path
    return {"bytes": out + depth + scene, "flops": px * spp * (60.0 + 300.0 * seg + 400.0 * ev)}


# ---- 64-bit values -----------------------------------------------------------------
def exact(case, seed):
    """Transmittance has a value of its own, exp(-sigma_t * integral of the
    density): the integral by midpoint sums in 64 bits over the input's octree.
    A rendered image is a sum over given random streams: each decision of a
    path is a comparison of 32-bit values, so no 64-bit value belongs to it."""
    if case["kind"] != "transmittance":
        return None
    st = prepare(case, seed)
    oc = st["octree"]
    dev = "cuda"
    ce = torch.as_tensor(np.ascontiguousarray(oc.nodes["ce"]), device=dev).double()
    chn = torch.as_tensor(np.ascontiguousarray(oc.nodes["chn"]).astype(np.int64), device=dev)
    volx = torch.as_tensor(np.ascontiguousarray(oc.nodes["volx"][:, 1]).astype(np.int64), device=dev)
    live = torch.as_tensor(np.ascontiguousarray(oc.nodes["qval"][:, 1]) > 0, device=dev)
    bricks = torch.as_tensor(oc.bricks, device=dev).double().reshape(-1)
    ss, sa, _ = W.medium_of(case["sigma_t"], case["albedo"], case["events"])
    sigma = float(np.float32(ss) + np.float32(sa))
    steps, far = 4096, 3.0
    dt = far / steps
    t = (torch.arange(steps, device=dev, dtype=torch.float64) + 0.5) * dt
    out = []
    for k in range(0, case["rays"], 512):
        ro, rd = st["ro"][k:k + 512].double(), st["rd"][k:k + 512].double()
        p = ro[:, None, :] + t[None, :, None] * rd[:, None, :]
        node = torch.zeros(p.shape[:2], dtype=torch.int64, device=dev)
        inside = ((p - ce[0, :3]).abs() < ce[0, 3]).all(-1)
        for _ in range(oc.mlevel + 1):
            slot = ((p >= ce[node][..., :3]).long() * torch.tensor([1, 2, 4], device=dev)).sum(-1)
            leaf = volx[node] != N.DR_NONE
            child = chn[node, slot]
            inside &= leaf | (child != 0)
            node = torch.where(leaf, node, child)
        inside &= (volx[node] != N.DR_NONE) & live[node]
        node = torch.where(inside, node, torch.zeros_like(node))
        c = ce[node]
        q = (0.5 * (p - (c[..., :3] - c[..., 3:4])) * 7.0 / c[..., 3:4]).clamp(0.0, 7.0)
        a = q.floor().clamp(max=6.0)
        f = q - a
        a = a.long()
        b0 = torch.where(inside, volx[node], torch.zeros_like(node)) * 512
        rho = torch.zeros_like(f[..., 0])
        for corner in range(8):
            o = [corner >> j & 1 for j in range(3)]
            w = torch.ones_like(rho)
            for j in range(3):
                w = w * (f[..., j] if o[j] else 1.0 - f[..., j])
            rho += w * bricks[b0 + (a[..., 2] + o[2]) * 64 + (a[..., 1] + o[1]) * 8 + a[..., 0] + o[0]]
        tau = torch.where(inside, rho, torch.zeros_like(rho)).sum(1) * dt
        out.append(torch.exp(-sigma * tau))
    return torch.cat(out)
