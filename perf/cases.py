"""The workloads the tracer's speed is measured on, each through the public entry points
(`naivetrace_b200.algo.GpuContext`, the object wrapper of the C ABI).

Kinds of work:
  render   a resident scene: the framebuffer is cleared, one pass of `spp` samples per pixel is
           rendered and the linear image is read back, as a viewer or a batch renderer does per
           frame (algo pt or pt2, pseudo- or quasi-random).
  guided   the same with a trained network guiding the scattering (guiding frozen).
  train    Adam steps of the guiding network on a batch of training records.
  rays     closest-hit and occlusion queries of a batch of rays in host memory.
  views    a batch of camera views of one scene in one call.
  open     a scene opened from host memory, its first image rendered and read back, closed.

All inputs are procedural (naivetrace_b200/scenes.py) and made from the seed: the camera pose,
the sampling seed, rays, records and network weights.
"""
import copy
import functools
import math

import numpy as np
import torch

from naivetrace_b200 import abi, scenes
from naivetrace_b200.algo import GpuContext
from naivetrace_b200.scene import CameraSpec, make_params

# Mean vertices of a path and rays per vertex, for the operation estimate of `work`.
PATH_VERTICES = {"cornell": 4.5, "materials": 6.0, "terrain": 1.7, "medium": 4.5, "mix": 5.0, "spheres": 5.0,
                 "planet": 2.5, "room": 5.0}


def listed():
    return [
        # The smallest call: a thumbnail of a box at one sample, as an editor redraws while a
        # parameter is dragged.  Launches and latency.
        {"name": "thumbnail_64", "kind": "render", "scene": "cornell", "xres": 64, "yres": 64, "spp": 1, "depth": 10,
         "algo": "pt", "qmc": False},
        # The standard small frame: the Cornell box at 256x256, 16 samples, depth 10.
        {"name": "cornell_256", "kind": "render", "scene": "cornell", "xres": 256, "yres": 256, "spp": 16,
         "depth": 10, "algo": "pt", "qmc": False},
        # One progressive pass over a large mesh in an odd-sized window, as a viewer runs first
        # after every camera move.
        {"name": "terrain_pass", "kind": "render", "scene": "terrain", "mesh": 1024, "xres": 641, "yres": 359,
         "spp": 1, "depth": 16, "algo": "pt", "qmc": False},
        # The largest: a full-HD frame of the mesh scene (2.75 M triangles) at 64 samples.
        {"name": "terrain_frame", "kind": "render", "scene": "terrain", "mesh": 1024, "xres": 1920, "yres": 1080,
         "spp": 64, "depth": 16, "algo": "pt", "qmc": False},
        # Homogeneous chromatic medium, deep paths.
        {"name": "medium_box", "kind": "render", "scene": "medium", "xres": 512, "yres": 512, "spp": 8, "depth": 32,
         "algo": "pt", "qmc": False},
        # A planet's tabulated atmosphere through a fisheye camera: heterogeneous tracking.
        {"name": "atmosphere", "kind": "render", "scene": "planet", "xres": 512, "yres": 512, "spp": 8, "depth": 32,
         "algo": "pt", "qmc": False},
        # The null-path tracer with quasi-random samples in overlapping media.
        {"name": "pt2_media", "kind": "render", "scene": "mix", "xres": 320, "yres": 240, "spp": 8, "depth": 25,
         "algo": "pt2", "qmc": True},
        # Guided rendering with a frozen network in the gap-lit room.
        {"name": "guided_room", "kind": "guided", "scene": "room", "xres": 1280, "yres": 720, "spp": 2, "depth": 12,
         "bounces": 2},
        # One training round of the network at its default batch and step count.
        {"name": "guide_training", "kind": "train", "records": 8192, "steps": 16},
        # Ray queries of another program (picking, baking): a ragged million rays.
        {"name": "ray_queries", "kind": "rays", "mesh": 1024, "rays": 1000003},
        # A batch of small views of the mesh scene, as for a dataset of renderings.
        {"name": "view_batch", "kind": "views", "mesh": 1024, "views": 24, "side": 256, "spp": 4, "depth": 16},
        # Opening the mesh scene: copy, upload, tree build, a first preview pass, read-back.
        {"name": "open_scene", "kind": "open", "mesh": 1024, "xres": 640, "yres": 360, "spp": 1, "depth": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render"] * 6 + ["guided", "train", "rays", "views", "open"])
    mesh = rng.choice([128, 256, 512, 1024])
    if kind == "render":
        scene = rng.choice(["cornell", "materials", "terrain", "terrain", "medium", "mix", "spheres", "planet", "room"])
        algo = rng.choice(["pt", "pt", "pt", "pt2"])
        paths = _log(rng, 1 << 10, 1 << (24 if scene in ("cornell", "terrain") else 21))
        spp = min(rng.choice([1, 1, 2, 3, 4, 8, 16, 64]), max(1, paths // 1024))
        pixels = min(max(1024, paths // spp), 1 << 21)
        xres = max(16, int(math.sqrt(pixels * rng.uniform(0.6, 2.0))))
        case = {"kind": kind, "scene": scene, "xres": xres, "yres": max(16, pixels // xres), "spp": spp,
                "depth": rng.randint(4, 31), "algo": algo, "qmc": algo == "pt2" and rng.random() < 0.5}
        if scene == "terrain":
            case["mesh"] = mesh
        return case
    if kind == "guided":
        return {"kind": kind, "scene": rng.choice(["room", "cornell"]), "xres": _log(rng, 96, 1400),
                "yres": _log(rng, 64, 800), "spp": rng.randint(1, 4), "depth": rng.randint(4, 16),
                "bounces": rng.randint(0, 3)}
    if kind == "train":
        return {"kind": kind, "records": _log(rng, 256, 1 << 18), "steps": rng.choice([1, 4, 16, 32])}
    if kind == "rays":
        return {"kind": kind, "mesh": mesh, "rays": _log(rng, 64, 1 << 21)}
    if kind == "views":
        return {"kind": kind, "mesh": mesh, "views": rng.randint(1, 40), "side": rng.choice([65, 96, 128, 200, 256]),
                "spp": rng.randint(1, 8), "depth": rng.randint(4, 16)}
    return {"kind": kind, "mesh": mesh, "xres": _log(rng, 64, 1280), "yres": _log(rng, 64, 720), "spp": 1,
            "depth": rng.randint(4, 16)}


@functools.lru_cache(maxsize=4)
def _terrain(mesh):
    """The mesh scene at `mesh` x `mesh` height samples (1024: 2.75 M triangles); geometry
    flattened once, shared by every camera."""
    level, count = {1024: (5, 32), 512: (5, 16), 256: (4, 8), 128: (3, 8)}[mesh]
    s = scenes.terrain_spheres(terrain_n=mesh, sphere_level=level, num_spheres=count,
                               env_w=2 * mesh, env_h=mesh)
    s.arrays()
    return s


def _with_camera(scene, case, rng):
    """A shallow copy of `scene` at the case's resolution, the camera nudged by the seed."""
    s = copy.copy(scene)
    c = scene.camera
    pos = tuple(float(p) for p in c.pos)
    if case.get("scene") != "planet":  # the planet's camera stands 2 m above ground
        pos = tuple(float(p + d) for p, d in zip(c.pos, rng.uniform(-0.02, 0.02, 3)))
    s.camera = CameraSpec(kind=c.kind, pos=pos, dir=c.dir, up=c.up, fov_deg=c.fov_deg, xres=case["xres"],
                          yres=case["yres"])
    return s


def _scene(case, rng):
    name = case.get("scene", "terrain")
    size = (case["xres"], case["yres"])
    if name == "terrain":
        return _with_camera(_terrain(case["mesh"]), case, rng)
    make = {"cornell": scenes.cornell_box, "materials": scenes.cornell_box_materials,
            "medium": scenes.cornell_box_medium, "mix": scenes.cornell_box_media_mix, "spheres": scenes.spheres_box,
            "planet": scenes.planet_atmosphere, "room": scenes.guiding_room}[name]
    return _with_camera(make(*size), case, rng)


def _network(rng):
    """Weights as a trained guide has them: He-uniform layers and output biases that give
    lobes of moderate concentration in all directions, sampled half of the time."""
    sizes = [(96, 64), (64, 64), (64, 64), (64, 64), (64, 48)]
    parts = []
    for k, (i, o) in enumerate(sizes):
        lim = math.sqrt(6.0 / i) * (0.1 if k == 4 else 1.0)
        parts.append(rng.uniform(-lim, lim, i * o))
        b = np.zeros(o)
        if k == 4:
            for lobe in range(8):
                v = rng.normal(size=3)
                b[5 * lobe + 1:5 * lobe + 4] = v / np.linalg.norm(v)
                b[5 * lobe + 4] = rng.uniform(0.0, 3.0)
        parts.append(b)
    return np.concatenate(parts).astype(np.float32)


def _records(n, rng):
    """Training records as a room gives them: points on its walls, normals inward, outgoing
    directions in the hemisphere, light from a bright opening, heavy-tailed weights."""
    r = np.zeros((n, 14), np.float32)
    pos = rng.random((n, 3))
    axis, side = rng.integers(0, 3, n), rng.integers(0, 2, n)
    rows = np.arange(n)
    pos[rows, axis] = side
    nrm = np.zeros((n, 3))
    nrm[rows, axis] = 1.0 - 2.0 * side

    def hemisphere(noise):
        flip = np.sign((noise * nrm).sum(1, keepdims=True))
        v = noise * np.where(flip == 0, 1.0, flip)
        return v / np.linalg.norm(v, axis=1, keepdims=True)

    to_gap = np.array([1.0, 0.5, 0.5]) - pos + rng.normal(scale=0.15, size=(n, 3))
    wi = hemisphere(to_gap)
    r[:, 0:3], r[:, 3:6], r[:, 6:9], r[:, 9:12] = pos, nrm, hemisphere(rng.normal(size=(n, 3))), wi
    r[:, 12] = np.maximum(1e-3, (wi * nrm).sum(1)) / math.pi
    r[:, 13] = np.exp(rng.normal(-1.0, 1.0, n))
    return r


def _rays(n, rng):
    """Half the rays from a camera-like point through a grid, half scattered off the ground;
    segments (with an end) for the occlusion query."""
    rays = np.zeros((n, 8), np.float32)
    h = n // 2
    rays[:h, 0:3] = np.array([0.0, 2.2, -6.5]) + rng.uniform(-0.1, 0.1, 3)
    d = rng.uniform(-0.6, 0.6, (h, 2))
    rays[:h, 4:7] = np.stack([d[:, 0], 0.5 * d[:, 1] - 0.3, np.ones(h)], 1)
    m = n - h
    rays[h:, 0] = rng.uniform(-4.5, 4.5, m)
    rays[h:, 1] = rng.uniform(0.25, 0.6, m)
    rays[h:, 2] = rng.uniform(-4.5, 4.5, m)
    rays[h:, 4:7] = rng.normal(size=(m, 3))
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7], axis=1, keepdims=True)
    rays[:, 7] = 1e30
    segments = rays.copy()
    segments[:, 7] = rng.uniform(0.5, 8.0, n)
    return rays, segments


def _views(case, rng):
    """Poses as scenes.terrain_views draws them; sides and samples cycle around the case's."""
    poses = scenes.terrain_views(case["views"], seed=int(rng.integers(1 << 30)))
    out = []
    for k, (cam, _) in enumerate(poses):
        side = case["side"] // (1, 2, 1, 4)[k % 4]
        out.append((CameraSpec(kind=cam.kind, pos=cam.pos, dir=cam.dir, up=cam.up, fov_deg=cam.fov_deg, xres=side,
                               yres=max(1, side - k % 3)), case["spp"] + k % 3))
    return out


def _params(case):
    return make_params(max_ray_depth=case["depth"], algo=abi.ALGO_PT2 if case.get("algo") == "pt2" else abi.ALGO_PT,
                       qmc=bool(case.get("qmc")))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"case": case, "seed": int(rng.integers(1, 1 << 31))}
    if kind == "open":
        state["scene"], state["params"] = _scene(case, rng), _params(case)
    elif kind in ("render", "guided"):
        ctx = GpuContext(_scene(case, rng), _params(case))
        if kind == "guided":
            ctx.set_guiding(True, train=0, max_depth=case["bounces"])
            ctx.guide_set_params(_network(rng))
        state["ctx"] = ctx
    elif kind == "train":
        ctx = GpuContext(scenes.cornell_box(16, 16), make_params(max_ray_depth=4))
        ctx.set_guiding(True, train=1)
        state.update(ctx=ctx, weights=_network(rng), records=_records(case["records"], rng))
    elif kind == "rays":
        state["ctx"] = GpuContext(_with_camera(_terrain(case["mesh"]), {"xres": 16, "yres": 16}, rng),
                                  make_params(max_ray_depth=4))
        state["rays"], state["segments"] = _rays(case["rays"], rng)
    else:
        state["ctx"] = GpuContext(_with_camera(_terrain(case["mesh"]), {"xres": 16, "yres": 16}, rng), _params(case))
        state["views"] = _views(case, rng)
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "open":
        ctx = GpuContext(state["scene"], state["params"])
        ctx.render(case["spp"], seed=state["seed"])
        rgb = ctx.framebuffer()
        ctx.close()
        return {"rgb": rgb}
    ctx = state["ctx"]
    if kind in ("render", "guided"):
        ctx.clear()
        ctx.render(case["spp"], seed=state["seed"])
        return {"rgb": ctx.framebuffer()}
    if kind == "train":
        ctx.guide_set_params(state["weights"])
        loss = ctx.guide_train(state["records"], case["steps"], 1e-3)
        return {"loss": loss, "params": ctx.guide_params()}
    if kind == "rays":
        prim, t, u, v = ctx.intersect(state["rays"])
        return {"prim": prim, "t": t, "u": u, "v": v, "occluded": ctx.occluded(state["segments"])}
    return {"rgb%d" % k: im for k, im in enumerate(ctx.render_views(state["views"], seed=state["seed"]))}


def _triangles(case):
    if "mesh" in case:
        n = case["mesh"]
        level, count = {1024: (5, 32), 512: (5, 16), 256: (4, 8), 128: (3, 8)}[n]
        return 2 * (n - 1) ** 2 + count * 20 * 4 ** level
    return {"mix": 1400}.get(case.get("scene"), 48)


def work(case):
    """Bytes: the scene read once (36 bytes per triangle; host to device for `open`), inputs
    and results once.  Operations: per ray one descent of a binary tree over the primitives
    (two boxes of 18 operations per level) and one primitive test (60), per vertex 300 for light
    and scattering samples; per training record and step the network's multiplications."""
    kind = case["kind"]
    if kind == "train":
        n = case["records"] * case["steps"]
        return {"bytes": 56.0 * case["records"] + 4.0 * 20784 * 2 * case["steps"], "flops": 6.0 * 19456 * n}
    tris = _triangles(case)
    ray = 36.0 * math.log2(tris + 1) + 60.0
    if kind == "rays":
        n = case["rays"]
        return {"bytes": 36.0 * tris + n * (2 * 32.0 + 16.0 + 1.0), "flops": 2 * n * ray}
    if kind == "views":
        sizes = [(case["side"] // (1, 2, 1, 4)[k % 4], case["spp"] + k % 3, k % 3) for k in range(case["views"])]
        pixels = sum(s * max(1, s - d) for s, _, d in sizes)
        paths = sum(s * max(1, s - d) * p for s, p, d in sizes)
    else:
        pixels = case["xres"] * case["yres"]
        paths = pixels * case["spp"]
    vertices = PATH_VERTICES[case.get("scene", "terrain")] * paths
    guide = 2.0 * 19456 * paths * 2 if kind == "guided" else 0.0
    return {"bytes": 36.0 * tris + 12.0 * pixels, "flops": vertices * (2 * ray + 300.0) + guide}


def _exact_training(weights, records, steps):
    """Loss of the last step and the parameters after `steps` Adam steps, in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sizes = [(96, 64), (64, 64), (64, 64), (64, 64), (64, 48)]
    p = torch.tensor(weights, dtype=torch.float64, device=dev)
    r = torch.tensor(records, dtype=torch.float64, device=dev)
    freq = torch.tensor([2.0 ** (j / 8.0) * math.pi for j in range(12)], dtype=torch.float64, device=dev)
    arg = r[:, 0:3, None] * freq
    enc = torch.stack([arg.sin(), arg.cos()], -1).reshape(len(r), 72)
    x = torch.cat([enc, r[:, 0:9], torch.ones_like(r[:, :1]), torch.zeros_like(r[:, :14])], 1)
    mid, half = (math.log(0.05) + math.log(40.0)) / 2, (math.log(40.0) - math.log(0.05)) / 2
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    loss = 0.0
    for step in range(1, steps + 1):
        w = p.clone().requires_grad_(True)
        h, at = x, 0
        for k, (i, o) in enumerate(sizes):
            h = h @ w[at:at + i * o].reshape(o, i).T + w[at + i * o:at + i * o + o]
            at += i * o + o
            h = torch.relu(h) if k < 4 else h
        lobes = h[:, :40].reshape(-1, 8, 5)
        weight = torch.softmax(lobes[:, :, 0], 1)
        mu = torch.nn.functional.normalize(lobes[:, :, 1:4], dim=2)
        kappa = torch.exp(mid + half * torch.tanh((lobes[:, :, 4] - mid) / half))
        cosine = (mu * r[:, None, 9:12]).sum(2)
        vmf = kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa))) * torch.exp(kappa * (cosine - 1))
        c = 0.05 + 0.9 * torch.sigmoid(h[:, 40])
        density = (1 - c) * r[:, 12] + c * (weight * vmf).sum(1)
        value = -(r[:, 13] * torch.log(density)).mean()
        g, = torch.autograd.grad(value, w)
        loss = float(value.detach())
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": loss, "params": p.cpu().numpy()}


def _exact_rays(case, rng):
    """Distance and barycentrics of the nearest triangle by testing every ray against every
    triangle in 64 bits (t = -1, u = v = 0 for a miss)."""
    verts, _, tris, _ = _terrain(case["mesh"]).arrays()
    _with_camera(_terrain(case["mesh"]), {"xres": 16, "yres": 16}, rng)
    rays, _ = _rays(case["rays"], rng)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.tensor(verts, dtype=torch.float64, device=dev)[torch.tensor(tris.astype(np.int64), device=dev)]
    v0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    r = torch.tensor(rays, dtype=torch.float64, device=dev)
    out = torch.zeros((len(r), 3), dtype=torch.float64, device=dev)
    chunk = max(1, (1 << 26) // len(tris))
    for a in range(0, len(r), chunk):
        o, d = r[a:a + chunk, 0:3], r[a:a + chunk, 4:7]
        den = -(d @ nrm.T)
        t = (o @ nrm.T - (v0 * nrm).sum(1)) / den
        # u and v from the moment of the ray about the triangle's origin: d x (o - v0).
        moment = torch.linalg.cross(o, d)
        u = (moment @ e2.T - d @ torch.linalg.cross(e2, v0).T) / den
        v = -(moment @ e1.T - d @ torch.linalg.cross(e1, v0).T) / den
        t[~((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (den != 0))] = math.inf
        best, at = t.min(1)
        rows = torch.arange(len(o), device=dev)
        hit = torch.isfinite(best)
        out[a:a + chunk, 0] = torch.where(hit, best, -1.0)
        out[a:a + chunk, 1] = torch.where(hit, u[rows, at], 0.0)
        out[a:a + chunk, 2] = torch.where(hit, v[rows, at], 0.0)
    out = out.cpu().numpy()
    return {"prim": None, "t": out[:, 0], "u": out[:, 1], "v": out[:, 2], "occluded": None}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    rng.integers(1, 1 << 31)
    if case["kind"] == "train" and case["records"] * case["steps"] <= 1 << 22:
        weights = _network(rng)
        return _exact_training(weights, _records(case["records"], rng), case["steps"])
    if case["kind"] == "rays" and float(case["rays"]) * _triangles(case) <= 4e10:
        return _exact_rays(case, rng)
    return None  # a Monte Carlo image has no value that plain array code gives in seconds
