"""Performance cases: the renders a user of this library asks for, and the photon-tree
build it offers to hosts, over the range of their sizes and options.

A case is a dict of plain values:
  kind        render   one progressive update of a resident scene: `iterations` more
                       iterations, then the image read back (a viewport that refreshes)
              frame    a whole render as the Blender add-on asks for it: init with the
                       scene's Blender arrays, render, image, release
              batch    one update of several resident scenes in one launch set, and
                       their images
              kd_tree  the photon tree in the caller's own device buffers
  scene       sphere (smooth glass over a plane), pool (rough or smooth water over a
              floor), gems (faceted, dispersive), displaced (noisy rough-glass spheres)
  size        sphere: subdivisions, pool: vertices per side, gems: gems, displaced: triangles
  paths       light paths per iteration (per scene of a batch: the geometric mean)
  sampler     uniform, hybrid (the reference's Metropolis scheme) or pssmlt

Every scene varies with the seed: geometry noise, light position and power, camera
height and the sample streams.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from realcausticsengine_gb300 import _native, abi, scenes
from realcausticsengine_gb300.scene import InitArgs, Light, Material, Mesh, look_at_camera
from realcausticsengine_gb300.session import Context, Renderer, batch_render

SAMPLERS = {"uniform": abi.SAMPLER_UNIFORM, "hybrid": abi.SAMPLER_HYBRID, "pssmlt": abi.SAMPLER_PSSMLT}
CHAINS = 65536
MAX_TREE = 1 << 19           # rc_kd_build_noalloc's largest photon count


def _render(name, scene, size, width, height, paths, depth, iterations, **more):
    c = {"kind": "render", "scene": scene, "size": size, "width": width, "height": height, "paths": paths,
         "depth": depth, "iterations": iterations, "sampler": "uniform", "light": "area", "roughness": 0.02,
         "learned": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest update: a thumbnail viewport, where launches and round trips are the time
        _render("viewport_96x64", "sphere", 4, 96, 64, 6144, 6, 1),
        # the first render of a new user: glass ball, point light, 512 x 512
        _render("sphere_512", "sphere", 5, 512, 512, 1 << 20, 8, 4, light="point", roughness=0.0),
        # the add-on's defaults (as many light paths as pixels, depth 6) on half-HD water
        _render("pool_960x540", "pool", 512, 960, 540, 518400, 6, 4),
        # ragged sizes throughout
        _render("pool_1283x717", "pool", 301, 1283, 717, 3000017, 7, 2),
        # the production water render: 16M light paths per iteration, full HD
        _render("pool_1080p", "pool", 512, 1920, 1080, 1 << 24, 8, 2),
        # emission drawn from the online-trained network, training included
        _render("pool_learned", "pool", 512, 1280, 720, 1 << 22, 8, 2, learned=True),
        # the reference's own sampler, many chains
        _render("pool_hybrid", "pool", 512, 960, 540, 518400, 6, 4, sampler="hybrid", roughness=0.0),
        # long paths through overlapping gems, uniform and Metropolis light paths
        _render("gems_1080p", "gems", 2000, 1920, 1080, 1 << 22, 8, 1),
        _render("gems_pssmlt", "gems", 2000, 1280, 720, 1 << 22, 8, 1, sampler="pssmlt"),
        # a farm's set of small scenes
        {"name": "batch_6", "kind": "batch", "scene": "displaced", "size": 20000, "scenes": 6, "width": 384,
         "height": 384, "paths": 1 << 20, "depth": 8, "iterations": 2},
        # a still of a fine mesh from the application's arrays to the image
        {"name": "frame_640x480", "kind": "frame", "scene": "displaced", "size": 100000, "width": 640, "height": 480,
         "paths": 307200, "depth": 6, "iterations": 4},
        # a host's photons turned into a tree in its own buffers
        {"name": "kd_tree_300k", "kind": "kd_tree", "photons": 300001},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "render", "render", "batch", "frame", "kd_tree"])
    if kind == "kd_tree":
        return {"kind": kind, "photons": _log(rng, 1000, MAX_TREE)}
    if kind == "batch":
        return {"kind": kind, "scene": "displaced", "size": _log(rng, 2000, 60000), "scenes": rng.randint(2, 6),
                "width": rng.randint(128, 400), "height": rng.randint(128, 400), "paths": _log(rng, 1 << 18, 1 << 20),
                "depth": rng.randint(5, 8), "iterations": rng.randint(1, 3)}
    width = _log(rng, 96, 1280)
    height = max(48, int(width * rng.uniform(0.5, 0.8)))
    if kind == "frame":
        return {"kind": kind, "scene": "displaced", "size": _log(rng, 2000, 150000), "width": min(width, 800),
                "height": min(height, 600), "paths": _log(rng, 1 << 14, 1 << 20), "depth": rng.randint(4, 8),
                "iterations": rng.randint(1, 6)}
    scene = rng.choice(["sphere", "pool", "pool", "gems"])
    sampler = rng.choice(["uniform", "uniform", "uniform", "hybrid", "pssmlt"])
    if scene == "gems":
        return _render(None, scene, _log(rng, 100, 2000), width, height, _log(rng, 1 << 16, 1 << 21), rng.randint(5, 8),
                       1, sampler=sampler)
    size = rng.randint(2, 5) if scene == "sphere" else rng.randint(64, 512)
    return _render(None, scene, size, width, height, _log(rng, 1 << 13, 1 << 23 if sampler == "uniform" else 1 << 20),
                   rng.randint(4, 8), rng.randint(1, 4), sampler=sampler,
                   light=rng.choice(["area", "point"]) if scene == "sphere" else "area",
                   roughness=rng.choice([0.0, 0.02, 0.05]), learned=sampler == "uniform" and rng.random() < 0.2)


# ---------------------------------------------------------------- scenes

def _mesh(V, N, F, material, matrix=None):
    return Mesh(V, N, F, np.zeros(len(F), np.int16), [material],
                np.eye(4, dtype=np.float32) if matrix is None else matrix)


def _sphere(case, rng):
    sc = scenes.glass_sphere_point(case["width"], case["height"], subdiv=int(case["size"]), light=case["light"])
    if case["roughness"] > 0:
        sc.materials[0] = Material("R", color=(1, 1, 1), ior=1.5, roughness=float(case["roughness"]))
    sc.meshes[0].matrix = scenes.translate(float(rng.uniform(-0.2, 0.2)), float(rng.uniform(-0.2, 0.2)), 1.2)
    return sc


def _pool(case, rng):
    sc = scenes.water_pool(case["width"], case["height"], grid=8, roughness=case["roughness"])
    if case["roughness"] == 0:
        sc.materials[0] = Material("G", color=(1, 1, 1), ior=1.33)
    V, N, F = scenes.water_heightfield(int(case["size"]), seed=int(rng.integers(1 << 30)))
    sc.meshes[0] = _mesh(V, N, F, 0)
    return sc


def _gems(case, rng):
    return scenes.gem_cluster(case["width"], case["height"], n_gems=int(case["size"]), seed=int(rng.integers(1 << 30)))


def _displaced(case, rng, tris, kinds):
    mats = [Material("R", color=(1, 1, 1), ior=float(rng.uniform(1.3, 1.8)), roughness=float(rng.uniform(0.0, 0.1))),
            Material("P", color=(0.8, 0.8, 0.8), roughness=1.0, specular=0.0)]
    V, N, F = scenes.displaced_glass_sphere(rng, tris, float(rng.uniform(0.0, 0.2)))
    sc = scenes.glass_sphere_point(case["width"], case["height"], subdiv=0)
    sc.materials = mats
    sc.meshes = [_mesh(V, N, F, 0, scenes.translate(0.0, 0.0, 1.4)), _mesh(*scenes.plane(8.0, 0.0), 1)]
    sc.lights = []
    for k in kinds:
        pos = (float(rng.uniform(-1.5, 1.5)), float(rng.uniform(-1.5, 1.5)), float(rng.uniform(4.0, 6.0)))
        size = {} if k == "P" else {"width": 1.0, "height": 1.0}
        sc.lights.append(Light(k, color=(1.0, 0.9, 0.8), position=pos, power=float(rng.uniform(15.0, 30.0)), **size))
    sc.camera = look_at_camera(case["width"], case["height"], (0.0, -5.0, 4.0), (0.0, 0.0, 0.6), (0, 0, 1), 45.0)
    sc.base_radius = 0.004
    return sc


def _scene(case, rng, index=0):
    if case["scene"] == "displaced":
        return _displaced(case, rng, _spread(case, "size", index), ("P", "PA", "AAP")[index % 3])
    sc = {"sphere": _sphere, "pool": _pool, "gems": _gems}[case["scene"]](case, rng)
    for light in sc.lights:
        light.position = tuple(float(p + rng.uniform(-0.2, 0.2)) for p in light.position)
        light.power *= float(rng.uniform(0.8, 1.25))
    return sc


def _spread(case, key, index):
    """Scene `index`'s value of `key`: the case's own, spread over a factor of 16 in a batch."""
    n = case.get("scenes", 1)
    return int(case[key] * 4.0 ** ((2 * index + 1) / n - 1.0))


class _Resident:
    """A scene held in a library context, released with this object."""

    def __init__(self, scene, **options):
        self.ctx = Context()
        with self.ctx:
            self.renderer = Renderer(scene, **options)
            self.renderer.prepare()

    def __del__(self):
        self.ctx.destroy()


def _options(case, seed, index=0):
    o = {"max_path_length": case["depth"], "photons_per_iter": _spread(case, "paths", index) if index or "scenes" in case
         else case["paths"], "seed": int(seed) * 64 + index + 1, "sampler": SAMPLERS[case.get("sampler", "uniform")]}
    if case.get("learned"):
        # a learning rate too small to move a weight: every training step runs, and the
        # draws stay those of the network's seeded initial weights, so that a pass can be
        # repeated (the order of the training sums is not fixed)
        o.update(learned_proposal=True, train_iterations=1 << 20, train_steps=64, learning_rate=1e-30)
    return o


# ---------------------------------------------------------------- passes

def prepare(case, seed):
    rng = np.random.default_rng(int(seed))
    kind = case["kind"]
    if kind == "kd_tree":
        return _tree_state(case, seed)
    if kind == "batch":
        held = [_Resident(_scene(case, rng, i), **_options(case, seed, i)) for i in range(case["scenes"])]
        return {"kind": kind, "held": held, "iterations": case["iterations"]}
    scene = _scene(case, rng)
    if kind == "render":
        return {"kind": kind, "held": _Resident(scene, **_options(case, seed)), "iterations": case["iterations"]}
    held = _Resident(scene, **_options(case, seed))
    with held.ctx:
        held.renderer.release()
    return {"kind": kind, "held": held, "args": InitArgs(scene), "iterations": case["iterations"]}


def run(state):
    kind = state["kind"]
    if kind == "kd_tree":
        return _tree_pass(state)
    if kind == "batch":
        held = state["held"]
        batch_render([h.ctx for h in held], state["iterations"])
        images = []
        for h in held:
            with h.ctx:
                images.append(h.renderer.image())
        return images
    held = state["held"]
    with held.ctx:
        if kind == "frame":
            state["args"].call(held.renderer.L.init)
        held.renderer.render(state["iterations"])
        image = held.renderer.image()
        if kind == "frame":
            held.renderer.release()
    return image


def _positions(case, seed):
    """Photon positions of a caustic: dense spots over a spread, on a shallow relief; every
    coordinate of an axis is distinct, so the tree is one and the same."""
    n = case["photons"]
    rng = np.random.default_rng(int(seed))
    spots = rng.uniform(1.0, 9.0, (24, 2))
    k = rng.integers(0, 24, n)
    xy = spots[k] + rng.normal(size=(n, 2)) * np.where(rng.uniform(size=n) < 0.6, 0.05, 0.5)[:, None]
    p = np.concatenate([xy, 2.0 + 0.1 * np.sin(xy.sum(1, keepdims=True)) + rng.uniform(0, 0.02, (n, 1))], 1)
    p = np.clip(p, 0.01, 10.0).astype(np.float32)
    for a in range(3):
        order = np.argsort(p[:, a], kind="stable")
        bits = p[order, a].view(np.int32).astype(np.int64)
        step = np.arange(n)
        bits = np.maximum.accumulate(bits - step) + step
        p[order, a] = bits.astype(np.int32).view(np.float32)
    return p


def _tree_state(case, seed):
    n = case["photons"]
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = _positions(case, seed)
    nodes = 1 << (int(math.log2(n)) + 1)
    dev = {"device": "cuda"}
    return {"kind": "kd_tree", "n": n, "positions": torch.from_numpy(p).cuda(),
            "nodes": torch.zeros((nodes, 2), dtype=torch.int32, **dev),
            "x": torch.zeros(n, **dev), "y": torch.zeros(n, **dev), "z": torch.zeros(n, **dev),
            "ids": torch.zeros(n, dtype=torch.int32, **dev)}


def _tree_pass(s):
    L = _native.lib()
    rc = L.rc_kd_build_noalloc(s["positions"].data_ptr(), s["n"], s["nodes"].data_ptr(), len(s["nodes"]),
                               s["x"].data_ptr(), s["y"].data_ptr(), s["z"].data_ptr(), s["ids"].data_ptr(),
                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError(L.rc_kd_noalloc_last_error().decode())
    return {k: s[k] for k in ("nodes", "x", "y", "z", "ids")}


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    if case["kind"] == "kd_tree":
        n = case["photons"]
        # positions in, tree order and nodes out; one comparison per photon and level
        return {"bytes": 16.0 * n + 16.0 * n + 16.0 * n, "flops": n * math.log2(n)}
    total = {"bytes": 0.0, "flops": 0.0}
    for i in range(case.get("scenes", 1)):
        size = _spread(case, "size", i) if case["scene"] == "displaced" else case["size"]
        tris = {"sphere": 20 * 4 ** size, "pool": 2 * size * size, "gems": 130 * size, "displaced": size}[case["scene"]]
        pixels = case["width"] * case["height"]
        paths = _spread(case, "paths", i)
        # every triangle record read once; per iteration the FP64 running sum read and
        # written; the image written
        total["bytes"] += 96.0 * tris + 48.0 * pixels * case["iterations"] + 12.0 * pixels
        # two rays per path, each through one box pair (24 operations) per level of the
        # tree, one triangle test (50) and one scattering event (300)
        total["flops"] += 2.0 * (paths + pixels) * case["iterations"] * (24.0 * math.log2(max(tris, 2)) + 350.0)
    return total


def exact(case, seed):
    """The photons in the order of the median-split tree, for the tree build.  A render's
    image has no value here: it is the sum over traced paths, each decided by rounding."""
    if case["kind"] != "kd_tree":
        return None
    p = _positions(case, seed)
    n = len(p)
    # level by level: the ranges of every node in one array, split at rank count / 2 along
    # the largest extent; an odd count keeps its median between the children's ranges
    order = np.arange(n)
    starts, count = np.array([0]), n
    while count > 1:
        inside = (starts[:, None] + np.arange(count)).reshape(-1)
        q = p[order[inside]].reshape(len(starts), count, 3)
        ext = q.max(1) - q.min(1)
        axis = np.argmax(ext, axis=1)
        key = np.take_along_axis(q, axis[:, None, None], 2)[:, :, 0]
        by = np.argsort(key, axis=1, kind="stable")
        order[inside] = np.take_along_axis(order[inside].reshape(len(starts), count), by, 1).reshape(-1)
        half = count // 2
        starts = np.stack([starts, starts + half + (count & 1)], 1).reshape(-1)
        count = half
    q = p[order].astype(np.float64)
    return {"nodes": None, "x": q[:, 0], "y": q[:, 1], "z": q[:, 2], "ids": None}
