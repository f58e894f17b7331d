"""What is timed on this framework: calls that a renderer, a picker or a fitting loop makes through
the Python layer over the C-ABI (barnacle_gb300.Context, Bundle, inverse.MaterialProblem).

Scenes are the procedural workloads of the repository (Bundle.generate): "cornell" (36 triangles),
"cornell-objects" (102,000 triangles, every material), "instances" (1,024 instances over 630,000
triangles), "materials" (cornell-objects with differentiable slots).  Sizes run from a single
picking query to the 16 views of the instanced workload.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np

from barnacle_gb300 import Bundle, Context, capi
from barnacle_gb300.inverse import MaterialProblem

# triangles, instances and mean rays per path (both kinds) of each scene, for work()
SCENES = {"cornell": (36, 8, 8), "cornell-objects": (102_438, 11, 8), "instances": (630_083, 1089, 4),
          "materials": (102_438, 14, 8)}
# the sizes of the instanced workload's views (seed 1), for every seed
VIEW_SIZES = [(1024, 768), (640, 480), (1600, 900), (1024, 576), (320, 240), (1920, 1080), (1280, 1024),
              (640, 360), (640, 480), (1280, 720), (1024, 576), (1600, 900), (1024, 576), (800, 600),
              (1920, 1080), (1600, 900)]


def listed():
    return [
        # an editor's pick / autofocus: a few rays into a small scene, where the call itself counts
        {"name": "trace-64-cornell", "kind": "trace", "scene": "cornell", "n": 64, "any": False, "watertight": False},
        # a batch of visibility rays of a baker over the mid-size scene, watertight, odd count
        {"name": "trace-any-131071", "kind": "trace", "scene": "cornell-objects", "n": 131_071, "any": True,
         "watertight": True},
        # a large batch of closest-hit queries (a lidar or light-probe sweep) over the instanced scene
        {"name": "trace-1000003-instances", "kind": "trace", "scene": "instances", "n": 1_000_003, "any": False,
         "watertight": False},
        # a preview frame: the smallest render, odd size, one sample, the default mode
        {"name": "render-preview", "kind": "render", "scene": "cornell", "mode": "mega", "width": 97, "height": 61,
         "spp": 1, "views": 1},
        # the Cornell workload as it is configured: 256^2, 64 spp, depth 8, the default mode
        {"name": "render-cornell", "kind": "render", "scene": "cornell", "mode": "mega", "width": 256, "height": 256,
         "spp": 64, "views": 1},
        # the mid-size scene with all materials at its configured size, a quarter frame of its samples
        {"name": "render-objects", "kind": "render", "scene": "cornell-objects", "mode": "mega", "width": 512,
         "height": 512, "spp": 32, "views": 1},
        # the instanced workload: all 16 views of their own sizes in one wavefront call
        {"name": "render-instances", "kind": "render", "scene": "instances", "mode": "wave", "width": 0, "height": 0,
         "spp": 4, "views": 16},
        # Metropolis light transport: the pssmlt workload's settings at 512^2
        {"name": "pssmlt-512", "kind": "mlt", "scene": "cornell-objects", "mode": "mega", "size": 512, "spp": 16,
         "bootstrap": 262_144, "chains": 65_536, "kelemen": True},
        # one forward render of the material-fitting loop's target (many samples)
        {"name": "fit-forward", "kind": "forward", "scene": "materials", "width": 256, "height": 256, "spp": 128},
        # one gradient of the material-fitting loop as it is configured (256^2, 16 spp, depth 8)
        {"name": "fit-gradient", "kind": "gradient", "scene": "materials", "width": 256, "height": 256, "spp": 16},
        # building a hierarchy over loose boxes (a particle or voxel scene) on the GPU
        {"name": "bvh-400000", "kind": "bvh", "scene": "boxes", "n": 400_000},
        # opening the instanced scene: upload, and the first rays through it
        {"name": "upload-instances", "kind": "upload", "scene": "instances", "n": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "render", "render", "render", "mlt", "forward", "gradient", "bvh", "upload"])
    if kind == "trace":
        return {"kind": kind, "scene": rng.choice(["cornell", "cornell-objects", "instances"]),
                "n": _log_int(rng, 64, 1_000_003), "any": rng.random() < 0.5, "watertight": rng.random() < 0.25}
    if kind == "render":
        scene = rng.choice(["cornell", "cornell-objects", "instances"])
        w, h = _log_int(rng, 48, 640), _log_int(rng, 48, 640)
        spp = _log_int(rng, 1, max(1, min(64, 8_000_000 // (w * h))))
        return {"kind": kind, "scene": scene, "mode": rng.choice(["mega", "wave"]), "width": w, "height": h, "spp": spp,
                "views": rng.choice([1, 1, 2]) if scene == "instances" else 1}
    if kind == "mlt":
        return {"kind": kind, "scene": "cornell-objects", "mode": rng.choice(["mega", "wave"]),
                "size": _log_int(rng, 64, 500), "spp": rng.randint(1, 15), "bootstrap": _log_int(rng, 4096, 262_144),
                "chains": _log_int(rng, 4096, 65_536), "kelemen": rng.random() < 0.5}
    if kind == "forward":
        return {"kind": kind, "scene": "materials", "width": _log_int(rng, 32, 256), "height": _log_int(rng, 32, 256),
                "spp": _log_int(rng, 1, 128)}
    if kind == "gradient":
        return {"kind": kind, "scene": "materials", "width": _log_int(rng, 32, 256), "height": _log_int(rng, 32, 256),
                "spp": _log_int(rng, 1, 16)}
    if kind == "bvh":
        return {"kind": kind, "scene": "boxes", "n": _log_int(rng, 300, 400_000)}
    return {"kind": kind, "scene": rng.choice(["cornell", "cornell-objects", "instances"]),
            "n": _log_int(rng, 64, 4096)}


# ------------------------------------------------------------------------------------------ inputs

def _rays(case, seed):
    """Rays as a batch of queries holds them: origins inside the scene, directions all around; any-hit
    rays end at a finite distance."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    rays = np.zeros(n, capi.RAY_DTYPE)
    if case["scene"] == "instances":
        lo, hi, reach = [-60.0, 0.1, -60.0], [60.0, 22.0, 60.0], 60.0
    else:
        lo, hi, reach = [0.05] * 3, [0.95] * 3, 1.2
    rays["origin"] = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    rays["direction"] = d / np.sqrt((d ** 2).sum(1, dtype=np.float32))[:, None]
    rays["t_max"] = rng.uniform(0.05, 1.0, n).astype(np.float32) * np.float32(reach) if case.get("any") else np.inf
    return rays


def _boxes(n, seed):
    """A cloud of boxes in the order and the unit (a power of two) of the seed: the tree then has the
    same number of nodes for every seed, so that builds of several seeds can be laid side by side."""
    rng = np.random.default_rng(n)
    centre = rng.normal(size=(n, 3)) * [40.0, 10.0, 40.0]
    half = np.exp(rng.normal(size=(n, 3)) * 0.7 - 2.0)
    boxes = np.concatenate([centre - half, centre + half], axis=1).astype(np.float32)
    rng = np.random.default_rng(seed)
    return boxes[rng.permutation(n)] * np.float32(2.0 ** int(rng.integers(-8, 9)))


def _scene(case, seed):
    b = Bundle.generate(case["scene"], 1 + seed % 1000)
    ctx = Context(0)
    ctx.upload(b)
    return ctx, b


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        ctx, b = _scene(case, seed)
        flags = (capi.BN_TRACE_ANY if case["any"] else 0) | (capi.BN_TRACE_WATERTIGHT if case["watertight"] else 0)
        return {"kind": kind, "ctx": ctx, "bundle": b, "rays": _rays(case, seed), "flags": flags}
    if kind in ("render", "mlt"):
        ctx, b = _scene(case, seed)
        d = b.render
        d.spp = case["spp"]
        d.frame_id = seed % 4096
        d.mode = capi.BN_MODE_WAVEFRONT if case["mode"] == "wave" else capi.BN_MODE_MEGAKERNEL
        views = b.views[: case.get("views", 1)]
        w, h = case.get("width", 0), case.get("height", 0)
        if kind == "mlt":
            w = h = case["size"]
            d.integrator = capi.BN_INTEGRATOR_PSSMLT
            d.n_bootstrap, d.n_chains = case["bootstrap"], case["chains"]
            d.large_step_prob = 0.3
            d.mutation = capi.BN_MUTATION_KELEMEN if case["kelemen"] else capi.BN_MUTATION_GAUSSIAN
            d.sigma, d.eps_min, d.eps_max = 1e-2, 1.0 / 1024.0, 1.0 / 64.0
        for i, v in enumerate(views):
            v.width, v.height = (w, h) if w else VIEW_SIZES[i]
        return {"kind": kind, "ctx": ctx, "bundle": b, "desc": d, "views": views}
    if kind in ("forward", "gradient"):
        b = Bundle.generate(case["scene"], 1 + seed % 1000)
        ctx = Context(0)
        problem = MaterialProblem(ctx, b, case["width"], case["height"], case["spp"])
        s = {"kind": kind, "ctx": ctx, "problem": problem, "frame": seed % 4096,
             "params": problem.project(problem.random_params(seed))}
        if kind == "gradient":  # the picture to fit: the scene's own materials, other samples
            s["target"] = problem.render(b.slot_params(), spp=64, frame=4096 + seed % 4096)
        return s
    if kind == "bvh":
        return {"kind": kind, "ctx": Context(0), "boxes": _boxes(case["n"], seed)}
    b = Bundle.generate(case["scene"], 1 + seed % 1000)
    return {"kind": kind, "ctx": Context(0), "bundle": b, "rays": _rays(case, seed),
            "n_instances": b.scene.contents.n_instances}


# --------------------------------------------------------------------------------------- one pass

def _hits(h, any_hit):
    # an any-hit query answers whether something is in the way, a closest-hit one with the whole record
    names = ("t", "instance") if any_hit else ("t", "u", "v", "instance", "primitive", "normal", "position")
    return {k: h[k] for k in names}


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "trace":
        return _hits(ctx.trace(state["rays"], state["flags"]), state["flags"] & capi.BN_TRACE_ANY)
    if kind in ("render", "mlt"):
        return ctx.render(state["desc"], state["views"])
    if kind == "forward":
        return state["problem"].render(state["params"], frame=state["frame"])
    if kind == "gradient":
        loss, grad = state["problem"].loss_and_grad(state["params"], state["target"], frame=state["frame"])
        # the optimiser's parameters are float32, and so is the gradient that it is handed
        return {"loss": loss, "grad": grad.astype(np.float32)}
    if kind == "bvh":
        nodes, perm = ctx.bvh_build(state["boxes"])
        return {"perm": perm, **{k: nodes[k] for k in nodes.dtype.names}}
    ctx.upload(state["bundle"])
    return {"order": ctx.instance_order(state["n_instances"]), **_hits(ctx.trace(state["rays"]), False)}


# --------------------------------------------------------------------------- what a pass needs at least

def _ray_flops(scene):
    # a walk down both levels, two boxes of 18 operations a step, then one triangle and a transform
    tris, insts, _ = SCENES[scene]
    return 36.0 * (math.log2(insts) + math.log2(max(2, tris / 4))) + 60.0 + 40.0


def _scene_bytes(scene):
    tris, insts, _ = SCENES[scene]
    return 48.0 * tris + 32.0 * tris + 152.0 * insts  # triangles, a node per triangle, instances




def _paths(case):
    if case["kind"] == "mlt":
        return float(case["bootstrap"] + case["chains"] + case["spp"] * case["size"] ** 2)
    pixels = case["width"] * case["height"] * case.get("views", 1) or sum(x * y for x, y in VIEW_SIZES)
    return float(pixels * case["spp"])


def work(case):
    kind, scene = case["kind"], case["scene"]
    if kind == "trace":
        ray = ctypes.sizeof(capi.bn_ray)
        return {"bytes": case["n"] * (ray + (8 if case["any"] else ctypes.sizeof(capi.bn_hit))) + _scene_bytes(scene),
                "flops": case["n"] * _ray_flops(scene)}
    if kind == "bvh":
        n = case["n"]
        # each box in, each node and index out; every level reads the boxes and bins them
        return {"bytes": n * (24.0 + 4.0) + n * 32.0, "flops": n * 30.0 * max(1.0, math.log2(n / 4))}
    if kind == "upload":
        tris, insts, _ = SCENES[scene]
        return {"bytes": tris * (6.0 + 12.0) + _scene_bytes(scene) + case["n"] * 72.0,
                "flops": tris * 30.0 * math.log2(max(2, tris / 4)) + case["n"] * _ray_flops(scene)}
    rays = SCENES[scene][2] * _paths(case)
    shade = 400.0 * rays / 2
    pixels = case["size"] ** 2 if kind == "mlt" else _paths(case) / case["spp"]
    passes = 2.0 if kind == "gradient" else 1.0  # the image, then its adjoint over the same paths
    return {"bytes": _scene_bytes(scene) + 12.0 * pixels * (2 if kind == "gradient" else 1),
            "flops": rays * _ray_flops(scene) + passes * shade}


# ------------------------------------------------------------------------------ the same in 64 bits

def _world_triangles(b):
    """Every triangle of a scene of mesh instances in world space, in 64 bits."""
    s = b.scene.contents
    out = []
    for i in range(s.n_instances):
        inst = s.instances[i]
        mesh = s.meshes[s.primitives[inst.primitive].mesh]
        v = np.ctypeslib.as_array(mesh.vertices, (mesh.n_vertices, 3)).astype(np.float64)
        k = np.ctypeslib.as_array(mesh.indices, (mesh.n_triangles, 3))
        m = np.array(list(inst.object_to_world), np.float64).reshape(4, 4)
        w = v @ m[:3, :3] + m[3, :3]
        # the shading normal follows the object-space frame: its tangents go through the matrix
        e0, e1 = v[k[:, 1]] - v[k[:, 0]], v[k[:, 2]] - v[k[:, 0]]
        n = np.cross(e0, e1)
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        axis = np.where(np.abs(n[:, :1]) > np.float32(0.1), [[0.0, 1.0, 0.0]], [[1.0, 0.0, 0.0]])
        t = np.cross(n, axis)
        t /= np.linalg.norm(t, axis=1, keepdims=True)
        bt = np.cross(n, t)
        t, bt = t @ m[:3, :3], bt @ m[:3, :3]
        t /= np.linalg.norm(t, axis=1, keepdims=True)
        bt /= np.linalg.norm(bt, axis=1, keepdims=True)
        out.append((w[k[:, 0]], w[k[:, 1]], w[k[:, 2]], np.cross(t, bt)))
    return [np.concatenate(x) for x in zip(*out)]


def exact(case, seed):
    """Closest hits in the small scene by testing every triangle.  Renders, chains and fits are sums over
    random walks whose turns follow the last bits of 32-bit arithmetic: they have no other value in 64
    bits than that of other walks.  Builds return copies of their inputs and whole numbers."""
    if case["kind"] != "trace" or case["scene"] != "cornell" or case["any"] or case["n"] > 200_000:
        return None
    b = Bundle.generate(case["scene"], 1 + seed % 1000)
    p0, p1, p2, normal = _world_triangles(b)
    r = _rays(case, seed)
    o, d = r["origin"].astype(np.float64), r["direction"].astype(np.float64)
    n = len(r)
    t, u, v, tri = np.full(n, np.inf), np.zeros(n), np.zeros(n), np.full(n, -1)
    for j in range(len(p0)):
        e0, e1, s = p1[j] - p0[j], p2[j] - p0[j], o - p0[j]
        c = np.cross(d, e1)
        with np.errstate(divide="ignore", invalid="ignore"):
            inv = 1.0 / (c @ e0)
            uu = inv * (s * c).sum(1)
            q = np.cross(s, e0)
            vv = inv * (d * q).sum(1)
            tt = inv * (q @ e1)
            hit = (uu >= 0) & (vv >= 0) & (uu + vv <= 1) & (tt > 1e-3) & (tt < t)
        t, u, v, tri = np.where(hit, tt, t), np.where(hit, uu, u), np.where(hit, vv, v), np.where(hit, j, tri)
    found = (tri >= 0)[:, None]
    position = np.where(found, o + np.where(found[:, 0], t, 0.0)[:, None] * d, 0.0)
    return {"t": t, "u": u, "v": v, "instance": None, "primitive": None,
            "normal": np.where(found, normal[tri], 0.0), "position": position}
