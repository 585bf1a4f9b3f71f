"""The work a user of the probe-update library has it do, as timed cases.

Every case goes through the calls a renderer or a training program makes:
whole and scheduled probe updates (`Context.update`,
`IrradianceProbes.update`), moving instances followed by an update, recorded
updates with their reverse pass, several volumes in one batch, loading a
scene, and the final gather that reads the atlases.  Outputs are the atlases
(zero-copy views of device memory), gradients and images.

The seed of a case draws what changes between a program's calls: the ray-set
rotations, the light, the albedos, the atlases and probe states left by
earlier frames, instance motion, G-buffers.  The geometry of a case is fixed
by the case itself, like a level's.

`exact` restates a case in 64 bits with plain torch for the room scenes
(boxes, traced analytically) and for the final gather.
"""
import functools
import math

import numpy as np
import torch

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Batch, Context, IrradianceProbes

FP32, BF16 = abi.PRECISION_FP32, abi.PRECISION_BF16
FRAMES = 16  # rotations (and instance motions) a state cycles through


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def room(boxes):
    return {"scene": "room", "boxes": boxes}


def terrain(cells, instances, boxes):
    return {"scene": "terrain", "cells": cells, "instances": instances, "boxes": boxes}


def grid(nx, ny, nz, rays, precision, color=8, depth=16):
    return {"nx": nx, "ny": ny, "nz": nz, "rays": rays, "precision": precision, "color": color, "depth": depth}


def listed():
    return [
        # one room of a small level refreshed every frame: latency and launches count
        dict(name="update_room_8x8x8", op="update", **room(200), **grid(8, 8, 8, 128, FP32)),
        # an odd grid, an odd ray count and the smaller tiles, 16-bit atlas
        dict(name="update_room_odd_bf16", op="update", **room(300), **grid(13, 7, 11, 100, BF16, 6, 14)),
        # the benchmark's open world: 4097 instances, 1M unique triangles, whole grid, 16-bit atlas ...
        dict(name="update_terrain_bf16", op="update", **terrain(512, 4096, 5000), **grid(32, 16, 32, 256, BF16)),
        # ... and the FP32 atlas
        dict(name="update_terrain_fp32", op="update", **terrain(512, 4096, 5000), **grid(32, 16, 32, 256, FP32)),
        # the reference class's own frame: classified probes, its default 192 rays, the
        # schedule's choice of probes, the hysteresis ramp
        dict(name="frame_terrain", op="frame", cap=0, **terrain(256, 1024, 2000), **grid(32, 16, 32, 192, FP32)),
        # a frame with a budget (ProbesPerUpdate) in an indoor scene
        dict(name="frame_room_budget", op="frame", cap=333, **room(500), **grid(16, 8, 16, 192, BF16)),
        # a frame of an indoor scene whose furniture moves: top-level refit, then the update
        dict(name="move_room", op="move", moving=64, rebuild=False, **room(1000), **grid(16, 8, 16, 128, FP32)),
        # fitting albedos and lights: eight recorded updates and their reverse pass
        dict(name="learn_room", op="learn", updates=8, **room(1000), **grid(16, 8, 16, 256, FP32)),
        # an editor or a server with many volumes, updated together
        dict(name="batch_12_volumes", op="batch", volumes=12, first=0),
        # loading a level: trees, probe classification, the first update
        dict(name="load_terrain", op="load", build="fast_trace", **terrain(512, 512, 5000),
             **grid(16, 8, 16, 128, BF16)),
        # the renderer's read of the atlases: a full-HD view, and a ragged preview
        dict(name="gather_1080p_bf16", op="gather", width=1920, height=1080, view="camera", reflection=True,
             **grid(32, 16, 32, 256, BF16)),
        dict(name="gather_643x361_fp32", op="gather", width=643, height=361, view="scattered", reflection=False,
             **grid(13, 7, 11, 128, FP32)),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    tiles = rng.choice([(8, 16), (8, 16), (6, 14), (7, 15)])
    op = rng.choice(["update", "update", "frame", "move", "learn", "batch", "load", "gather"])
    if op == "batch":
        return {"op": "batch", "volumes": rng.randint(2, 6), "first": rng.randint(1, 12)}
    outdoor = op in ("update", "frame", "load") and rng.random() < 0.5
    if op == "learn":
        g = grid(log(4, 16), log(3, 8), log(4, 16), rng.choice([64, 100, 192, 256]), FP32, *tiles)
        return dict(op="learn", updates=rng.randint(1, 8), **room(log(20, 1000)), **g)
    g = grid(log(4, 32), log(3, 16), log(4, 32), rng.choice([32, 64, 100, 128, 144, 192, 256]),
             rng.choice([FP32, BF16]), *tiles)
    if op == "gather":
        w = log(160, 1920)
        return dict(op="gather", width=w, height=max(1, w * 9 // 16 + rng.randint(-3, 0)),
                    view=rng.choice(["camera", "scattered"]), reflection=rng.random() < 0.5, **g)
    s = terrain(log(48, 256), log(16, 2048), log(50, 3000)) if outdoor else room(log(10, 2000))
    if op == "frame":
        return dict(op="frame", cap=rng.choice([0, log(16, 2000)]), **s, **g)
    if op == "move":
        return dict(op="move", moving=min(s["boxes"], log(1, 500)), rebuild=rng.random() < 0.3, **s, **g)
    if op == "load":
        return dict(op="load", build=rng.choice(["fast_trace", "fast_trace", "fast_build"]), **s, **g)
    return dict(op="update", **s, **g)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _room_geometry(boxes):
    sc = scenes.room_with_boxes(1234, boxes)
    sc.bounds = (np.zeros(3), np.array([10.0, 6.0, 10.0]))  # the grid spans the room
    return sc


@functools.lru_cache(maxsize=3)
def _terrain_geometry(cells, instances, boxes):
    return scenes.terrain_with_clusters(1235, n_instances=instances, boxes_per_cluster=boxes, cells=cells,
                                        size=cells * 0.5)


@functools.lru_cache(maxsize=2)
def _volume_geometry(first, count):
    return scenes.batch_workloads(count=first + count)[first:]


def _scene(case, rng):
    """The case's geometry with the seed's albedos."""
    if case["scene"] == "room":
        g = _room_geometry(case["boxes"])
    else:
        g = _terrain_geometry(case["cells"], case["instances"], case["boxes"])
    m = g.materials.copy()
    m["base_color"] = rng.uniform(0.1, 0.9, size=(len(m), 3))
    return scenes.Scene(g.vertices, g.indices, g.meshes, g.instances, g.offsets, m, g.bounds)


def _grid_desc(case, bounds):
    lo, hi = bounds
    return abi.make_grid(lo.astype(np.float32), hi.astype(np.float32), (case["nx"], case["ny"], case["nz"]),
                         case["rays"], case["color"], case["depth"], precision=case["precision"])


def _light(rng):
    d = np.array([rng.uniform(-0.6, 0.6), 1.0, rng.uniform(-0.6, 0.6)])
    return abi.make_light(d / np.linalg.norm(d), rng.uniform(2.0, 4.0, 3), rng.uniform(0.3, 0.8, 3))


def _rotations(seed, n=FRAMES):
    return [scenes.random_orientation(seed, k) for k in range(n)]


def _atlases(g, seed):
    """Atlases as earlier frames leave them: every probe has its own tint and
    depth, every texel a little of its own; values a 16-bit atlas holds."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    out = []
    for kind in (abi.ATLAS_COLOR, abi.ATLAS_DEPTH):
        h, w, c = g.atlas_shape(kind)
        side = g.color_res if kind == abi.ATLAS_COLOR else g.depth_res
        base = torch.rand((h // side, w // side, 4), device="cuda", generator=gen)
        base = base.repeat_interleave(side, 0).repeat_interleave(side, 1)
        own = torch.rand((h, w, 4), device="cuda", generator=gen)
        if kind == abi.ATLAS_COLOR:
            t = 0.05 + 0.5 * base + 0.1 * own
            t[..., 3] = 1.0
        else:
            e = [(b - a) / (r - 1) for a, b, r in zip(g.extent_min, g.extent_max, g.resolution)]
            cell = math.sqrt(sum(x * x for x in e))
            mean = cell * (0.25 + 0.6 * base[..., 0] + 0.15 * own[..., 0])
            t = torch.stack([mean, mean * mean * (1.0 + 0.2 * own[..., 1])], -1)
        out.append(t.half().float().cpu().numpy())
    return out


def _set_atlases(ctx, seed):
    c, d = _atlases(ctx.grid, seed)
    ctx.set_atlas(abi.ATLAS_COLOR, c)
    ctx.set_atlas(abi.ATLAS_DEPTH, d)


def _states(g, seed):
    """Probe states of a game that has run a while (0 off, 1..8 refresh period)."""
    return np.random.default_rng([int(seed), 3]).choice(
        np.arange(9, dtype=np.uint32), size=g.probe_count(),
        p=[0.1, 0.35, 0.1, 0.1, 0.1, 0.05, 0.05, 0.05, 0.1]).astype(np.uint32)


def _motion(case, scene, rng):
    """FRAMES transforms of the first `moving` boxes: drift and turn."""
    m = case["moving"]
    base = scene.instances["transform"][1:1 + m].astype(np.float64).reshape(m, 3, 4)
    step, turn = rng.uniform(-0.05, 0.05, (m, 3)), rng.uniform(-0.1, 0.1, m)
    out = []
    for k in range(1, FRAMES + 1):
        t = base.copy()
        c, s, z = np.cos(turn * k), np.sin(turn * k), np.zeros(m)
        R = np.stack([np.stack([c, z, s], -1), np.stack([z, z + 1, z], -1), np.stack([-s, z, c], -1)], 1)
        t[:, :, :3] = R @ t[:, :, :3]
        t[:, :, 3] += step * k
        out.append(t.reshape(m, 12).astype(np.float32))
    return np.arange(1, m + 1, dtype=np.uint32), out


def _gbuffer(case, seed):
    """G-buffer on the GPU: a camera view over rolling ground under a sky, or
    (scattered) pixels that share nothing with their neighbours."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    h, w, n = case["height"], case["width"], case["height"] * case["width"]

    def u(*shape):
        return torch.rand(shape, device="cuda", generator=gen)

    if case["view"] == "camera":
        y, x = torch.meshgrid(torch.linspace(1, -1, h, device="cuda"), torch.linspace(-1, 1, w, device="cuda"),
                              indexing="ij")
        ph = 6.28 * u(2)
        d = torch.stack([0.9 * x, 0.55 * y - 0.35, torch.ones_like(x)], -1)
        d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)
        eye = torch.tensor([5.0, 3.5, 0.3], device="cuda")
        t = torch.where(d[:, 1] < -0.05, -3.2 / d[:, 1].clamp(max=-0.05), torch.zeros(n, device="cuda"))
        pos = eye + t[:, None] * d
        pos[:, 1] += 0.25 * torch.sin(pos[:, 0] * 1.7 + ph[0]) * torch.sin(pos[:, 2] * 1.3 + ph[1])
        nx = -0.4 * torch.cos(pos[:, 0] * 1.7 + ph[0])
        nz = -0.3 * torch.cos(pos[:, 2] * 1.3 + ph[1])
        nrm = torch.stack([nx, torch.ones_like(nx), nz], -1)
        depth = torch.where((t > 0) & (t < 12.0), t, torch.zeros_like(t))
        origin = [5.0, 3.5, 0.3]
    else:
        pos = u(n, 3) * torch.tensor([10.0, 6.0, 10.0], device="cuda")
        nrm = torch.randn((n, 3), device="cuda", generator=gen)
        depth = torch.where(u(n) < 0.1, 0.0, 1.0)
        origin = [5.0, 3.0, 5.0]
    gb = {"position_depth": torch.cat([pos, depth[:, None]], 1), "normal_metalness": torch.cat([nrm, u(n, 1)], 1),
          "albedo_roughness": torch.cat([u(n, 3), 0.2 + 0.8 * u(n, 1)], 1), "emissive": 0.1 * u(n, 4)}
    gb = {k: v.reshape(h, w, 4).contiguous() for k, v in gb.items()}
    gb["direct_light"] = u(h, w)
    if case["reflection"]:
        gb["reflection"] = u(h, w, 4)
    return gb, origin


class _DeviceArray:
    """Device memory of `owner`, which lives as long as the tensor over it."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _views(ctx):
    """The context's atlases where they are: what a renderer binds."""
    typestr = "<f2" if ctx.grid.precision == BF16 else "<f4"
    return [torch.as_tensor(_DeviceArray(ctx, ctx.atlas_device_ptr(kind), ctx.atlas_shape(kind), typestr),
                            device="cuda")
            for kind in (abi.ATLAS_COLOR, abi.ATLAS_DEPTH)]


def prepare(case, seed):
    op = case["op"]
    rng = np.random.default_rng([int(seed), 17])
    s = {"op": op, "k": 0, "rotations": _rotations(seed)}
    if op == "batch":
        ws = _volume_geometry(case["first"], case["volumes"])
        s["contexts"] = []
        for v, w in enumerate(ws):
            ctx = Context(w.grid)
            ctx.build_scene(w.scene)
            ctx.set_light(_light(rng))
            _set_atlases(ctx, seed + v)
            s["contexts"].append(ctx)
        s["batch"] = Batch(s["contexts"])
        s["rotations"] = [np.stack([scenes.random_orientation(seed + 31 * v, k) for v in range(len(ws))])
                          for k in range(FRAMES)]
        return s
    if op == "gather":
        s["ctx"] = Context(_grid_desc(case, (np.zeros(3), np.array([10.0, 6.0, 10.0]))))
        s["ctx"].set_light(_light(rng))
        _set_atlases(s["ctx"], seed)
        s["ctx"].set_probe_states(_states(s["ctx"].grid, seed))
        s["gbuffer"], s["origin"] = _gbuffer(case, seed)
        s["out"] = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        return s
    scene = _scene(case, rng)
    g = _grid_desc(case, scene.bounds)
    if op == "frame":
        p = IrradianceProbes()
        p.GridParameters = g
        p.ProbesPerUpdate = case["cap"]
        p.init(*[b.astype(np.float32) for b in scene.bounds])
        p.setScene(scene)
        p.setLightBuffer(_light(rng))
        if case["scene"] == "terrain":
            p.initProbes(s["rotations"][-1])
        else:
            p.ctx.set_probe_states(_states(g, seed))
        _set_atlases(p.ctx, seed)
        s["probes"] = p
        return s
    ctx = s["ctx"] = Context(g)
    if op == "load":
        ctx.set_build_mode(case["build"])
        s["scene"] = scene
    else:
        ctx.build_scene(scene)
    ctx.set_light(_light(rng))
    _set_atlases(ctx, seed)
    if op == "move":
        s["ids"], s["motion"], s["rebuild"] = *_motion(case, scene, rng), case["rebuild"]
    if op == "learn":
        s["updates"], s["materials"] = case["updates"], len(scene.materials)
        s["grad"] = rng.standard_normal(ctx.atlas_shape(abi.ATLAS_COLOR), np.float32)
        s["rotations"] = [np.stack(_rotations(seed + 1000 * k, case["updates"])) for k in range(4)]
    return s


def run(s):
    op, k = s["op"], s["k"] % len(s["rotations"])
    rotation = s["rotations"][k]
    s["k"] += 1
    if op == "update":
        s["ctx"].update(rotation)
        return _views(s["ctx"])
    if op == "frame":
        s["probes"].update(rotation)
        return _views(s["probes"].ctx)
    if op == "gather":
        s["ctx"].final_gather(s["gbuffer"], s["origin"], s["out"])
        return s["out"]
    if op == "move":
        s["ctx"].update_instances(s["motion"][k], s["ids"], rebuild=s["rebuild"])
        s["ctx"].update(rotation)
        return _views(s["ctx"])
    if op == "learn":
        s["ctx"].forward_record(rotation, 2)
        return [*s["ctx"].backward(s["grad"], s["materials"]), *_views(s["ctx"])]
    if op == "batch":
        s["batch"].update(rotation)
        return [_views(c) for c in s["contexts"]]
    s["ctx"].build_scene(s["scene"])
    s["ctx"].init_probes(s["rotations"][-1])
    s["ctx"].update(rotation)
    return _views(s["ctx"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
LOOKUP = 8 * 60  # operations of one eight-probe atlas lookup


def _update_work(probes, rays, color, depth, precision, triangles, instances, listed_probes=None):
    """Scene and atlases read once, atlases written once; a ray's walk down
    one path of balanced trees (two box tests a level), one triangle test, the
    shading of its hit with two lookups; the blend."""
    p = probes if listed_probes is None else listed_probes
    n = p * rays
    half = precision == BF16
    # FP32 atlas: read + write; 16-bit: read, write, and its 32-bit accumulator read and written
    texel = (8 + 8 + 32, 4 + 4 + 16) if half else (32, 16)
    levels = math.log2(max(triangles, 2)) + math.log2(max(instances, 2))
    nc, nd = (color - 2) ** 2, (depth - 2) ** 2
    return {"bytes": triangles * 48 + instances * 64 + p * (color ** 2 * texel[0] + depth ** 2 * texel[1]),
            "flops": n * (levels * 24 + 60 + 2 * LOOKUP + 2 * (nc * 3 + nd * 2))}


def work(case):
    op = case["op"]
    if op == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for w in _volume_geometry(case["first"], case["volumes"]):
            g = w.grid
            one = _update_work(g.probe_count(), g.rays_per_probe, g.color_res, g.depth_res, g.precision,
                               w.scene.unique_triangle_count, len(w.scene.instances))
            total = {k: total[k] + one[k] for k in total}
        return total
    probes = case["nx"] * case["ny"] * case["nz"]
    if op == "gather":
        px = case["width"] * case["height"]
        half = case["precision"] == BF16
        atlas = probes * (case["color"] ** 2 * (8 if half else 16) + case["depth"] ** 2 * (4 if half else 8))
        return {"bytes": px * (16 * (5 + case["reflection"]) + 4) + atlas, "flops": px * (LOOKUP + 150)}
    if case["scene"] == "room":
        triangles, instances = 24, case["boxes"] + 1
    else:
        triangles, instances = 2 * case["cells"] ** 2 + 8 * 12 * case["boxes"], case["instances"] + 1
    chosen = probes
    if op == "frame":
        chosen = min(case["cap"] or probes, probes) if case["cap"] else probes // 4
    one = _update_work(probes, case["rays"], case["color"], case["depth"], case["precision"], triangles, instances,
                       chosen)
    if op == "learn":
        return {k: 3 * case["updates"] * v for k, v in one.items()}
    if op == "load":  # vertices and indices read, nodes written; 512 classification rays a probe
        one["bytes"] += triangles * (12 + 32 + 64 + 48)
        one["flops"] += triangles * math.log2(triangles) * 60 + probes * 512 * 24 * math.log2(triangles * instances)
    return one


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
PI = 3.1415926538


def _f64(x):
    return torch.as_tensor(np.asarray(x, np.float64), device="cuda")


def _directions(m, n):
    """The ray table: float by definition, operation by operation."""
    f = np.float32
    i = np.arange(n, dtype=f)
    a = i * (np.sqrt(f(5.0)) * f(0.5) + f(0.5) - f(1.0))
    phi = (f(2.0) * f(PI)) * (a - np.floor(a))
    ct = f(1.0) - (f(2.0) * i + f(1.0)) * (f(1.0) / f(n))
    st = np.sqrt(np.clip(f(1.0) - ct * ct, f(0.0), f(1.0)))
    v = [np.cos(phi.astype(np.float64)).astype(f) * st, np.sin(phi.astype(np.float64)).astype(f) * st, ct]
    m = np.asarray(m, f).reshape(3, 3)
    return _f64(np.stack([(m[r, 0] * v[0] + m[r, 1] * v[1]) + m[r, 2] * v[2] for r in range(3)], -1))


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _oct_uv(d):
    s = torch.sign(d)
    o = d / (d * s).sum(-1, keepdim=True)
    fold = s[..., :2] * (1.0 - o.abs()[..., [1, 0]])
    return torch.where(o[..., 2:] < 0, fold, o[..., :2]) * 0.5 + 0.5


def _texel_directions(side):
    n = side - 2
    scale = float(np.float32(0.33333 if n == 6 else 0.142857 if n == 14 else 2.0 / n))
    c = scale * (torch.arange(n, dtype=torch.float64, device="cuda") - 0.5 * (n - 1))
    y, x = torch.meshgrid(c, c, indexing="ij")
    v = torch.stack([x, y, 1.0 - x.abs() - y.abs()], -1)
    fold = (1.0 - v[..., [1, 0]].abs()) * torch.where(v[..., :2] >= 0, 1.0, -1.0)
    v = torch.cat([torch.where(v[..., 2:] < 0, fold, v[..., :2]), v[..., 2:]], -1)
    return _unit(v).reshape(-1, 3)


def _bilinear(tex, u, v):
    h, w = tex.shape[:2]
    x, y = u * w - 0.5, v * h - 0.5
    i, j = x.floor(), y.floor()
    ax, ay = (x - i)[..., None], (y - j)[..., None]
    i, j = i.long().clamp(min=0), j.long().clamp(min=0)
    i1, j1 = (i + 1).clamp(max=w - 1), (j + 1).clamp(max=h - 1)
    top = tex[j, i] * (1 - ax) + tex[j, i1] * ax
    return top * (1 - ay) + (tex[j1, i] * (1 - ax) + tex[j1, i1] * ax) * ay


class _Grid64:
    def __init__(self, g):
        self.g, self.res = g, [int(r) for r in g.resolution]
        lo, hi = (np.array(list(e), np.float32) for e in (g.extent_min, g.extent_max))
        self.lo = _f64(lo)
        self.cell = _f64((hi - lo) / np.float32([r - 1 for r in self.res]))
        self.cell_len = float(self.cell.norm())
        self.tmax = float(np.linalg.norm((hi - lo).astype(np.float64)))

    def probes(self):
        x, y, z = self.res
        p = torch.arange(x * y * z, device="cuda")
        return torch.stack([p % x, p % (x * y) // x, p // (x * y)], -1)


def _lookup(G, pos, nrm, cam, states, color, depth):
    """Irradiance at `pos` towards `nrm` from the eight probes around it."""
    g, (rx, ry, rz) = G.g, G.res
    at = (pos - G.lo) / G.cell
    inside = (at >= 0).all(-1)
    f = at.clamp(min=0).floor().long()
    alpha = ((pos - (f * G.cell + G.lo)) / G.cell).clamp(0, 1)
    biased = pos + (nrm + cam) * float(g.shadow_bias)
    nuv = _oct_uv(nrm)
    fc = fb = torch.zeros_like(pos)
    tw = tf = torch.zeros(len(pos), dtype=torch.float64, device="cuda")
    limit = torch.tensor([rx - 1, ry - 1, rz - 1], device="cuda")
    for i in range(8):
        o = torch.tensor([i & 1, i >> 1 & 1, i >> 2], device="cuda")
        p = f + o
        ok = (p <= limit).all(-1)
        p = torch.minimum(p, limit)
        ok = ok & (states[p[:, 0] + rx * p[:, 1] + rx * ry * p[:, 2]] != 0)
        pp = p * G.cell + G.lo
        to = _unit(pp - pos)
        tile = p[:, 1] * rx + p[:, 0]
        tri = torch.where(o == 1, alpha, 1 - alpha).prod(-1) + 0.001
        away = pp - biased
        dist = away.norm(dim=-1)
        duv = _oct_uv(-away / dist[:, None])

        def uv(side, q):
            return ((side * tile + 1) / side + (side - 2) / side * q[:, 0]) / (rx * ry), \
                   ((side * p[:, 2] + 1) / side + (side - 2) / side * q[:, 1]) / rz

        facing = (((to * nrm).sum(-1) + 1) * 0.5).clamp(min=0.0001)
        w = wf = facing * facing + 0.2
        dd = _bilinear(depth, *uv(g.depth_res, duv))
        var = (dd[:, 0] ** 2 - dd[:, 1]).abs()
        dm = (dist - dd[:, 0]).clamp(min=0.0001)
        cheb = (var / (var + dm * dm)) ** 3
        w = (w * torch.where(dist <= dd[:, 0], 1.0, cheb)).clamp(min=0.000001)
        w = torch.where(w < 0.2, w * w * w * 25.0, w) * tri
        wf = wf * tri
        zero = torch.zeros_like(w)
        w, wf = torch.where(ok, w, zero), torch.where(ok, wf, zero)
        c = _bilinear(color[..., :3], *uv(g.color_res, nuv)).sqrt()
        fc, fb, tw, tf = fc + c * w[:, None], fb + c * wf[:, None], tw + w, tf + wf
    fc = fc / torch.where(tw > 1e-3, tw, 1.0)[:, None]
    fb = fb / torch.where(tf > 1e-3, tf, 1.0)[:, None]
    k = (8.0 * tw.clamp(0, 0.125))[:, None]
    return torch.where(inside[:, None], fb * fb * (1 - k) + fc * fc * k, 0.0)


def _sun(n, v, light, to_sun, albedo, metal, rough):
    spec = 0.04 * (1 - metal) + albedo * metal
    r90 = (spec.amax(-1, keepdim=True) * 25).clamp(0, 1)
    l = _unit(to_sun)
    h = _unit(l + v)
    nl = (n * l).sum(-1, keepdim=True).clamp(0.001, 1)
    nv = (n * v).sum(-1, keepdim=True).abs().clamp(0.001, 1)
    nh = (n * h).sum(-1, keepdim=True).clamp(0, 1)
    vh = (v * h).sum(-1, keepdim=True).clamp(0, 1)
    F = spec + (r90 - spec) * (1 - vh).clamp(0, 1) ** 5
    al = rough * rough
    a2 = al * al
    G = 2 * nl / (nl + (a2 + (1 - a2) * nl * nl).sqrt()) * 2 * nv / (nv + (a2 + (1 - a2) * nv * nv).sqrt())
    a = nh * al
    D = ((al / ((1 - nh * nh) + a * a)) ** 2 / PI).clamp(0, 4)
    return light * ((1 - F) * albedo * 0.96 * (1 - metal) / PI + F * (G * D / (4 * nl * nv))) * nl


class _Room64:
    """The room and its boxes as slabs in object space."""

    def __init__(self, scene, transforms):
        t = transforms.astype(np.float64).reshape(-1, 3, 4)
        inv = np.linalg.inv(t[:, :, :3])
        self.A = _f64(inv)
        self.b = _f64(-np.einsum("nij,nj->ni", inv, t[:, :, 3]))
        n = len(t)
        lo, hi = np.full((n, 3), -0.5), np.full((n, 3), 0.5)
        lo[0], hi[0] = 0.0, (10.0, 6.0, 10.0)  # the room itself, seen from inside
        self.lo, self.hi = _f64(lo), _f64(hi)
        self.material = torch.as_tensor(scene.offsets["material_index"].astype(np.int64), device="cuda")

    def hit(self, o, d, tmin, tmax):
        """(t, object, axis, side, leaving) of the closest hit; t = inf on a miss."""
        out = []
        for q in range(0, len(o), 1 << 15):
            oo = torch.einsum("nij,rj->rni", self.A, o[q:q + (1 << 15)]) + self.b
            od = torch.einsum("nij,rj->rni", self.A, d[q:q + (1 << 15)])
            od = torch.where(od == 0, 1e-30, od)
            t0, t1 = (self.lo - oo) / od, (self.hi - oo) / od
            near, na = torch.minimum(t0, t1).max(-1)
            far, fa = torch.maximum(t0, t1).min(-1)
            ok = near <= far
            inf = torch.full_like(near, math.inf)
            enter = torch.where(ok & (near >= tmin) & (near <= tmax), near, inf)
            leave = torch.where(ok & (far >= tmin) & (far <= tmax), far, inf)
            t = torch.minimum(enter, leave)
            best, k = t.min(-1)
            r = torch.arange(len(k), device="cuda")
            out_ = leave[r, k] < enter[r, k]
            axis = torch.where(out_, fa[r, k], na[r, k])
            side = torch.sign(od[r, k, axis]) * torch.where(out_, 1.0, -1.0)
            out.append((best, k, axis, side, out_))
        return [torch.cat(v) for v in zip(*out)]


def _update64(G, geo, light, albedo, sky, sun, rotation, probes, states, color, depth, hyst):
    """One update of the listed probes; the new atlases."""
    g, R = G.g, int(G.g.rays_per_probe)
    dirs = _directions(rotation, R)
    at = G.probes()[probes]
    with torch.no_grad():
        o = (at * G.cell + G.lo).repeat_interleave(R, 0)
        d = dirs.repeat(len(probes), 1)
        t, obj, axis, side, leaving = geo.hit(o, d, 0.01, G.tmax)
        miss = torch.isinf(t)
        back = ~miss & (leaving != (obj == 0))  # boxes face outward, the room inward
        front = (~miss & ~back).nonzero()[:, 0]
        pos = o[front] + d[front] * t[front, None]
        on = torch.zeros((len(front), 3), dtype=torch.float64, device="cuda")
        on[torch.arange(len(front), device="cuda"), axis[front]] = side[front]
        on = torch.where((obj[front] == 0)[:, None], -on, on)
        nrm = _unit(torch.einsum("rij,ri->rj", geo.A[obj[front]], on))
        shadow = ~torch.isinf(geo.hit(pos, light.expand(len(pos), 3), 0.1, 1e4)[0])
        dist = torch.where(miss, -1.0, torch.where(back, 0.8 * t, t))
    df = d[front]
    refl = df - nrm * (2 * (nrm * df).sum(-1, keepdim=True))
    alb = albedo[geo.material[obj[front]]]
    zero, one = (torch.full((len(front), 1), x, dtype=torch.float64, device="cuda") for x in (0.0, 1.0))
    c = 0.04 * _lookup(G, pos, refl, -df, states, color, depth)
    c = c + _lookup(G, pos, nrm, -df, states, color, depth) * alb * 0.96
    c = c + torch.where(shadow[:, None], 0.0, _sun(nrm, _unit(-df), sun, light, alb, zero, one))
    rec = torch.where(miss[:, None], sky, torch.zeros((len(o), 3), dtype=torch.float64, device="cuda"))
    rec = rec.index_put((front,), c).reshape(len(probes), R, 3)
    dep = dist.reshape(len(probes), R).clamp(max=G.cell_len)
    dep = torch.where(dep < 0, G.cell_len, dep)
    dep = torch.stack([dep, dep * dep], -1)
    new = []
    for side_, tex, val, sharp in ((g.color_res, color, rec, 1.0), (g.depth_res, depth, dep, float(g.depth_sharpness))):
        n, ch = side_ - 2, val.shape[-1]
        w = (_texel_directions(side_) @ dirs.T).clamp(min=0)
        w = w if sharp == 1.0 else w ** sharp
        s = w.sum(-1)
        b = torch.einsum("tr,prc->ptc", w, val) / torch.where(s > 1e-3, s, 1.0)[:, None]
        x0, y0 = side_ * (at[:, 1] * G.res[0] + at[:, 0]), side_ * at[:, 2]
        k = torch.arange(n * n, device="cuda")
        X, Y = x0[:, None] + 1 + k % n, y0[:, None] + 1 + k // n
        b = torch.cat([b * (1 - hyst) + tex[Y, X][..., :ch] * hyst, tex[Y, X][..., ch:]], -1)
        tex = tex.index_put((Y, X), b)
        e = torch.arange(1, n + 1, device="cuda")
        lo_, hi_, m = torch.zeros_like(e), torch.full_like(e, side_ - 1), side_ - 1 - e
        bx = torch.cat([lo_, hi_, e, e, torch.tensor([0, 0, side_ - 1, side_ - 1], device="cuda")])
        by = torch.cat([e, e, lo_, hi_, torch.tensor([0, side_ - 1, 0, side_ - 1], device="cuda")])
        sx = torch.cat([lo_ + 1, hi_ - 1, m, m, torch.tensor([side_ - 2, side_ - 2, 1, 1], device="cuda")])
        sy = torch.cat([m, m, lo_ + 1, hi_ - 1, torch.tensor([side_ - 2, 1, side_ - 2, 1], device="cuda")])
        tex = tex.index_put((y0[:, None] + by, x0[:, None] + bx), tex[y0[:, None] + sy, x0[:, None] + sx])
        new.append(tex)
    return new


def _exact_gather(case, seed):
    rng = np.random.default_rng([int(seed), 17])
    g = _grid_desc(case, (np.zeros(3), np.array([10.0, 6.0, 10.0])))
    light = _light(rng)
    color, depth = (_f64(a) for a in _atlases(g, seed))
    states = torch.as_tensor(_states(g, seed).astype(np.int64), device="cuda")
    gb, origin = _gbuffer(case, seed)
    q = {k: v.double().reshape(-1, 4 if v.dim() == 3 else 1) for k, v in gb.items()}
    pos, depth_px = q["position_depth"][:, :3], q["position_depth"][:, 3:]
    nrm, metal = _unit(q["normal_metalness"][:, :3]), q["normal_metalness"][:, 3:]
    alb, rough = q["albedo_roughness"][:, :3], q["albedo_roughness"][:, 3:]
    view = _unit(_f64(origin) - pos)
    c = _sun(nrm, view, _f64(light.color[:3]), _f64(light.direction[:3]), alb, metal, rough) * q["direct_light"]
    if "reflection" in q:
        c = c + (0.004 * (1 - metal) + alb * metal) * q["reflection"][:, :3]
    c = c + _lookup(_Grid64(g), pos, nrm, view, states, color, depth) * alb * 0.996 * (1 - metal)
    c = torch.where(depth_px > 0, c + q["emissive"][:, :3], _f64(light.sky[:3]))
    return torch.cat([c, torch.ones_like(depth_px)], -1).reshape(case["height"], case["width"], 4)


def exact(case, seed):
    if case["op"] == "gather":
        return _exact_gather(case, seed)
    if case["op"] in ("batch", "load") or case["scene"] != "room":
        return None
    rng = np.random.default_rng([int(seed), 17])
    scene = _scene(case, rng)
    g = _grid_desc(case, scene.bounds)
    G = _Grid64(g)
    L = _light(rng)
    color, depth = (_f64(a) for a in _atlases(g, seed))
    P = g.probe_count()
    states = np.ones(P, np.int64)
    probes = torch.arange(P, device="cuda")
    transforms = scene.instances["transform"].copy()
    rotations = _rotations(seed, 1)
    hyst = float(np.float32(g.hysteresis))
    if case["op"] == "frame":  # the schedule's first visit; probe i is due when i % state == 0
        states = _states(g, seed).astype(np.int64)
        due = np.nonzero((states != 0) & (np.arange(P) % np.maximum(states, 1) == 0))[0]
        probes = torch.as_tensor(due[:case["cap"]] if case["cap"] else due, device="cuda")
    if case["op"] == "move":
        ids, motion = _motion(case, scene, rng)
        transforms[ids] = motion[0]
    if case["op"] == "learn":
        grad = rng.standard_normal(g.atlas_shape(abi.ATLAS_COLOR), np.float32)
        rotations = _rotations(seed, case["updates"])
    geo = _Room64(scene, transforms)
    states = torch.as_tensor(states, device="cuda")
    params = [_f64(scene.materials["base_color"]), _f64(L.color[:3]), _f64(L.sky[:3])]
    for p in params:
        p.requires_grad_(case["op"] == "learn")
    for r in rotations:
        # (updates of one context also refresh the probe states, none of which becomes or leaves 0)
        color, depth = _update64(G, geo, _f64(L.direction[:3]), params[0], params[2], params[1], r, probes, states,
                                 color, depth, hyst)
    if case["op"] != "learn":
        return [color, depth]
    grads = torch.autograd.grad((color[..., :3] * _f64(grad)[..., :3]).sum(), params)
    return [*grads, color.detach(), depth.detach()]
