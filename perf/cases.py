"""The workloads whose speed is tracked: what a host of this library has it do, through the
package's public classes (Scene, Renderer, Batch, LightBvh), from the smallest calls to the largest.

  frame        one rendered frame of a flushed scene: an editor's preview, an interactive view, a
               final still; with entities, without light-tree NEE, with the voxel id target
  adjoint      one backward call: the gradients of a frame with respect to albedo and power
  light_bvh    one light-tree build from brick light records on the device
  edit         a player's edit: changed bricks uploaded again, then the flush that applies them
  stream       a moving view: some bricks leave the world, others come, then the flush
  batch        many viewports of many scenes in one call, every light tree rebuilt

Worlds are this package's seeded generators (caelix_b200.workloads): "cube", the plain trace scene's
noise world (30 % of a cubic grid occupied, half of the voxels solid, 1 % of the bricks emissive),
and "terrain", the large trace scene's (a flat grid 47.7 % occupied, a quarter of the voxels solid,
5 % of the bricks emissive). Block-ID values unless a case says packed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "caelix-renderer_b200"))
import caelix_b200  # noqa: E402
from caelix_b200 import workloads  # noqa: E402


def listed():
    return [
        # An editor's preview of a small model: the smallest frame, launches and latency.
        _frame("frame_preview", bricks=150, width=160, height=90, bounces=2),
        # The plain trace scene's frame (16^3-brick grid, 512 x 512, 1 sample, 4 bounces).
        _frame("frame_plain", bricks=1229, width=512, height=512, bounces=4),
        # A small still of good quality: several samples of few pixels, ragged sides.
        _frame("frame_samples", bricks=5003, width=333, height=251, spp=8, bounces=3),
        # A full-HD frame of a large world (4 samples, 6 bounces): the largest frame.
        _frame("frame_hd", world="terrain", bricks=300_000, width=1920, height=1080, spp=4, bounces=6),
        # Moving objects in view: the plain frame with 16 entities of 2 x 2 x 2 bricks, lit.
        _frame("frame_entities", bricks=1229, width=512, height=512, bounces=4, entities=16),
        # The differentiation workload: the solid-brick world, 256 x 256, 8 samples, 3 bounces.
        {"name": "adjoint", "kind": "adjoint", "records": 4096, "width": 256, "height": 256, "spp": 8, "bounces": 3},
        # The plain light-tree build (one group) and a large world's (render groups, frames).
        {"name": "light_bvh_small", "kind": "light_bvh", "records": 4096, "grouped": False},
        {"name": "light_bvh_large", "kind": "light_bvh", "records": 2_000_003, "grouped": True},
        # An edit of 1 % of a large world's bricks.
        {"name": "edit", "kind": "edit", "world": "terrain", "bricks": 300_000, "share": 0.01, "packed": False},
        # A moving view over a packed-encoding world: 1 % of the bricks leave, as many come.
        {"name": "stream", "kind": "stream", "world": "terrain", "bricks": 100_000, "share": 0.01, "packed": True},
        # Many scenes at once (2 samples, 4 bounces, brick counts log-uniform as in the batched benchmark).
        {"name": "batch", "kind": "batch", "scenes": 12, "min_bricks": 1000, "max_bricks": 50_000, "side": 512,
         "spp": 2, "bounces": 4},
    ]


def _frame(name, world="cube", bricks=0, width=0, height=0, spp=1, bounces=4, entities=0, nee=True, voxel_id=False):
    return {"name": name, "kind": "frame", "world": world, "bricks": bricks, "width": width, "height": height,
            "spp": spp, "bounces": bounces, "entities": entities, "nee": nee, "voxel_id": voxel_id}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 5 + ["adjoint", "light_bvh", "edit", "stream", "batch"])
    if kind == "frame":
        bricks = _log(rng, 100, 250_000)
        c = _frame("", world="terrain" if bricks > 50_000 or rng.random() < 0.3 else "cube", bricks=bricks,
                   width=_log(rng, 80, 1920), height=_log(rng, 60, 1080), spp=rng.choice([1, 1, 2, 3, 4, 8]),
                   bounces=rng.randint(1, 6), entities=rng.choice([0, 0, 0, rng.randint(1, 24)]),
                   nee=rng.random() < 0.9, voxel_id=rng.random() < 0.2)
        c["spp"] = max(1, min(c["spp"], 4 * 1920 * 1080 // (c["width"] * c["height"])))
        del c["name"]
        return c
    if kind == "adjoint":
        return {"kind": kind, "records": _log(rng, 256, 4096), "width": rng.randint(48, 256),
                "height": rng.randint(48, 256), "spp": rng.choice([1, 2, 4, 8]), "bounces": rng.randint(1, 3)}
    if kind == "light_bvh":
        n = _log(rng, 200, 2_000_000)
        return {"kind": kind, "records": n, "grouped": n > 20_000 or rng.random() < 0.5}
    if kind == "edit":
        return {"kind": kind, "world": rng.choice(["cube", "terrain"]), "bricks": _log(rng, 2000, 250_000),
                "share": round(rng.uniform(0.002, 0.01), 4), "packed": rng.random() < 0.4}
    if kind == "stream":
        return {"kind": kind, "world": rng.choice(["cube", "terrain"]), "bricks": _log(rng, 2000, 90_000),
                "share": round(rng.uniform(0.002, 0.01), 4), "packed": rng.random() < 0.5}
    return {"kind": kind, "scenes": rng.randint(2, 10), "min_bricks": 1000, "max_bricks": _log(rng, 4000, 50_000),
            "side": rng.choice([200, 256, 384, 500]), "spp": rng.choice([1, 2]), "bounces": rng.randint(2, 4)}


# ---- inputs ----

_device = None


def _dev():
    global _device
    if _device is None:
        _device = caelix_b200.Device(torch.cuda.current_device())
    return _device


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _world(kind, bricks, seed, aspect=1.0):
    """A generated world with a camera that has most of it in view."""
    if kind == "cube":
        side = max(2, math.ceil((bricks / 0.30) ** (1 / 3)))
        grid, fill, lit, scale = (side, side, side), 0.5, 0.01, 0.25
    else:
        side = max(2, math.ceil((bricks / 0.477 / 16) ** (1 / 3)))
        grid, fill, lit, scale = (4 * side, 4 * side, side), 0.25, 0.05, 1.0 / 16
    size = np.array(grid, np.float64) * 8
    at, to = ((-0.25, 1.2, -0.35), (0.5, 0.35, 0.5)) if kind == "cube" else ((-0.05, 1.1, -0.3), (0.45, 0.3, 0.45))
    camera = workloads.look_at(size * np.array(at), size * np.array(to), aspect=aspect)
    return workloads.noise_world_large(grid_bricks=grid, occupied_bricks=bricks, voxel_fill=fill,
                                       emissive_bricks=max(1, round(lit * bricks)), seed=seed, brick_scale=scale,
                                       voxel_scale=0.25 if kind == "cube" else 0.125, camera=camera)


def _small(seed):
    """A seed the generators take."""
    return 2 + seed % 399_989


def _painted(kind, bricks, seed):
    """A world whose shape follows from its size, so that its tables have one shape, and whose
    materials and brick powers follow from the seed."""
    vs = _world(kind, bricks, 2 + bricks)
    rng = np.random.default_rng(seed)
    paint = torch.from_numpy(rng.integers(0, 64, (vs.brick_count, 1))).cuda().int()
    v = torch.from_numpy(vs.voxels.astype(np.int32)).cuda()
    v = torch.where(v == 0, v, 0x8000 | 1 + ((v & 0x7F) - 1 + paint) % 64)
    power = np.where(vs.power > 0, rng.lognormal(0.0, 1.0, vs.brick_count), 0.0).astype(np.float32)
    return vs.like(voxels=v.cpu().numpy().astype(np.uint16), power=power)


def _packed(vs):
    """The world in the packed encoding: opaque colours, one voxel in 64 translucent, the emissive
    bricks' voxels of an emissive code (brick power 1)."""
    v = torch.from_numpy(vs.voxels.astype(np.int32)).cuda()
    material = v & 0x7F
    colour = 0x8000 | ((material * 0x1235) & 0x7FFF)
    brick = torch.arange(v.shape[0], device="cuda")[:, None] * 512 + torch.arange(512, device="cuda")[None]
    colour = torch.where(((brick * 40503) >> 4) % 64 == 0, 1 + material, colour)
    lamp = 0x4000 | ((material * 0x5A5) & 0xFFF | 0x111) << 2 | 3  # every colour bright enough to be a light
    on = torch.from_numpy(vs.power > 0).cuda()[:, None]
    out = torch.where(v == 0, torch.zeros_like(v), torch.where(on, lamp, colour))
    return vs.like(voxels=out.cpu().numpy().astype(np.uint16), power=np.ones(vs.brick_count, np.float32), albedo=None,
                   encoding=workloads.ENCODING_PACKED, min_emission=20.0)


def _torch_rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


class _Memory:
    """`count` elements at a device address, for torch.as_tensor; keeps the owner of the memory alive."""

    def __init__(self, owner, address, count, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (count,), "typestr": kind, "version": 3}


class _Views:
    """Tensors over the device arrays of a library object, made once for each array."""

    def __init__(self, owner):
        self.owner, self.known = owner, {}

    def __call__(self, address, count, kind="<i4"):
        key = (address, count, kind)
        t = self.known.get(key)
        if t is None:
            t = self.known[key] = (torch.as_tensor(_Memory(self.owner, address, count, kind), device="cuda") if count
                                   else torch.zeros(0, device="cuda"))
        return t


def _tree(view, header, nodes, leaves, node_count, leaf_count):
    """A light tree's header, 4-wide nodes and leaves: their floats and their words."""
    out = {"header": view(header, 12, "<f4"), "header_words": view(header + 48, 3)}
    f, w = view(nodes, node_count * 56, "<f4"), view(nodes, node_count * 56)
    if node_count:
        out["nodes"], out["node_words"] = f.view(-1, 56)[:, :48], w.view(-1, 56)[:, 48:54]
    if leaf_count:
        out["leaves"] = view(leaves, leaf_count * 16, "<f4").view(-1, 16)[:, :12]
        words = view(leaves, leaf_count * 16).view(-1, 16)
        out["leaf_owner"], out["leaf_parent"] = words[:, 12:14], words[:, 15]
    return out


def _tables(view, scene):
    """A flushed scene's tables, light records and light tree."""
    v = scene.view()
    m = v.light_count
    out = {"records": view(v.records, 274 * v.brick_count), "keys": view(v.keys, 3 * v.brick_count),
           "hash_slots": view(v.hash_slots, 4 * v.hash_slot_count),
           "bitmap": view(v.bitmap, (v.grid[0] * v.grid[1] * v.grid[2] + 31) // 32),
           "heap": view(v.heap, v.heap_words), "group_rows": view(v.group_rows, 8 * v.group_count)}
    if m:
        out["light_faces"] = view(v.light_headers, 12 * m, "<f4").view(-1, 12)[:, :6]
        out["light_words"] = view(v.light_headers, 12 * m).view(-1, 12)[:, 6:]
        out["light_brick"] = view(v.light_brick, m)
        out |= _tree(view, v.tree_header, v.tree_nodes, v.tree_leaves, m, m)
    return out


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _add_entities(scene, vs, count, seed):
    """Entities of 2 x 2 x 2 bricks at random places and rotations, half of their bricks emitting."""
    rng = np.random.default_rng(seed)
    size = np.array(vs.grid, np.float64) * 8
    for i in range(count):
        ent = workloads.noise_world(grid_bricks=(2, 2, 2), brick_occupancy=1.0, emissive_fraction=0.0, seed=seed + 100 + i)
        q = rng.normal(size=4)
        e = scene.add_entity(tuple(size * rng.uniform(0.06, 0.9, 3)), tuple(q / np.linalg.norm(q)))
        scene.upload_bricks(ent.keys, ent.voxels, entity=e)
        power = np.where(rng.random(ent.brick_count) < 0.5, rng.lognormal(0.0, 1.0, ent.brick_count), 0.0)
        scene.set_brick_power(ent.keys, power.astype(np.float32), entity=e)
        scene.set_entity_motion(e, i % 2)
    scene.flush(_stream())


def _prepare_frame(case, seed):
    w, h = case["width"], case["height"]
    vs = _world(case["world"], case["bricks"], _small(seed), aspect=w / h)
    scene = caelix_b200.Scene.from_voxel_scene(_dev(), vs)
    if case["entities"]:
        _add_entities(scene, vs, case["entities"], _small(seed))
    renderer = caelix_b200.Renderer(_dev(), scene)
    if not case["nee"]:
        renderer.set_light_nee(False)
    return {"run": _run_frame, "case": case, "renderer": renderer, "camera": caelix_b200.camera_struct(vs.camera),
            "radiance": torch.zeros(h, w, 3, device="cuda"), "seed": 1 + seed % 1000,
            "voxel_id": torch.zeros(h, w, 2, dtype=torch.int32, device="cuda") if case["voxel_id"] else None}


def _run_frame(s):
    c = s["case"]
    s["renderer"].render(s["radiance"], c["width"], c["height"], s["camera"], bounces=c["bounces"], seed=s["seed"],
                         spp=c["spp"], stream=_stream(), voxel_id=s["voxel_id"])
    return {"radiance": s["radiance"], "voxel_id": s["voxel_id"]}


def _prepare_adjoint(case, seed):
    vs = workloads.solid_brick_scene(n=case["records"], seed=_small(seed))
    vs.camera["aspect"] = np.float32(case["width"] / case["height"])
    scene = caelix_b200.Scene.from_voxel_scene(_dev(), vs)
    shape = (case["height"], case["width"], 3)
    return {"run": _run_adjoint, "case": case, "renderer": caelix_b200.Renderer(_dev(), scene),
            "camera": caelix_b200.camera_struct(vs.camera), "seed": 1 + seed % 1000,
            "d_radiance": torch.randn(shape, device="cuda", generator=_torch_rng(seed)),
            "image": torch.zeros(shape, device="cuda"), "d_albedo": torch.zeros(65536, 3, device="cuda"),
            "d_power": torch.zeros(case["records"], device="cuda")}  # a repeated record is one brick


def _run_adjoint(s):
    c = s["case"]
    s["renderer"].backward(s["d_radiance"], c["width"], c["height"], s["camera"], s["d_albedo"], s["d_power"],
                           bounces=c["bounces"], seed=s["seed"], spp=c["spp"], image=s["image"], stream=_stream())
    return {"image": s["image"], "d_albedo": s["d_albedo"], "d_power": s["d_power"]}


def _light_records(case, seed):
    """Brick light records [n, 12] (int32 words), their groups and the group frames: brick
    coordinates uniform in the grid, power log-normal(0, 1) split evenly over the six faces."""
    n, g = case["records"], _torch_rng(seed)
    shift, edge = (4, 1024) if case["grouped"] else (0, 32)
    at = torch.randint(0, edge, (n, 3), device="cuda", generator=g)
    power = torch.exp(torch.randn(n, device="cuda", generator=g))
    local = at & 15 if case["grouped"] else at
    lo = local * 8
    rec = torch.zeros(n, 12, dtype=torch.int32, device="cuda")
    rec[:, :6] = (power / 6.0)[:, None].expand(n, 6).contiguous().view(torch.int32)
    rec[:, 6] = (lo[:, 0] | lo[:, 1] << 10 | lo[:, 2] << 20).to(torch.int32)
    rec[:, 7] = (lo[:, 0] + 8 | lo[:, 1] + 8 << 10 | lo[:, 2] + 8 << 20).to(torch.int32)
    rec[:, 8] = (local[:, 0] | local[:, 1] << 4 | local[:, 2] << 8).to(torch.int32)
    if not case["grouped"]:
        return rec, None, None, at * 8
    groups = edge >> shift
    cell = at >> shift
    group = (cell[:, 0] + groups * (cell[:, 1] + groups * cell[:, 2])).to(torch.int32)
    index = torch.arange(groups ** 3, device="cuda")
    frames = torch.zeros(groups ** 3, 15, device="cuda")
    for k in range(3):
        frames[:, k] = ((index // groups ** k) % groups * (8 << shift)).float()
        frames[:, 3 + 4 * k] = 1.0
    return rec, group, frames, at * 8


def _prepare_light_bvh(case, seed):
    rec, group, frames, _ = _light_records(case, seed)
    bvh = caelix_b200.LightBvh(_dev(), case["records"])
    view, v = _Views(bvh), bvh.view()
    view(v.nodes, case["records"] * 56).zero_()  # a build writes as many rows as the tree has nodes
    return {"run": _run_light_bvh, "case": case, "bvh": bvh, "records": rec, "group": group, "frames": frames, "view": view}


def _run_light_bvh(s):
    n, frames = s["case"]["records"], s["frames"]
    s["bvh"].build(s["records"], n, record_group=s["group"], group_frames=frames,
                   group_count=None if frames is None else len(frames), stream=_stream())
    v = s["bvh"].view()
    return _tree(s["view"], v.header, v.nodes, v.leaves, n, n)


def _prepare_edit(case, seed):
    vs = _painted(case["world"], case["bricks"], seed)
    rng = np.random.default_rng(case["bricks"])
    if case["packed"]:
        vs = _packed(vs)
    scene = caelix_b200.Scene.from_voxel_scene(_dev(), vs)
    at = np.sort(rng.choice(vs.brick_count, max(1, round(case["share"] * vs.brick_count)), replace=False))
    # Dug: a twentieth of the voxels of the edited bricks removed, then put back.
    before = np.ascontiguousarray(vs.voxels[at])
    after = np.where(rng.random(before.shape) < 0.05, np.uint16(0), before)
    v = scene.view()
    view = _Views(scene)
    view(v.tree_nodes, 56 * v.light_count).zero_()  # a build writes as many rows as the tree has nodes
    return {"run": _run_edit, "scene": scene, "keys": np.ascontiguousarray(vs.keys[at]), "voxels": [after, before],
            "turn": 0, "view": view}


def _run_edit(s):
    s["scene"].upload_bricks(s["keys"], s["voxels"][s["turn"]])
    s["scene"].flush(_stream())
    s["turn"] ^= 1
    return _tables(s["view"], s["scene"])


def _prepare_stream(case, seed):
    vs = _painted(case["world"], case["bricks"], seed)
    if case["packed"]:
        vs = _packed(vs)
    # Two sets of bricks at opposite sides of the first axis: one is in the world at a time.
    k = max(1, round(case["share"] * vs.brick_count))
    order = np.argsort(vs.keys[:, 0], kind="stable")
    sets = [np.sort(order[:k]), np.sort(order[-k:])]
    stay = np.ones(vs.brick_count, bool)
    stay[sets[1]] = False
    scene = caelix_b200.Scene.for_voxel_scene(_dev(), vs)
    scene.upload_bricks(vs.keys[stay], vs.voxels[stay])
    scene.set_brick_power(vs.keys, vs.power)
    scene.flush(_stream())
    v = scene.view()
    view = _Views(scene)
    view(v.tree_nodes, 56 * v.light_count).zero_()  # a build writes as many rows as the tree has nodes
    return {"run": _run_stream, "scene": scene, "keys": [np.ascontiguousarray(vs.keys[i]) for i in sets],
            "voxels": [np.ascontiguousarray(vs.voxels[i]) for i in sets],
            "power": [np.ascontiguousarray(vs.power[i]) for i in sets], "turn": 0, "view": view}


def _run_stream(s):
    scene, turn = s["scene"], s["turn"]
    scene.remove_bricks(s["keys"][turn])
    scene.upload_bricks(s["keys"][turn ^ 1], s["voxels"][turn ^ 1])
    scene.set_brick_power(s["keys"][turn ^ 1], s["power"][turn ^ 1])
    scene.flush(_stream())
    s["turn"] ^= 1
    return _tables(s["view"], scene)


def _batch_bricks(case):
    """The scenes' brick counts: even steps of the logarithm."""
    n = case["scenes"]
    lo, hi = math.log(case["min_bricks"]), math.log(case["max_bricks"])
    return [round(math.exp(lo + (hi - lo) * (i + 0.5) / n)) for i in range(n)]


def _prepare_batch(case, seed):
    views, images, side = [], [], case["side"]
    for i, bricks in enumerate(_batch_bricks(case)):
        vs = _world("cube", bricks, _small(97 * seed + i))
        renderer = caelix_b200.Renderer(_dev(), caelix_b200.Scene.from_voxel_scene(_dev(), vs))
        at = side if i % 2 else side // 2  # viewports of two sizes
        images.append(torch.zeros(at, at, 3, device="cuda"))
        views.append((renderer, images[-1], at, at, vs.camera, case["bounces"], 1 + i, case["spp"]))
    return {"run": _run_batch, "batch": caelix_b200.Batch(_dev(), views, rebuild_light_trees=True), "images": images}


def _run_batch(s):
    s["batch"].run(_stream())
    return s["images"]


# ---- what a pass cannot do without ----

_RECORD = 1096  # a brick record
_BRICK = 1024   # a brick's voxel values


def work(case):
    """Inputs read once, outputs written once; operations of the parts every pass has (a camera ray's
    set-up and its walk through one grid cell, the union of two summaries, a voxel's finalize)."""
    kind = case["kind"]
    if kind == "frame" or kind == "adjoint":
        rays = case["width"] * case["height"] * case["spp"]
        bricks = case["bricks"] if kind == "frame" else case["records"]
        out = 12 * case["width"] * case["height"]
        # The bricks in view: at most one per camera ray.
        return {"bytes": _RECORD * min(bricks, rays) + out * (1 if kind == "frame" else 2), "flops": 100 * rays}
    if kind == "light_bvh":
        n = case["records"]
        return {"bytes": n * (48 + 64 + 224 / 2), "flops": 100 * n}
    if kind == "edit":
        k = max(1, round(case["share"] * case["bricks"]))
        lights = (0.01 if case["world"] == "cube" else 0.05) * case["bricks"]
        # The edited bricks come in, their records and their neighbours' go out, the light tree is built.
        return {"bytes": k * (2 * _BRICK + _RECORD) + lights * (48 + 64 + 224 / 2), "flops": 512 * 10 * k + 100 * lights}
    if kind == "stream":
        n = case["bricks"]
        return {"bytes": n * (_BRICK + _RECORD), "flops": 512 * 10 * n}
    total = {"bytes": 0, "flops": 0}
    for i, bricks in enumerate(_batch_bricks(case)):
        side = case["side"] if i % 2 else case["side"] // 2
        rays = side * side * case["spp"]
        total["bytes"] += _RECORD * min(bricks, rays) + 12 * side * side
        total["flops"] += 100 * rays
    return total


def exact(case, seed):
    """The light tree's leaves and root in 64 bits. A path-traced image has no such value here (every
    decision of a path follows from its 32-bit arithmetic), a flush's tables are whole numbers."""
    if case["kind"] != "light_bvh":
        return None
    rec, _, _, lo = _light_records(case, seed)
    face = rec[:, :6].contiguous().view(torch.float32).double()
    lo = lo.double()
    box = torch.cat([lo, lo + 8.0], 1)
    header = torch.cat([face.sum(0), box[:, :3].amin(0), box[:, 3:].amax(0)])
    return {"header": header, "header_words": None, "nodes": None, "node_words": None,
            "leaves": torch.cat([face, box], 1), "leaf_owner": None, "leaf_parent": None}
