"""Timed cases of the framework's public entry points, at the sizes its users run them.

Three families, as an editing program has them:
- edits: one brush stroke at a time (`MyGPUHashDAG.edit`), groups of strokes (`edit_batch`), a stretch
  of a session with its collection (`edit_batch` and `garbage_collect`);
- views: the primary-ray hit buffer of a frame (`trace`) and its shading (`resolve_lighting`);
- data: lookups in a slab hash table (`HashTable.find` / `read`) and building a scene.

Scenes are the procedural terrains of `svdag.workloads` (8 octaves, 4096 structures at depth 17, fewer
on smaller grids by their surface), the edits lie on the surface and their shapes and mix are those of
`c2_edits`, `c3_edits` and `c4_stream`.

A single edit is followed by the voxels of its region, as an editor reads them back, and an undo, so
that every pass starts from the same scene. Batches hold additions, removals and paints only: they
leave the same voxels however often they are applied. Item handles depend on the order in which
concurrent inserts land, so cases return voxels, hit records, colours and item words, never handles.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-svdag-editing_b200"))

import svdag  # noqa: E402
from svdag import workloads as wl  # noqa: E402

GIB = 1 << 30
TOOLS = {
    "sphere_add": svdag.TOOL_SPHERE_ADD, "sphere_remove": svdag.TOOL_SPHERE_REMOVE, "box_add": svdag.TOOL_BOX_ADD,
    "box_remove": svdag.TOOL_BOX_REMOVE, "sphere_paint": svdag.TOOL_SPHERE_PAINT, "copy": svdag.TOOL_COPY,
    "noise_paint": svdag.TOOL_BOX_PAINT_NOISE, "erode": svdag.TOOL_SPHERE_ERODE,
}


def listed():
    return [
        # the smallest stroke of an interactive brush (radius 9 voxels): latency and launches
        {"name": "edit_small", "kind": "edit", "levels": 13, "tool": "sphere_add", "radius": 9.0, "persistent": False},
        # an ordinary carve, odd radius
        {"name": "edit_carve", "kind": "edit", "levels": 14, "tool": "sphere_remove", "radius": 133.0, "persistent": False},
        # the at-scale carve of c2_edits (radius 2048 at depth 17), here a radius of 1024 at depth 15
        {"name": "edit_carve_large", "kind": "edit", "levels": 15, "tool": "sphere_remove", "radius": 1024.0, "persistent": False},
        # copy-paste of a region, the 512^3 box of c2_edits
        {"name": "edit_copy", "kind": "edit", "levels": 15, "tool": "copy", "radius": 256.0, "persistent": False},
        # material paint of a 1024^3 box from value noise, the largest edit of c2_edits
        {"name": "edit_noise_paint", "kind": "edit", "levels": 15, "tool": "noise_paint", "radius": 512.0, "persistent": False},
        # smoothing a surface with the erosion brush
        {"name": "edit_erode", "kind": "edit", "levels": 13, "tool": "erode", "radius": 40.0, "persistent": False},
        # many small strokes at once, scattered over the scene (several users, or a replay)
        {"name": "batch_small", "kind": "batch", "levels": 15, "count": 256, "rmin": 4.0, "rmax": 16.0, "collect": False},
        # a stretch of the served stream: uneven strokes, then the collection that follows them
        {"name": "session", "kind": "batch", "levels": 14, "count": 64, "rmin": 2.0, "rmax": 512.0, "collect": True},
        # the frame of a full-size view
        {"name": "trace_1080p", "kind": "trace", "levels": 15, "width": 1920, "height": 1080},
        # shading a frame: sun shadows and 4 ambient-occlusion rays a pixel
        {"name": "shade_720p", "kind": "shade", "levels": 14, "width": 1280, "height": 720, "ao": 4},
        # lookups in a table of 2^24 stored items at 16 items a bucket, half of them hits
        {"name": "table_find", "kind": "find", "keys": 1 << 24, "load": 16, "lanes": 1},
        # building a scene from nothing: every phase of construction, every item inserted
        {"name": "build_scene", "kind": "build", "levels": 13, "octaves": 8, "structures": 16},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["edit", "edit", "edit", "batch", "batch", "trace", "shade", "find", "build"])
    if kind == "edit":
        tool = rng.choice(sorted(TOOLS))
        hi = {"erode": 60.0, "copy": 256.0, "noise_paint": 400.0, "sphere_paint": 600.0}.get(tool, 1024.0)
        radius = float(round(log(2.0, hi), rng.choice([0, 0, 0, 2])))
        return {"kind": kind, "levels": rng.randint(12, 15), "tool": tool, "radius": radius, "persistent": rng.random() < 0.3}
    if kind == "batch":
        collect = rng.random() < 0.5
        return {"kind": kind, "levels": rng.randint(12, 15), "count": int(log(2, 64 if collect else 256)), "rmin": 2.0,
                "rmax": float(round(log(6.0, 256.0 if collect else 24.0))), "collect": collect}
    if kind == "trace":
        return {"kind": kind, "levels": rng.randint(10, 15), "width": int(log(33, 1920)), "height": int(log(17, 1080))}
    if kind == "shade":
        return {"kind": kind, "levels": rng.randint(10, 14), "width": int(log(33, 1280)), "height": int(log(17, 720)),
                "ao": rng.choice([0, 1, 2, 4])}
    if kind == "find":
        return {"kind": kind, "keys": int(log(1000, 1 << 24)), "load": rng.choice([8, 16, 32, 96]), "lanes": rng.choice([1, 1, 1, 4, 8])}
    return {"kind": kind, "levels": rng.randint(10, 13), "octaves": rng.randint(3, 8), "structures": rng.randint(0, 40)}


# ------------------------------------------------------------------ what a program has before the call

def _terrain(levels, seed):
    structures = 4096 >> (2 * max(0, wl.C2_LEVELS - levels))
    return dict(wl.C2_TERRAIN, seed=seed & 0x7FFFFFFF, num_structures=structures, structure_seed=(seed + 11) & 0x7FFFFFFF)


def _scene(levels, seed, pool, scratch, persistent=False):
    terrain = _terrain(levels, seed)
    dag = svdag.MyGPUHashDAG(levels, pool_bytes=pool, scratch_bytes=scratch, persistent=persistent)
    dag.build_terrain(**terrain)
    return dag, terrain


def _surface(rng, levels, terrain, margin, spread):
    g = 1 << levels
    margin = min(margin, g // 2 - 1)
    x, z = rng.randrange(margin, g - margin), rng.randrange(margin, g - margin)
    y = svdag.scene_height(levels, x, z, **terrain)
    return [float(x), float(y + rng.randint(-spread, spread)), float(z)]


def _region(center, reach, points, g):
    """Voxels of the box of half extent `reach` around `center`, `points` an axis."""
    offsets = np.round(np.linspace(-reach, reach, points)).astype(np.int64)
    axes = [np.clip(np.int64(c) + offsets, 0, g - 1) for c in center]
    grid = np.stack(np.meshgrid(*axes, indexing="ij"), axis=-1).reshape(-1, 3)
    return grid.astype(np.int32)


def _prepare_edit(case, seed):
    levels, radius, tool = case["levels"], case["radius"], case["tool"]
    g = 1 << levels
    dag, terrain = _scene(levels, seed, 8 * GIB, 3 * GIB, case["persistent"])
    rng = random.Random(seed)
    center = _surface(rng, levels, terrain, int(3 * radius) + 4, 32 if radius > 64 else 4)
    where = center
    if tool == "copy":
        where = [center[0] + float(rng.choice([-1, 1]) * int(1.5 * radius + 3)), center[1] + float(rng.randint(-2, 2)), center[2]]
    edit = wl.make_edit(TOOLS[tool], rng.randrange(16), center, radius, src=center, dst=where,
                        noise_seed={"erode": 13, "noise_paint": 17}.get(tool, 0), noise_cell_log2=4)
    xyz = torch.from_numpy(_region(where, radius + 2, min(48 if radius < 150 else 112, 2 * int(radius) + 5), g)).cuda()
    return {"kind": "edit", "dag": dag, "edit": edit, "xyz": xyz, "voxels": torch.empty(len(xyz), dtype=torch.int32, device="cuda")}


def _prepare_batch(case, seed):
    levels = case["levels"]
    g = 1 << levels
    dag, terrain = _scene(levels, seed, 10 * GIB, 3 * GIB, persistent=True)
    rng = random.Random(seed)
    edits, regions = [], []
    for _ in range(case["count"]):
        radius = float(int(math.exp(rng.uniform(math.log(case["rmin"]), math.log(case["rmax"])))))
        center = _surface(rng, levels, terrain, 1, 32 if radius > 64 else 4)
        sphere, u = rng.random() < 0.5, rng.random()
        if u < 0.4:
            tool = "sphere_add" if sphere else "box_add"
        elif u < 0.8:
            tool = "sphere_remove" if sphere else "box_remove"
        else:
            tool = "sphere_paint"
        edits.append(wl.make_edit(TOOLS[tool], rng.randrange(16), center, radius))
        regions.append(_region(center, radius + 2, 8 if case["rmax"] < 100 else 20, g))
    xyz = torch.from_numpy(np.concatenate(regions)).cuda()
    return {"kind": "batch", "dag": dag, "edits": edits, "collect": case["collect"], "xyz": xyz,
            "voxels": torch.empty(len(xyz), dtype=torch.int32, device="cuda")}


def _view(case, seed, levels):
    """A camera above the surface of the scene's middle, looking down across it (as the frames of the benchmark)."""
    g = float(1 << levels)
    a = random.Random(seed).uniform(0, 2 * math.pi)
    back = 0.065 * g
    return svdag.get_trace_params((0.5 * g - back * math.cos(a), 0.62 * g, 0.5 * g - back * math.sin(a)),
                                  (0.5 * g, 0.52 * g, 0.5 * g), case["width"], case["height"])


def _prepare_view(case, seed):
    levels = case["levels"]
    dag, _ = _scene(levels, seed, 6 * GIB, 2 * GIB)
    state = {"kind": case["kind"], "dag": dag, "params": _view(case, seed, levels),
             "tracer": svdag.DAGTracer(case["width"], case["height"])}
    if case["kind"] == "shade":
        state["tracer"].resolve_paths(state["params"], dag)
        state["shade"] = svdag.shade_params(levels, shadows=True, ao_samples=case["ao"], ao_ray_length=float(max(1 << (levels - 10), 8)))
    return state


def _node_keys(n, generator, first):
    """n distinct inner nodes: a child mask with 1..8 bits, then a child word a bit (28 bits); the
    first children are the numbers from `first` on, so no two nodes are equal."""
    order = torch.rand((n, 8), generator=generator, device="cuda").argsort(1)
    children = torch.randint(1, 9, (n,), generator=generator, device="cuda")
    mask = torch.zeros(n, dtype=torch.int64, device="cuda")
    for j in range(8):
        mask |= torch.where(children > j, torch.ones_like(mask) << order[:, j], torch.zeros_like(mask))
    words = torch.randint(0, 1 << 28, (n, 9), generator=generator, device="cuda", dtype=torch.int32)
    words[:, 0] = mask.to(torch.int32)
    words[:, 1] = first + torch.randperm(n, generator=generator, device="cuda").to(torch.int32)
    return words, 1 + children


def _packed(words, sizes):
    used = torch.arange(9, device="cuda")[None, :] < sizes[:, None]
    offsets = torch.cumsum(sizes, 0) - sizes
    return words[used].contiguous(), offsets.to(torch.int32)


def _lookup_keys(case, seed):
    """Stored keys, asked keys (half of them stored ones, in another order) and which are stored."""
    n = case["keys"]
    generator = torch.Generator(device="cuda").manual_seed(seed)
    stored, stored_sizes = _node_keys(n, generator, 0)
    fresh, fresh_sizes = _node_keys(n - n // 2, generator, n)
    known = torch.randperm(n, generator=generator, device="cuda")[: n // 2]
    mix = torch.randperm(n, generator=generator, device="cuda")
    asked = torch.cat([stored[known], fresh])[mix]
    sizes = torch.cat([stored_sizes[known], fresh_sizes])[mix]
    hit = mix < n // 2
    return stored, stored_sizes, asked, sizes, hit


def _prepare_find(case, seed):
    n = case["keys"]
    dag = svdag.MyGPUHashDAG(10, pool_bytes=6 * GIB, scratch_bytes=GIB)
    stored, stored_sizes, asked, sizes, _ = _lookup_keys(case, seed)
    per_size = torch.bincount(stored_sizes - 2, minlength=9)[:9].cpu().numpy()
    table = dag.create_table(svdag.KIND_NODE, np.maximum(1, per_size // case["load"] + 1))
    words, offsets = _packed(stored, stored_sizes)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    table.add(words, offsets, n, len(words), out)
    torch.cuda.synchronize()
    dag.sync()
    words, offsets = _packed(asked, sizes)
    return {"kind": "find", "dag": dag, "table": table, "words": words, "offsets": offsets, "count": n, "lanes": case["lanes"],
            "handles": out, "items": torch.empty((n, svdag.MAX_ITEM_WORDS), dtype=torch.int32, device="cuda")}


def _prepare_build(case, seed):
    levels = case["levels"]
    g = 1 << levels
    terrain = dict(_terrain(levels, seed), octaves=case["octaves"], num_structures=case["structures"])
    dag = svdag.MyGPUHashDAG(levels, pool_bytes=6 * GIB, scratch_bytes=3 * GIB)
    rng = np.random.default_rng(seed)
    columns = rng.integers(0, g, (16384, 2))
    heights = np.array([svdag.scene_height(levels, int(x), int(z), **terrain) for x, z in columns])
    y = np.clip(heights[:, None] + np.arange(-16, 16)[None, :], 0, g - 1)
    xyz = np.stack([np.repeat(columns[:, 0], 32), y.reshape(-1), np.repeat(columns[:, 1], 32)], axis=1).astype(np.int32)
    xyz = torch.from_numpy(xyz).cuda()
    return {"kind": "build", "dag": dag, "terrain": terrain, "xyz": xyz,
            "voxels": torch.empty(len(xyz), dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "edit":
        return _prepare_edit(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind in ("trace", "shade"):
        return _prepare_view(case, seed)
    if kind == "find":
        return _prepare_find(case, seed)
    return _prepare_build(case, seed)


# ------------------------------------------------------------------ one pass

def run(state):
    kind, dag = state["kind"], state["dag"]
    if kind == "edit":
        dag.edit(state["edit"])
        dag.sample_voxels(state["xyz"], len(state["xyz"]), state["voxels"])
        dag.undo()
        return state["voxels"]
    if kind == "batch":
        dag.edit_batch(state["edits"])
        if state["collect"]:
            dag.garbage_collect(keep_history=True)
        dag.sample_voxels(state["xyz"], len(state["xyz"]), state["voxels"])
        return state["voxels"]
    if kind == "trace":
        state["tracer"].resolve_paths(state["params"], dag)
        return state["tracer"].hits
    if kind == "shade":
        return state["tracer"].resolve_lighting(state["params"], dag, state["shade"]), state["tracer"].hits
    if kind == "find":
        table, n = state["table"], state["count"]
        table.find(state["words"], state["offsets"], n, len(state["words"]), state["handles"], lanes=state["lanes"])
        table.read(state["handles"], n, state["items"])
        return state["items"]
    dag.build_terrain(**state["terrain"])
    dag.sample_voxels(state["xyz"], len(state["xyz"]), state["voxels"])
    return state["voxels"]


def exact(case, seed):
    """Lookups: the words of each stored key, zeros for the others. Voxels, hit records and colours of
    a procedural scene are whole numbers and bytes that plain array code would take minutes for."""
    if case["kind"] != "find":
        return None
    _, _, asked, sizes, hit = _lookup_keys(case, seed)
    used = torch.arange(9, device="cuda")[None, :] < sizes[:, None]
    items = torch.zeros((case["keys"], svdag.MAX_ITEM_WORDS), dtype=torch.int32, device="cuda")
    items[:, :9] = torch.where(used & hit[:, None], asked, torch.zeros_like(asked))
    return items


# ------------------------------------------------------------------ the work of one pass

def _edit_leaves(tool, radius):
    """4^3 leaves that an edit of this shape on a half-filled region has to rewrite."""
    r = radius / 4.0
    if tool in ("copy", "noise_paint"):
        return max(1.0, 4.0 * r ** 3)
    if tool == "erode":
        return max(1.0, 2.0 / 3.0 * math.pi * r ** 3)
    if tool == "sphere_paint":
        return max(1.0, 2.0 * math.pi * r * r * 1.5)
    if tool.startswith("box"):
        return max(1.0, 24.0 * r * r)
    return max(1.0, 4.0 * math.pi * r * r * 1.5)


def work(case):
    """Bytes of one pass: per rewritten leaf its old and its new item (40 bytes each), a third more for
    the nodes above, and the path to the root; hit records and one descent a ray; keys, headers and items."""
    kind = case["kind"]
    if kind == "edit":
        return {"bytes": 80.0 * (_edit_leaves(case["tool"], case["radius"]) * 4 / 3 + case["levels"]), "flops": 0.0}
    if kind == "batch":
        lo, hi, n = case["rmin"], max(case["rmax"], case["rmin"] + 1), 64
        radii = [lo * (hi / lo) ** ((i + 0.5) / n) for i in range(n)]
        leaves = sum(_edit_leaves("sphere_add", r) for r in radii) / n
        out = case["count"] * 80.0 * (leaves * 4 / 3 + case["levels"])
        if case["collect"]:  # every reachable item is read once
            out += 40.0 * 6.0 * 4 ** (case["levels"] - 4)
        return {"bytes": out, "flops": 0.0}
    if kind == "trace":
        return {"bytes": case["width"] * case["height"] * (68.0 + 8.0 * case["levels"]), "flops": 0.0}
    if kind == "shade":
        rays = 1 + case["ao"]
        return {"bytes": case["width"] * case["height"] * (68.0 + 4.0 + 4.0 + 8.0 * case["levels"] * rays), "flops": 0.0}
    if kind == "find":  # 5.5 words a key on average
        return {"bytes": case["keys"] * (2 * 22.0 + 4 + 32 + 11.0 + 4 + 4 + 40.0 + 11.0), "flops": 0.0}
    return {"bytes": 40.0 * 6.0 * 4 ** (case["levels"] - 4), "flops": 0.0}
