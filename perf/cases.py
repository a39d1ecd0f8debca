"""The work this library is used for, as cases that can be timed.

Every case is one call pattern of a program that keeps a hash DAG on the GPU:
frames of an interactive viewer, many views at once, single edits as a user
draws them, batches of edits, coloured edits with undo, garbage collection,
loading a scene and a served stream of edits and renders.  The scenes are the
seeded scenes of the library's own benchmark and tests (2^10 to 2^15 voxels
an edge, solid or, with colours, surface shell); what varies with the seed is
what a user's input varies: camera poses, tools, radii, places and request
traces.

A case that edits starts every pass from the loaded scene's root (or undoes
its edits at the end of the pass), so that each pass applies the same edits
to the same scene: a first pass adds nodes, later ones mostly find them.  The
garbage collection case drops what it added, so each of its passes adds.

Outputs are what the calls return or write: paths, shadow masks, colours,
edit counters, the root and every bucket's size (both of which follow from
the contents and order of all nodes ever added).
"""
import ctypes as C
import math

import numpy as np
import torch

import hashdag_gb300 as hd
from hashdag_gb300 import _capi, workloads

LIGHT = (0.3, 1.0, 0.2)
BIAS = 1.0

# BasicDAG words of the scenes, once per process: the scene file a program
# loads, in host memory.
_words = {}
# Scenes that are only read (frames, views): one resident copy per process,
# as a viewer keeps it.
_scenes = {}


def _scene_words(depth, shell):
    key = (depth, shell)
    if key not in _words:
        d = hd.HashDAG(depth)
        d.generate_scene(workloads.SEED_SCENE, shell=shell)
        _words[key] = d.export_basic_dag()
        d.free()
    return _words[key]


def _load(depth, colors=False):
    """A context of its own with the scene loaded."""
    d = hd.HashDAG(depth)
    d.load_from_DAG(_scene_words(depth, colors))
    if colors:
        d.colors_from_scene(workloads.SEED_COLORS)
    return d


def _shared(depth, colors=False):
    key = (depth, colors)
    if key not in _scenes:
        _scenes[key] = _load(depth, colors)
    return _scenes[key]


class _DeviceWords:
    """The context's bucket sizes in place, as an array torch can view."""

    def __init__(self, dag):
        self.dag = dag  # keeps the memory alive
        _, _, sizes = dag.device_table()
        n = C.c_uint64()
        dag._check(_capi.lib().hd_table_sizes(dag.handle, C.byref(n), None, None))
        self.__cuda_array_interface__ = {"shape": (n.value,), "typestr": "<i4", "data": (sizes, False), "version": 2}


def _bucket_sizes(dag):
    return torch.as_tensor(_DeviceWords(dag), device="cuda")


def _counters(stats):
    """What an edit call reports about its result (the words its probes
    scanned and its times say how it was done)."""
    return np.array([[s.num_voxels, s.num_nodes, s.find_or_add_calls, s.nodes_added] for s in stats], np.int64)


def listed():
    return [
        # The smallest frame: the preview of a small scene at the library's
        # own smoke-test size; launches and host time count.
        {"name": "frame_small", "kind": "frame", "depth": 10, "width": 320, "height": 180},
        # An interactive viewer's frame of the benchmark scene: primary and
        # shadow rays of one camera, one call each.
        {"name": "frame_1080p", "kind": "frame", "depth": 15, "width": 1920, "height": 1080},
        # The benchmark's step: primary and shadow rays of 16 poses of a
        # camera path, outputs left on the device.
        {"name": "views_16x1080p", "kind": "views", "depth": 15, "width": 1920, "height": 1080, "views": 16},
        # The same call end to end, results in pinned host memory.
        {"name": "views_host_8x1080p", "kind": "views_host", "depth": 15, "width": 1920, "height": 1080, "views": 8},
        # A coloured frame in a window of no round size, read back to the host.
        {"name": "colour_frame_ragged", "kind": "colour_frame", "depth": 13, "width": 1277, "height": 717},
        # 16 brush strokes of a user, one call each (sphere carves of radius
        # 16 to 48, the small scene of the tests).
        {"name": "edits_single_small", "kind": "edits_single", "depth": 10, "edits": 16, "r0": 16.0, "r1": 48.0},
        # Mixed single edits of the full radius range on the benchmark scene.
        {"name": "edits_single_large", "kind": "edits_single", "depth": 15, "edits": 8, "r0": 4.0, "r1": 512.0},
        # A batch of many small edits.
        {"name": "edit_batch_small", "kind": "edit_batch", "depth": 12, "edits": 64, "r0": 4.0, "r1": 48.0},
        # The benchmark's batch (a quarter of it): radius 4 to 512.
        {"name": "edit_batch_large", "kind": "edit_batch", "depth": 15, "edits": 64, "r0": 4.0, "r1": 512.0},
        # Every tool on a coloured scene, each edit undone at the end, the
        # colours of picked voxels read back before that.
        {"name": "coloured_tools", "kind": "coloured", "depth": 13, "edits": 12, "r0": 8.0, "r1": 64.0},
        # Edits, undone, then the garbage collection that drops them.
        {"name": "edit_undo_gc", "kind": "gc", "depth": 14, "edits": 16, "r0": 4.0, "r1": 256.0},
        # A served trace: edits in batches while renders are in flight.
        {"name": "serve", "kind": "serve", "depth": 13, "requests": 40, "r0": 4.0, "r1": 128.0},
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["frame", "views", "views_host", "colour_frame", "edits_single", "edit_batch", "coloured", "gc",
                       "serve"])
    c = {"kind": kind, "depth": rng.randint(10, 15)}
    if kind in ("frame", "colour_frame", "views", "views_host"):
        if kind == "colour_frame":
            c["depth"] = rng.randint(10, 13)
        c["width"] = int(_log(rng, 161, 2560))
        c["height"] = max(1, int(c["width"] * rng.uniform(0.4, 0.8)))
        if kind in ("views", "views_host"):
            pixels = 16 * 1920 * 1080 if kind == "views" else 8 * 1920 * 1080
            c["views"] = rng.randint(1, min(24, max(1, pixels // (c["width"] * c["height"]))))
        return c
    if kind == "coloured":
        c["depth"] = rng.randint(10, 13)
        c["edits"] = rng.randint(1, 12)
        c["r0"], c["r1"] = 6.0, round(_log(rng, 12, min(64.0, 2.0 ** c["depth"] / 32)), 2)
        return c
    if kind == "serve":
        c["depth"] = rng.randint(10, 13)
        c["requests"] = rng.randint(4, 40)
    else:
        if kind == "gc":
            c["depth"] = rng.randint(10, 14)
        c["edits"] = int(_log(rng, 1, {"edits_single": 9, "edit_batch": 65, "gc": 17}[kind]))
    c["r0"], c["r1"] = 4.0, round(_log(rng, 16, {"gc": 256.0, "serve": 128.0}.get(kind, 512.0)), 2)
    # a tool no larger than an eighth of the scene
    c["r1"] = min(c["r1"], 2.0 ** c["depth"] / 16)
    return c


def _cameras(case, seed, n):
    """n poses spread over a seeded camera path around the scene."""
    return [_capi.Camera.from_params(p)
            for p in workloads.catmull_rom_path(case["depth"], n, case["width"], case["height"], seed=seed)]


def _mixed(case, seed):
    return [hd.editor_from_tuple(e)
            for e in workloads.mixed_edits(case["depth"], case["edits"], (case["r0"], case["r1"]), seed=seed)]


def _coloured_editors(case, seed):
    """Carves, fills, paints, copies, noise spheres and flood fills in turn,
    and 4096 voxels around them."""
    n, depth, r = case["edits"], case["depth"], (case["r0"], case["r1"])
    rng = np.random.default_rng(seed)
    paint = workloads.paint_copy_edits(depth, n, n, r, copy_radius=r[1], copy_offset=1 << (depth - 4), seed=seed)
    noise = workloads.noise_fill_edits(depth, n, n, r, (r[0], max(r[0] + 1.0, r[1] / 2)), seed=seed)
    mixed = workloads.mixed_edits(depth, n, r, seed=seed, mix=(0.5, 0.5))
    picks = [mixed, paint[:n], mixed, paint[n:], noise[:n], noise[n:]]
    edits = [picks[i % 6][i] for i in range(n)]
    centres = np.array([e[1] for e in edits])[rng.integers(0, n, 4096)]
    points = centres + rng.uniform(-r[1], r[1], (4096, 3))
    points = np.clip(np.floor(points), 0, (1 << depth) - 1).astype(np.uint32)
    return [hd.editor_from_tuple(e) for e in edits], points


def prepare(case, seed):
    kind, depth = case["kind"], case["depth"]
    s = {"case": dict(case), "kind": kind}
    if kind in ("frame", "colour_frame"):
        s["dag"] = _shared(depth, kind == "colour_frame")
        s["camera"] = _cameras(case, seed, 8)[seed % 8]
        s["tracer"] = hd.DAGTracer(case["width"], case["height"])
    elif kind in ("views", "views_host"):
        n, px = case["views"], case["width"] * case["height"]
        s["dag"] = _shared(depth)
        s["cameras"] = (_capi.Camera * n)(*_cameras(case, seed, n))
        s["light"] = (C.c_float * 3)(*LIGHT)
        on = {"device": "cuda"} if kind == "views" else {"pin_memory": True}
        s["paths"] = torch.zeros((n, case["height"], case["width"], 4), dtype=torch.int32, **on)
        s["mask"] = torch.zeros((n, case["height"], case["width"]), dtype=torch.uint8, **on)
        assert px * n < 2 ** 32
    elif kind == "coloured":
        s["dag"] = _load(depth, True)
        s["editors"], s["points"] = _coloured_editors(case, seed)
    elif kind == "serve":
        s["dag"] = _load(depth)
        trace = workloads.serving_trace(depth, case["requests"], 400.0, seed=seed, r_range=(case["r0"], case["r1"]),
                                        resolutions=workloads.RESOLUTIONS[:2])
        reqs = []
        for what, at, p in trace:
            if what == "edit":  # without colours a paint becomes a fill
                reqs.append(hd.edit_request(at, hd.editor_from_tuple((1 if p[0] == 4 else p[0], p[1], p[2]))))
            else:
                reqs.append(hd.render_request(at, p[0], p[1], p[2]))
        s["requests"] = reqs
    else:
        s["dag"] = _load(depth)
        if kind == "edits_single" and depth == 10:
            s["editors"] = [hd.editor_from_tuple(e) for e in
                            workloads.carve_edits(depth, case["edits"], (case["r0"], case["r1"]), seed=seed)]
        else:
            s["editors"] = _mixed(case, seed)
    if kind in ("edits_single", "edit_batch", "gc", "serve"):
        s["root"] = s["dag"].firstNodeIndex
    return s


def run(s):
    kind, dag = s["kind"], s["dag"]
    if kind == "frame":
        tr = s["tracer"]
        tr.resolve_paths(s["camera"], dag)
        tr.resolve_shadows(s["camera"], dag, BIAS, LIGHT)
        return tr.paths, tr.shadows
    if kind == "colour_frame":
        tr = s["tracer"]
        tr.resolve_paths(s["camera"], dag)
        return tr.paths, tr.resolve_colors(dag).view(np.int32)
    if kind in ("views", "views_host"):
        c = s["case"]
        args = (dag.handle, s["cameras"], c["views"], c["width"], c["height"], s["paths"].data_ptr(), s["light"], BIAS,
                s["mask"].data_ptr())
        if kind == "views":
            dag._check(_capi.lib().hd_trace_views(*args, None))
        else:
            dag._check(_capi.lib().hd_trace_views_host(*args, 0, None))
        return s["paths"], s["mask"]
    if kind == "coloured":
        stats = [dag.edit_threads(e) for e in s["editors"]]
        root = dag.firstNodeIndex
        colours = dag.get_colors(s["points"]).astype(np.int64)
        for _ in s["editors"]:
            dag.undo()
        return {"counters": _counters(stats), "root": root, "colours": colours, "sizes": _bucket_sizes(dag)}
    dag.firstNodeIndex = s["root"]
    if kind == "edits_single":
        stats = [dag.edit_threads(e) for e in s["editors"]]
        return {"counters": _counters(stats), "root": dag.firstNodeIndex, "sizes": _bucket_sizes(dag)}
    if kind == "edit_batch":
        _, per = dag.edit_batch(s["editors"], per_edit=True)
        return {"counters": _counters(per), "root": dag.firstNodeIndex, "sizes": _bucket_sizes(dag)}
    if kind == "gc":
        total = dag.edit_batch(s["editors"])
        dag.firstNodeIndex = s["root"]
        dag.remove_stale_nodes()
        s["root"] = dag.firstNodeIndex
        return {"counters": _counters([total]), "root": s["root"], "sizes": _bucket_sizes(dag)}
    results, stats = dag.serve(s["requests"], continuous=True, max_renders=3, realtime=False, light=LIGHT,
                               shadow_bias=BIAS)
    rows = np.array([[r.root, r.status, r.edits_before, r.num_voxels] for r in results], np.int64)
    sums = np.array([r.checksum for r in results], np.uint64).view(np.int64)
    return {"results": rows, "checksums": sums, "refused": int(stats.refused), "sizes": _bucket_sizes(dag)}


def exact(case, seed):
    """Every output is a whole number."""
    return None


def _table_words(depth):
    """Words of the solid scene's nodes, about (152 M at depth 15)."""
    return 152.0e6 / 3.4 ** (15 - depth)


def _edit_bytes(r):
    """One edit of radius r: the 4^3 leaves its surface crosses read and
    written (8 B each way), and about half as many interior words above."""
    leaves = max(1.0, 4 * math.pi * r * r / 16 * 1.5)
    return leaves * 24 + 2048


def work(case):
    kind = case["kind"]
    if "r0" in case:
        a, b = case["r0"], case["r1"]
        # mean over a log-uniform radius
        per_edit = sum(_edit_bytes(a * (b / a) ** (i / 16)) for i in range(17)) / 17
    if kind in ("frame", "views", "views_host", "colour_frame"):
        # a path (16 B) and a mask byte or a colour out per pixel, and the
        # leaf a pixel's ray ends in
        px = case["width"] * case["height"] * case.get("views", 1)
        return {"bytes": px * (16.0 + (4 if kind == "colour_frame" else 1) + 8), "flops": 0.0}
    if kind in ("edits_single", "edit_batch"):
        return {"bytes": case["edits"] * per_edit, "flops": 0.0}
    if kind == "coloured":
        # the tool's voxels on the surface carry a colour: 8 B read and 8 B
        # written each, besides the nodes
        r = math.sqrt(case["r0"] * case["r1"])
        return {"bytes": case["edits"] * (per_edit + 16 * math.pi * r * r), "flops": 0.0}
    if kind == "gc":
        return {"bytes": case["edits"] * per_edit + 8 * _table_words(case["depth"]), "flops": 0.0}
    renders = 0.3 * case["requests"]
    return {"bytes": 0.7 * case["requests"] * per_edit + renders * 1.5e6 * 25, "flops": 0.0}
