"""hd_edit_apply's two geometry paths (the persistent launch; level by level
for edits of over 2^22 entries in a level) against the oracle on both sides
of the line, and edits of two contexts from two threads at once."""
import threading

import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
DEPTH = 10


@pytest.mark.parametrize("radius", [2.0, 300.0, 330.0])
def test_paint_on_both_sides_of_the_entry_line(gpu, radius):
    """A paint (no is_full / is_empty exits) descends into every node of its
    sphere: 8 x 77^3 entries bound the leaf level at radius 300, 8 x 84^3 (over
    2^22) at 330."""
    T = workloads.color_tree_levels(DEPTH)
    words = po.generate_basic_dag(workloads.SEED_SCENE, DEPTH, T, flags=po.SCENE_SHELL)
    ot = po.Table(po.default_config(DEPTH, T))
    ot.load_basic_dag(words)
    col = po.Colors(ot)
    col.from_scene(workloads.SEED_COLORS)
    d = hd.HashDAG(DEPTH)
    d.load_from_DAG(words)
    d.colors_from_scene(workloads.SEED_COLORS)
    rng = np.random.default_rng(3)
    surface = scene.surface_points(workloads.SEED_SCENE, DEPTH, 500, rng)
    near = surface[np.argsort(np.abs(surface - 512.0).sum(axis=1))]  # the most central first
    c = tuple(float(v) + 0.5 for v in near[0])
    carve = min(radius, 40.0)
    for tool, editor, r in ((4, hd.SpherePaintEditor(c, radius), radius),
                            (0, hd.SphereEditor(c, carve, adding=False), carve)):
        so, s = col.edit(tool, c, r), d.edit_threads(editor)
        assert (s.num_voxels, s.num_nodes, s.find_or_add_calls, s.nodes_added) == \
            (so.num_voxels, so.num_nodes, so.find_or_add_calls, so.nodes_added)
        assert d.firstNodeIndex == ot.root
    assert d.history() == (2, 0)
    pts = near.astype(np.uint32)
    pts = pts[d.get_values(pts).astype(bool)]
    assert len(pts)
    got = d.get_colors(pts)
    assert [tuple(int(v) for v in row) for row in got] == [col.get_color(*(int(v) for v in p)) for p in pts]
    d.free()


def test_two_threads_edit_their_contexts(gpu):
    import torch
    edits = [workloads.mixed_edits(DEPTH, 24, (4.0, 64.0), seed=s) for s in (41, 42)]
    want = []
    for e in edits:
        d = hd.HashDAG(DEPTH)
        d.generate_scene(workloads.SEED_SCENE)
        want.append([(d.edit_threads(hd.editor_from_tuple(x)).num_voxels, d.firstNodeIndex) for x in e])
        d.free()
    dags, got, errors = [], [None, None], []
    for _ in edits:
        d = hd.HashDAG(DEPTH)
        d.generate_scene(workloads.SEED_SCENE)
        s = torch.cuda.Stream()
        d._check(hd._capi.lib().hd_set_stream(d.handle, s.cuda_stream))
        dags.append((d, s))

    def work(k):
        try:
            d = dags[k][0]
            got[k] = [(d.edit_threads(hd.editor_from_tuple(x)).num_voxels, d.firstNodeIndex) for x in edits[k]]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    assert got == want
    for d, _ in dags:
        d.free()
