"""Undo and redo of edits that replace few or many colour leaves (up to 2^14 come
back with the edit's counts, more on their own), against the oracle."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


# tasks of 8^3 voxels: at most 24^3, and at least 27^3
@pytest.mark.parametrize("radius, many", [(88.0, False), (112.0, True)])
def test_undo_and_redo_of_a_filled_box(gpu, radius, many):
    depth, T = 10, 7
    words = po.generate_basic_dag(workloads.SEED_SCENE, depth, T, flags=po.SCENE_SHELL)
    ot = po.Table(po.default_config(depth, T))
    ot.load_basic_dag(words)
    col = po.Colors(ot)
    col.from_scene(workloads.SEED_COLORS)
    d = hd.HashDAG(config=hd.default_config(depth, color_tree_levels=T))
    d.load_from_DAG(words)
    d.colors_from_scene(workloads.SEED_COLORS)
    rng = np.random.default_rng(5)
    s = scene.surface_points(workloads.SEED_SCENE, depth, 3000, rng)
    c = tuple(float(v) for v in s[np.argsort(np.abs(s - 512.0).sum(axis=1))][0])
    pts = np.concatenate([s, np.array(c) + rng.uniform(-1.2 * radius, 1.2 * radius, (20000, 3))]).astype(np.uint32)

    def state():
        v = d.get_values(pts) != 0
        assert [tuple(int(x) for x in row) for row in d.get_colors(pts[v])] == \
            [tuple(col.get_color(*(int(x) for x in p))) for p in pts[v]]
        return v.sum()

    edits = [(4, hd.SpherePaintEditor(c, 0.6 * radius, 0x30A0C0), 0.6 * radius), (3, hd.BoxEditor(c, radius, True), radius),
             (4, hd.SpherePaintEditor(c, 0.9 * radius, 0xC03060), 0.9 * radius)]
    before = state()
    for tool, editor, r in edits:
        d.edit_threads(editor)
        col.edit(tool, c, r, rgb={0.6 * radius: 0x30A0C0, 0.9 * radius: 0xC03060}.get(r, 0xFF0000))
        assert d.firstNodeIndex == ot.root
        after = state()
    assert after > before
    for _ in edits:
        d.undo()
        col.undo()
        state()
    assert state() == before
    for _ in edits:
        d.redo()
    assert (d.get_values(pts) != 0).sum() == after
    d.free()
