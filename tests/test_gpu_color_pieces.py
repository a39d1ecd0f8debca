"""Colour leaves packed in pieces: tasks whose colours fill several pieces and
more than one macro block (solid balls: up to 32^3 colours in a task), with
and without weights, against the oracle."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [4.0, 9.5, 45.0])
def test_packed_leaves_match_oracle(gpu, radius):
    depth = 10
    T = workloads.color_tree_levels(depth)
    words = po.generate_basic_dag(workloads.SEED_SCENE, depth, T, flags=po.SCENE_SHELL)
    ot = po.Table(po.default_config(depth, T))
    ot.load_basic_dag(words)
    col = po.Colors(ot)
    col.from_scene(workloads.SEED_COLORS)
    d = hd.HashDAG(depth)
    d.load_from_DAG(words)
    d.colors_from_scene(workloads.SEED_COLORS)
    rng = np.random.default_rng(7)
    s = scene.surface_points(workloads.SEED_SCENE, depth, 200, rng)
    c = tuple(float(v) + 0.5 for v in s[np.argsort(np.abs(s - 512.0).sum(axis=1))][0])
    r = radius
    shift = (c[0] + r * 0.5, c[1], c[2])
    for tool, editor, centre, rad in [
            (1, hd.SphereEditor(c, r, adding=True), c, r),
            (4, hd.SpherePaintEditor(shift, r, 0x20C040), shift, r),
            (hd.TOOL_NOISE_ADD, hd.editor_from_tuple((hd.TOOL_NOISE_ADD, shift, r)), shift, r),
            (0, hd.SphereEditor(c, r * 0.4, adding=False), c, r * 0.4)]:
        got = d.edit_threads(editor)
        want = col.edit(tool, centre, rad, rgb=0x20C040 if tool == 4 else 0xFF0000)
        assert d.firstNodeIndex == ot.root, tool
        assert (got.num_voxels, got.num_nodes) == (want.num_voxels, want.num_nodes), tool
    pts = (np.asarray(c) + rng.uniform(-1.7 * r - 4, 1.7 * r + 4, (30000, 3))).astype(np.uint32)
    pts = pts[d.get_values(pts) != 0]
    assert len(pts) > 100
    assert [tuple(int(v) for v in row) for row in d.get_colors(pts)] == \
        [tuple(col.get_color(*(int(v) for v in p))) for p in pts]
    d.free()


def test_many_tasks_match_oracle(gpu):
    """A paint over most of a 2^11 scene: thousands of tasks, over 2^13 pieces."""
    depth = 11
    T = workloads.color_tree_levels(depth)
    words = po.generate_basic_dag(workloads.SEED_SCENE, depth, T, flags=po.SCENE_SHELL)
    ot = po.Table(po.default_config(depth, T))
    ot.load_basic_dag(words)
    col = po.Colors(ot)
    col.from_scene(workloads.SEED_COLORS)
    d = hd.HashDAG(depth)
    d.load_from_DAG(words)
    d.colors_from_scene(workloads.SEED_COLORS)
    rng = np.random.default_rng(9)
    s = scene.surface_points(workloads.SEED_SCENE, depth, 3000, rng)
    c = tuple(float(v) + 0.5 for v in s[np.argsort(np.abs(s - 1024.0).sum(axis=1))][0])
    got = d.edit_threads(hd.SpherePaintEditor(c, 800.0, 0x40A0F0))
    want = col.edit(4, c, 800.0, rgb=0x40A0F0)
    assert d.firstNodeIndex == ot.root
    assert (got.num_voxels, got.num_nodes) == (want.num_voxels, want.num_nodes)
    assert got.num_voxels > 256 * 8192
    pts = s.astype(np.uint32)
    pts = pts[d.get_values(pts) != 0]
    assert len(pts) > 100

    def colours():
        return [tuple(int(v) for v in row) for row in d.get_colors(pts)]

    painted = colours()
    assert painted == [tuple(col.get_color(*(int(v) for v in p))) for p in pts]
    d.undo()
    assert colours() != painted
    d.redo()
    assert colours() == painted
    d.free()
