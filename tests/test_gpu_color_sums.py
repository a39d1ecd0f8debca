"""Fills on both sides of 2^15 pieces of colours, from which on the pieces are
summed by a scan over the grid, against the oracle."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius, over", [(60.0, False), (112.0, True)])
def test_filled_box_matches_oracle(gpu, radius, over):
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
    rng = np.random.default_rng(4)
    s = scene.surface_points(workloads.SEED_SCENE, depth, 200, rng)
    c = tuple(float(v) for v in s[np.argsort(np.abs(s - 512.0).sum(axis=1))][0])
    # 32^3 voxels a task: 128 pieces of 256 colours
    assert (2 * radius) ** 3 / 256 > 1 << 15 if over else ((2 * radius + 64) / 32) ** 3 * 128 < 1 << 15
    paint = tuple(v + radius for v in c)  # weights beside plain colours
    for tool, editor, centre, r in ((4, hd.SpherePaintEditor(paint, 40.0, 0x20C040), paint, 40.0),
                                    (3, hd.BoxEditor(c, radius, True), c, radius),
                                    (4, hd.SpherePaintEditor(c, radius, 0x4060F0), c, radius)):
        got = d.edit_threads(editor)
        want = col.edit(tool, centre, r, rgb={40.0: 0x20C040}.get(r, 0x4060F0) if tool == 4 else 0xFF0000)
        assert d.firstNodeIndex == ot.root
        assert (got.num_voxels, got.num_nodes) == (want.num_voxels, want.num_nodes)
    pts = (np.asarray(c) + rng.uniform(-1.2 * radius, 1.2 * radius, (30000, 3))).astype(np.uint32)
    pts = pts[d.get_values(pts) != 0]
    assert len(pts) > 10000
    assert [tuple(int(v) for v in row) for row in d.get_colors(pts)] == \
        [tuple(col.get_color(*(int(v) for v in p))) for p in pts]
    d.free()
