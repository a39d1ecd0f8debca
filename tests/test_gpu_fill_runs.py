"""The flood fill's runs: boxes whose rows are shorter than, equal to and longer
than a warp's 32 voxels, of odd and even size, against the oracle."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def test_fills_match_oracle(gpu):
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
    rng = np.random.default_rng(31)
    for r in (1.0, 7.5, 15.5, 16.0, 16.5, 33.0, 47.5):
        x, z = (int(v) for v in rng.integers(100, 900, 2))
        y = next(y for y in range(1022, 0, -1) if ot.get_value(x, y, z))
        # a few walls, so that components meet round corners
        for k in range(3):
            w = (x + 0.5 + 5 * k, y + 0.6 * r, z + 0.5 - 4 * k)
            d.edit_threads(hd.editor_from_tuple((hd.TOOL_BOX_ADD, w, 0.2 * r + 1)))
            col.edit(hd.TOOL_BOX_ADD, w, 0.2 * r + 1)
        c = (x + 0.5, y + 0.3 * r + 1.5, z + 0.5)
        got = d.edit_threads(hd.editor_from_tuple((hd.TOOL_FILL, c, r)))
        want = col.edit(hd.TOOL_FILL, c, r)
        assert d.firstNodeIndex == ot.root, r
        assert (got.num_voxels, got.num_nodes) == (want.num_voxels, want.num_nodes), r
        pts = (np.asarray(c) + rng.uniform(-r, r, (3000, 3))).astype(np.uint32)
        pts = pts[d.get_values(pts) != 0]
        assert [tuple(int(v) for v in row) for row in d.get_colors(pts)] == \
            [tuple(col.get_color(*(int(v) for v in p))) for p in pts], r
    d.free()
