"""Find-or-add of big levels through the CTAs' queues, and by the grid's sort
when a queue overflows (the equal candidates of a box's faces), on both sides
of the sizes at which one CTA, the queues and the sort take a level over:
against the oracle, in a batch and edit by edit."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
SPHERE_REMOVE, SPHERE_ADD, BOX_REMOVE, BOX_ADD = range(4)


@pytest.mark.parametrize("batch", [False, True])
def test_levels_of_all_sizes_match_oracle(gpu, batch):
    depth = 11
    T = workloads.color_tree_levels(depth)
    words = po.generate_basic_dag(workloads.SEED_SCENE, depth, T)
    ot = po.Table(po.default_config(depth, T))
    ot.load_basic_dag(words)
    d = hd.HashDAG(depth)
    d.load_from_DAG(words)
    rng = np.random.default_rng(17)
    places = scene.surface_points(workloads.SEED_SCENE, depth, 64, rng)
    edits = []
    for k, r in enumerate((6.0, 9.5, 13.0, 17.0, 24.0, 33.0, 47.0, 90.0, 200.0)):
        for tool in (SPHERE_ADD, BOX_ADD, SPHERE_REMOVE, BOX_REMOVE):
            edits.append((tool, tuple(float(v) + 0.5 for v in places[(4 * k + tool) % 64]), r))
    want = [ot.edit(*e) for e in edits]
    ed = [hd.editor_from_tuple(e) for e in edits]
    got = d.edit_batch(ed, per_edit=True)[1] if batch else [d.edit_threads(e) for e in ed]
    for e, g, w in zip(edits, got, want):
        assert (g.num_voxels, g.num_nodes, g.find_or_add_calls, g.nodes_added) == \
            (w.num_voxels, w.num_nodes, w.find_or_add_calls, w.nodes_added), e
    assert d.firstNodeIndex == ot.root
    d.free()
