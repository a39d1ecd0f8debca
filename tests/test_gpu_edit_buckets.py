"""Edits of tables whose levels have other numbers of buckets than the
defaults' 2^10 to 2^17, against the oracle: single edits and the same edits as
one batch."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
DEPTH = 10
# levels of some 200,000 entries and 80,000 candidates, a sphere's distinct
# ones and a box's equal ones, then small edits
EDITS = [(1, (512.0, 512.0, 512.0), 300.0), (3, (500.0, 510.0, 490.0), 181.0), (0, (512.0, 512.0, 512.0), 260.0),
         (0, (300.5, 640.0, 512.25), 33.0), (2, (512.0, 400.0, 512.0), 6.0)]


def check(kw, batched, mode=1):
    words = po.generate_basic_dag(workloads.SEED_SCENE, DEPTH, workloads.color_tree_levels(DEPTH))
    cfg = po.default_config(DEPTH)
    for k, v in kw.items():
        setattr(cfg, k, v)
    ot = po.Table(cfg)
    ot.load_basic_dag(words)
    want = [ot.edit(*e) for e in EDITS]
    d = hd.HashDAG(config=hd.default_config(DEPTH, **kw))
    d.load_from_DAG(words)
    eds = [hd.editor_from_tuple(e) for e in EDITS]
    if batched:
        d.batch_tuning = hd.BatchTuning(4, 4, 304, mode)
        _, got = d.edit_batch(eds, per_edit=True)
    else:
        got = [d.edit_threads(e) for e in eds]
    for a, b in zip(got, want):
        assert (a.num_voxels, a.num_nodes, a.find_or_add_calls, a.nodes_added) == \
            (b.num_voxels, b.num_nodes, b.find_or_add_calls, b.nodes_added)
    assert d.firstNodeIndex == ot.root
    assert np.array_equal(d.export_table()["bucket_sizes"], ot.export()["bucket_sizes"])
    d.free()


@pytest.mark.parametrize("batched", [False, True])
def test_few_buckets(gpu, batched):
    """2^6 buckets: two sort passes of 16 digits, fewer than a warp's lanes."""
    check({"top_bucket_bits": 6, "top_bucket_size": 1 << 16, "pool_pages": 200000}, batched)


@pytest.mark.parametrize("batched, mode", [(False, 1), (True, 1), (True, 0)])
def test_many_buckets(gpu, batched, mode):
    """2^18 and 2^19 buckets, more than two passes of 2^9 digits sort: such
    edits are made level by level."""
    check({"top_levels": 7, "top_bucket_bits": 18, "top_bucket_size": 512, "low_bucket_bits": 19,
           "low_bucket_size": 512, "pool_pages": 400000}, batched, mode)
