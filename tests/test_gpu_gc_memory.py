"""A GC without room for the nodes it stages gathers every level again, with the
same result; without room for that either it is refused and changes nothing."""
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import _capi, workloads
from tests.helpers import table_digest

pytestmark = pytest.mark.gpu
DEPTH = 10


def _edited():
    d = hd.HashDAG(DEPTH)
    d.generate_scene(workloads.SEED_SCENE)
    for e in workloads.mixed_edits(DEPTH, 6, (16.0, 200.0), seed=8):
        d.edit_threads(hd.editor_from_tuple(e))
    return d


@pytest.mark.parametrize("release", [False, True])
def test_gc_without_room(gpu, release):
    want, got, none = _edited(), _edited(), _edited()
    want.remove_stale_nodes(release_pages=release)
    limit = want.memory_stats()["scratch"] - 1
    got.set_test_scratch_limit(limit)
    got.remove_stale_nodes(release_pages=release)
    assert got.memory_stats()["scratch"] <= limit
    assert want.firstNodeIndex == got.firstNodeIndex
    got.set_test_scratch_limit(0)
    assert table_digest(want.export_table(), DEPTH) == table_digest(got.export_table(), DEPTH)
    root, table = none.firstNodeIndex, table_digest(none.export_table(), DEPTH)
    none.set_test_scratch_limit(1 << 20)
    with pytest.raises(hd.HashDagError) as ei:
        none.remove_stale_nodes(release_pages=release)
    assert ei.value.status == _capi.HD_ERR_OOM
    none.set_test_scratch_limit(0)
    assert none.firstNodeIndex == root and table_digest(none.export_table(), DEPTH) == table
    none.remove_stale_nodes(release_pages=release)
    assert none.firstNodeIndex == want.firstNodeIndex
    for d in (want, got, none):
        d.free()
