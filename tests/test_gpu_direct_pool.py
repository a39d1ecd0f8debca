"""A direct-mapped pool (a page for every virtual page, the default) against
a pool whose pages are handed out in claim order: the same table by virtual
address, page counts, frames and exports, through edits, both GCs and tables
carried from one kind to the other."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads
from tests.helpers import table_digest

pytestmark = pytest.mark.gpu


def _pair(depth):
    """(direct, paged) contexts with the seeded scene."""
    a = hd.HashDAG(depth)
    a.generate_scene(workloads.SEED_SCENE)
    b = hd.HashDAG(config=hd.default_config(depth, pool_pages=int(a.config.pool_pages) // 2))
    b.generate_scene(workloads.SEED_SCENE)
    return a, b


def _same(a, b, depth):
    sa, sb = a.level_stats(), b.level_stats()
    assert a.firstNodeIndex == b.firstNodeIndex
    assert sa.pages_used == sb.pages_used
    assert list(sa.words) == list(sb.words) and list(sa.nodes) == list(sb.nodes)
    bits = workloads.top_bucket_bits(depth)
    assert table_digest(a.export_table(), depth, bits) == table_digest(b.export_table(), depth, bits)
    cam = workloads.orbit_camera(depth, 203, 117)
    frames = []
    for d in (a, b):
        tr = hd.DAGTracer(203, 117)
        tr.resolve_paths(cam, d)
        tr.resolve_shadows(cam, d)
        frames.append((tr.get_paths(), tr.get_shadows()))
    assert np.array_equal(frames[0][0], frames[1][0]) and np.array_equal(frames[0][1], frames[1][1])


@pytest.mark.parametrize("depth", [8, 11])
def test_edits_gcs_and_round_trips(gpu, depth, tmp_path):
    a, b = _pair(depth)
    _same(a, b, depth)
    edits = [hd.editor_from_tuple(e) for e in workloads.mixed_edits(depth, 12, (4.0, 2.0 ** depth / 16), seed=31)]
    for release in (False, True):
        for d in (a, b):
            d.edit_batch(edits[:8])
            for e in edits[8:]:
                d.edit_threads(e)
        _same(a, b, depth)
        for d in (a, b):
            d.remove_stale_nodes(release_pages=release)
        _same(a, b, depth)
    # exports, each loaded into the other kind; snapshots alike
    ta, tb = a.export_table(), b.export_table()
    a.import_table(tb)
    b.import_table(ta)
    _same(a, b, depth)
    back = a.export_table()  # page numbers and pages as they came
    assert all(np.array_equal(back[k], tb[k]) for k in ("page_table", "pool", "bucket_sizes"))
    pa, pb = str(tmp_path / "a"), str(tmp_path / "b")
    a.save_snapshot(pa)
    b.save_snapshot(pb)
    a.load_snapshot(pb)
    b.load_snapshot(pa)
    _same(a, b, depth)
    for d in (a, b):
        for e in edits:
            d.edit_threads(e)
    _same(a, b, depth)
    a.free()
    b.free()


def test_addresses_past_the_table_read_as_empty(gpu):
    """A corrupt child pointer outside the virtual space: the walk finds an
    empty node there, whichever way pages are placed."""
    depth = 8
    a, b = _pair(depth)
    for d in (a, b):
        t = d.export_table()
        root = int(t["root"])
        at = int(t["page_table"][root // 512]) * 512 + root % 512
        n = bin(int(t["pool"][at]) & 0xFF).count("1")
        t["pool"][at + 1:at + 1 + n] = 0xFFFFFE00
        d.import_table(t)
        tr = hd.DAGTracer(64, 48)
        tr.resolve_paths(workloads.orbit_camera(depth, 64, 48), d)
        assert not tr.get_paths().any()
        d.free()
