"""Single edits whose persistent launch cannot finish: a CTA that never reaches a
grid barrier (bounded waits, tests' hook), or a launch that the device refuses.
The edit is then made level by level: the same voxels, colours and counters as
without the failure, one undo frame, and the context goes on."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import scene, workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
DEPTH = 10
SKIP, REFUSED = 5, 1 << 20


def _context(colors):
    d = hd.HashDAG(DEPTH)
    d.generate_scene(workloads.SEED_SCENE, shell=colors)
    if colors:
        d.colors_from_scene(workloads.SEED_COLORS)
    return d


def _fingerprint(d):
    t = d.export_table()
    ot = po.Table(po.default_config(DEPTH, pool_pages=int(t["pool"].size // 512) + 8))
    ot.import_(t)
    return ot.fingerprint()


@pytest.mark.parametrize("cta", [SKIP, REFUSED])
@pytest.mark.parametrize("colors", [False, True])
# by CTA 0 alone; with grid steps; a copy, which is not the same when made twice
@pytest.mark.parametrize("kind", ["small", "large", "copy"])
def test_edit_is_made_level_by_level(gpu, kind, colors, cta):
    rng = np.random.default_rng(11)
    near = scene.surface_points(workloads.SEED_SCENE, DEPTH, 300, rng)
    near = near[np.argsort(np.abs(near - 512.0).sum(axis=1))]
    c = tuple(float(v) for v in near[0])
    edit = {"small": hd.SphereEditor(c, 5.0, adding=False),
            "large": hd.SphereEditor(c, 150.0, adding=False),
            "copy": hd.CopyEditor(c, 20.0, c, tuple(v + 16.0 for v in c))}[kind]
    after = hd.SphereEditor(tuple(float(v) for v in near[40]), 30.0, adding=True)
    want, got = _context(colors), _context(colors)
    a = want.edit_threads(edit)
    got.set_test_barrier_skip(cta, 20)
    b = got.edit_threads(edit)
    assert (a.num_voxels, a.num_nodes, a.find_or_add_calls) == (b.num_voxels, b.num_nodes, b.find_or_add_calls)
    if cta == REFUSED:  # nothing had been appended
        assert a.nodes_added == b.nodes_added and want.firstNodeIndex == got.firstNodeIndex
    assert got.history() == (1, 0)
    for d in (want, got):  # (the failure was for that one launch)
        d.edit_batch([after])
    pts = np.clip(np.concatenate([near, np.array(c) + rng.uniform(-160, 160, (30000, 3))]), 0, 1023).astype(np.uint32)
    for _ in range(3):  # after both edits, with one undone, with both
        v = want.get_values(pts)
        assert np.array_equal(v, got.get_values(pts))
        if colors:
            assert np.array_equal(want.get_colors(pts[v != 0]), got.get_colors(pts[v != 0]))
        assert _fingerprint(want) == _fingerprint(got)
        if got.history()[0]:
            for d in (want, got):
                d.undo()
    want.free()
    got.free()


@pytest.mark.parametrize("share", [0.99, 0.95, 0.62])
@pytest.mark.parametrize("colors", [False, True])
def test_edit_without_room_for_its_bounds(gpu, colors, share):
    """The launch's arrays are bounds on an edit's entries.  An edit that does
    not get them (or the colours' beside them) takes the entries' own: half the
    memory, the same result."""
    rng = np.random.default_rng(12)
    near = scene.surface_points(workloads.SEED_SCENE, DEPTH, 300, rng)
    near = near[np.argsort(np.abs(near - 512.0).sum(axis=1))]
    c = tuple(float(v) for v in near[0])
    edits = [hd.SpherePaintEditor(c, 150.0), hd.SphereEditor((512.0, 512.0, 512.0), 300.0, adding=False),
             hd.SphereEditor(c, 20.0, adding=True)]
    for edit in edits[:2]:
        want, got = _context(colors), _context(colors)
        a = want.edit_threads(edit)
        before = got.memory_stats()["scratch"]
        limit = before + int(share * (want.memory_stats()["scratch"] - before))
        got.set_test_scratch_limit(limit)
        b = got.edit_threads(edit)
        assert got.memory_stats()["scratch"] <= limit
        assert (a.num_voxels, a.num_nodes, a.find_or_add_calls) == (b.num_voxels, b.num_nodes, b.find_or_add_calls)
        for d in (want, got):
            d.edit_threads(edits[2])
        assert got.history() == (2, 0)
        got.set_test_scratch_limit(0)
        pts = np.clip(np.concatenate([near, 512.0 + rng.uniform(-310, 310, (30000, 3))]), 0, 1023).astype(np.uint32)
        v = want.get_values(pts)
        assert np.array_equal(v, got.get_values(pts))
        if colors:
            assert np.array_equal(want.get_colors(pts[v != 0]), got.get_colors(pts[v != 0]))
        assert _fingerprint(want) == _fingerprint(got)
        # too little for that as well is an error, and leaves the context as it is
        root = got.firstNodeIndex
        got.set_test_scratch_limit(1)
        if share < 0.9:
            with pytest.raises(hd.HashDagError) as ei:
                got.edit_threads(hd.SphereEditor((512.0, 512.0, 512.0), 460.0, adding=False))
            assert ei.value.status == hd._capi.HD_ERR_OOM
            assert got.firstNodeIndex == root and got.history() == (2, 0)
        want.free()
        got.free()


@pytest.mark.parametrize("mode", [1, 0])
def test_batch_without_room_for_its_bounds(gpu, mode):
    """A batch whose level arrays do not fit is made edit by edit."""
    edits = [hd.editor_from_tuple(e) for e in workloads.mixed_edits(DEPTH, 10, (8.0, 60.0), seed=9)]
    edits.insert(4, hd.SphereEditor((512.0, 512.0, 512.0), 300.0, adding=False))
    want, got = _context(False), _context(False)
    for d in (want, got):
        d.batch_tuning = hd.BatchTuning(4, 4, 304, mode)
    _, a = want.edit_batch(edits, per_edit=True)
    got.set_test_scratch_limit(want.memory_stats()["scratch"] * 6 // 10)
    _, b = got.edit_batch(edits, per_edit=True)
    assert [(s.num_voxels, s.num_nodes, s.find_or_add_calls, s.nodes_added) for s in a] == \
        [(s.num_voxels, s.num_nodes, s.find_or_add_calls, s.nodes_added) for s in b]
    assert want.firstNodeIndex == got.firstNodeIndex and want.history() == got.history() == (11, 0)
    want.free()
    got.free()
