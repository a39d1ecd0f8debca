"""A served batch whose edits are made one by one (a noise sphere among them)
and that fills the pool: the edits before the full one count once, the rest are
refused, as when each is applied by itself."""
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import _capi, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plain_first", [False, True])
def test_full_pool_in_a_batch_of_single_edits(gpu, plain_first):
    depth = 10
    d = hd.HashDAG(depth)
    d.generate_scene(workloads.SEED_SCENE)
    used = int(d.level_stats().pages_used)
    d.free()
    cfg = hd.default_config(depth)
    cfg.pool_pages = used + 80
    edits = workloads.mixed_edits(depth, 8, (6.0, 12.0), seed=5)
    if plain_first:  # carves and fills alone: a batch of another kind before it
        edits = edits[:6] + workloads.noise_fill_edits(depth, 16, 0, (8.0, 32.0))
    else:
        edits = edits[:2] + workloads.noise_fill_edits(depth, 16, 0, (8.0, 32.0))
    eds = [hd.editor_from_tuple(e) for e in edits]
    one = hd.HashDAG(config=cfg)
    one.generate_scene(workloads.SEED_SCENE)
    want = []
    for e in eds:
        try:
            one.edit_threads(e)
            want.append(0)
        except hd.HashDagError as x:
            assert x.status == _capi.HD_ERR_POOL_FULL
            want.append(x.status)
    assert 0 < want.count(0) < len(eds)
    served = hd.HashDAG(config=cfg)
    served.generate_scene(workloads.SEED_SCENE)
    if plain_first:
        served.edit_batch(eds[:6])
    done = 6 if plain_first else 0
    res, st = served.serve([hd.edit_request(0.0, e) for e in eds[done:]], continuous=True, realtime=False,
                           gc_free_fraction=0.0, batch_edits=True)
    assert [r.status for r in res] == want[done:]
    assert served.firstNodeIndex == one.firstNodeIndex
    assert served.history() == one.history()
    assert st.refused == len(want) - want.count(0)
    one.free()
    served.free()
