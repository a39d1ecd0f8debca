"""GCs inside the serving loop of a pool a little larger than the scene: one
edit after the other, pages kept by the GCs, nothing refused, and a GC only
after a part of the pool was claimed (one per edit or two maps pages with each
run, and fills the pool by itself)."""
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("release", [False, True])
def test_small_pool_refuses_nothing(gpu, release):
    depth = 13
    d = hd.HashDAG(depth)
    d.generate_scene(workloads.SEED_SCENE)
    pool = int(d.level_stats().pages_used * 1.12) + 1
    d.free()
    cfg = hd.default_config(depth)
    cfg.pool_pages = pool
    d = hd.HashDAG(config=cfg)
    d.generate_scene(workloads.SEED_SCENE)
    reqs = []
    for what, at, p in workloads.serving_trace(depth, 300, 400.0, r_range=(4.0, 128.0)):
        if what == "edit":
            reqs.append(hd.edit_request(at, hd.editor_from_tuple((1 if p[0] == 4 else p[0], p[1], p[2]))))
    res, st = d.serve(reqs, continuous=False, realtime=False, gc_free_fraction=0.1, release_pages=release,
                      batch_edits=False)
    s = st.as_dict()
    assert s["refused"] == 0
    assert s["edits"] == len(reqs)
    assert 0 < s["gcs"] < len(reqs) // 8
    d.free()
