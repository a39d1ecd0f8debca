"""Tables go in and out of a direct-mapped pool through a staging buffer: with
little room on the device in smaller pieces, the same arrays and files."""
import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [200 << 10, 1 << 20, 6 << 20])
def test_small_staging(gpu, limit, tmp_path):
    d = hd.HashDAG(10)
    d.generate_scene(workloads.SEED_SCENE)
    d.edit_threads(hd.SphereEditor((512.0, 512.0, 512.0), 60.0, adding=False))
    want = d.export_table()
    d.save_snapshot(str(tmp_path / "a"))
    e = hd.HashDAG(10)
    for x in (d, e):
        x.set_test_scratch_limit(limit + x.memory_stats()["scratch"])
    got = d.export_table()
    assert want.keys() == got.keys() and all(np.array_equal(want[k], got[k]) for k in want)
    d.save_snapshot(str(tmp_path / "b"))
    assert (tmp_path / "a").read_bytes() == (tmp_path / "b").read_bytes()
    e.import_table(want)
    back = e.export_table()
    assert all(np.array_equal(want[k], back[k]) for k in want)
    d.free()
    e.free()
