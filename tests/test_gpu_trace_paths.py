"""The forms a walk can take - rays along the axes and from far outside (the
walk that expects infinities), tiles whose rays all miss the root, the last
rays of a shadow pass shared among a warp's lanes - against the oracle, in the
single-view and the many-view launches."""
import ctypes as C
import os

import numpy as np
import pytest

import hashdag_gb300 as hd
from hashdag_gb300 import workloads
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
DEPTH = 8
_cache = {}


def _scene():
    if not _cache:
        d = hd.HashDAG(DEPTH)
        d.generate_scene(workloads.SEED_SCENE)
        t = po.Table(po.default_config(DEPTH))
        t.load_basic_dag(po.generate_basic_dag(workloads.SEED_SCENE, DEPTH, workloads.color_tree_levels(DEPTH)))
        _cache["s"] = d, t
    return _cache["s"]


def _cameras(w, h):
    e = float(1 << DEPTH)
    mid = np.full(3, e / 2)
    cams = [workloads.orbit_camera(DEPTH, w, h)]
    for pos, look in [
        (mid + [1.5 * e, 0, 0], mid),                        # along x: zero components in the middle
        (mid + [0, 0.02 * e, -1.2 * e], mid),                # a zero x component
        (mid + [0.3, 0.7 * e / 2, 0.1], mid + [9, 0, 4]),    # inside the root
        (mid + [1.5 * e, e, 0.2 * e], mid + [4 * e, e, 0]),  # away from it: every ray misses
        (mid + [2.0 ** 25, 2.0 ** 24, 2.0 ** 23], mid),      # far outside
        (np.array([e, e, e]) + 1.0, mid),                    # beside a corner
    ]:
        cams.append(workloads.trace_params(np.asarray(pos, float), np.asarray(look, float), w, h))
    return cams


@pytest.mark.parametrize("fp_mode", [0, 1])
@pytest.mark.parametrize("light", [(0.3, 1.0, 0.2), (0.0, 1.0, 0.0), (-1.0, 0.0, 0.0), (-0.6, 0.1, -1e-30)])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 5), (65, 33)])
def test_walk_forms_match_oracle(gpu, w, h, light, fp_mode):
    import torch
    d, t = _scene()
    d.set_fp_mode(fp_mode)
    poses = _cameras(w, h)
    n = len(poses)
    cams = (hd._capi.Camera * n)(*[hd._capi.Camera.from_params(p) for p in poses])
    paths = torch.full((n * w * h * 4,), -1, dtype=torch.int32, device="cuda")
    mask = torch.full((n * w * h,), 9, dtype=torch.uint8, device="cuda")
    ms = (C.c_float * 2)()
    d._check(hd._capi.lib().hd_trace_views(d.handle, cams, n, w, h, paths.data_ptr(), (C.c_float * 3)(*light), 1.0,
                                           mask.data_ptr(), ms))
    paths = paths.cpu().numpy().view(np.uint32).reshape(n, h, w, 4)
    mask = mask.cpu().numpy().reshape(n, h, w)
    tr = hd.DAGTracer(w, h)
    for v, pose in enumerate(poses):
        want_p, want_m = t.trace_frame(pose, w, h, light, 1.0, fp_mode=fp_mode, threads=os.cpu_count() or 4)
        assert np.array_equal(paths[v], want_p), v
        assert np.array_equal(mask[v], want_m), v
        tr.resolve_paths(pose, d)
        tr.resolve_shadows(pose, d, 1.0, light)
        assert np.array_equal(tr.get_paths().reshape(h, w, 4), want_p), v
        assert np.array_equal(tr.get_shadows(), want_m), v
    d.set_fp_mode(0)
