"""hd_autotune_batch's device copy of a table (tests/copy_table_check.cu, built
with nvcc against the library's objects)."""
import glob
import os
import subprocess

import pytest

from hashdag_gb300 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_copies_are_the_table(gpu, tmp_path):
    build.build()
    objs = [o for o in glob.glob(os.path.join(build.OUT_DIR, "*.o")) if not o.endswith("hd_edit_batch.o")]
    exe = str(tmp_path / "copy_table_check")
    r = subprocess.run([build._nvcc()] + build.ARCH + build.NVCC_FLAGS +
                       ["-I", build.INCLUDE, os.path.join(ROOT, "tests", "copy_table_check.cu")] + objs +
                       ["-o", exe, "-lcudart"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
