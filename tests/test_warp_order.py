"""Places where lanes of a warp hand each other data through memory: ballots and
shuffles order no memory, so a __syncwarp stands between the write and the
read.  Read from the kernels' sources; the GPU tests cover the results."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hashdag_gb300", "csrc")


def body(file, name):
    """The body of function `name`, comments taken out."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    at = src.index("{", re.search(r"\b" + name + r"\([^;{]*\)\s*\{", src).start())
    depth = 0
    for k in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[at:k + 1]
    raise AssertionError(name)


def test_split_walks_reads_a_givers_stack_behind_its_writes():
    b = body("hd_trace.cu", "split_walks")
    reads = [m.start() for m in re.finditer(r"stack\.(index_of|masks_of)\(", b)]
    syncs = [m.start() for m in re.finditer(r"__syncwarp\(\)", b)]
    # after the givers' writes (before the call), and before their next ones
    assert len(reads) == 2
    assert any(s < min(reads) for s in syncs) and any(s > max(reads) for s in syncs)


def test_tiny_candidates_returns_behind_a_warp_barrier():
    """Its entries' results are read by other lanes at the level above."""
    b = body("hd_edit_persist.cu", "tiny_candidates")
    for m in re.finditer(r"\breturn\b", b):
        before = b[:m.start()].rstrip()
        assert re.search(r"__syncwarp\(\);(\s*\{)?$", before), before[-120:]
