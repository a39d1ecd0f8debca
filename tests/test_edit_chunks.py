"""The persistent edit kernel's split of a level over its CTAs
(csrc/hd_chunks.cuh), for every grid size a device or a slice of one may have:
CTA k works chunk k and has a row of digit counts, so a level has no more
chunks than the grid has CTAs and its chunks cover it.  Compiled and run on
the host."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hashdag_gb300", "csrc")


def run_host(tmp_path, body, headers):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src = tmp_path / "t.cpp"
    src.write_text("".join(f'#include "{h}"\n' for h in headers) +
                   "#include <cstdio>\nusing namespace hd;\nint main() {\n" + body + "\nreturn 0; }\n")
    exe = str(tmp_path / "t")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_a_level_has_a_chunk_a_cta_at_most(tmp_path):
    run_host(tmp_path, """
    for (uint32_t G = 1; G <= 256; G++) {
        uint32_t before = 1;
        for (uint64_t n = 0; n < (1u << 22); n = n < 70000 ? n + 97 : n * 5 / 4 + 1) {
            const uint32_t nb = sort_chunks(uint32_t(n), G);
            const uint64_t chunk = chunk_len(uint32_t(n), nb, kChunkAlign);
            // as many chunks as CTAs at most, all of the level in them, and
            // no fewer than a smaller level's (whose rows they reuse)
            if (nb < 1 || nb > G || nb * chunk < n || nb < before) {
                std::printf("n %llu G %u: %u chunks\\n", (unsigned long long)n, G, nb);
                return 1;
            }
            before = nb;
        }
    }""", ["hd_chunks.cuh"])
