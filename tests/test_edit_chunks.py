"""The persistent edit kernel's split of a level over its CTAs
(csrc/hd_chunks.cuh), for every grid size a device or a slice of one may have:
CTA k works chunk k and has a row of digit counts, so a level has no more
chunks than the grid has CTAs and its chunks cover it.  Compiled and run on
the host."""
import os
import re
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
                   "#include <cstdio>\n#include <initializer_list>\nusing namespace hd;\nint main() {\n" + body + "\nreturn 0; }\n")
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


def test_barrier_word(tmp_path):
    """Arrivals past 2^32 stay clear of the abort flag, and the flag of them."""
    run_host(tmp_path, """
    for (uint64_t k : {1ull, 5ull, 28256363ull, 28256364ull, 0xFFFFFFFEull})
        for (uint32_t G : {1u, 32u, 152u, 1024u}) {
            const unsigned long long t = barrier_target(uint32_t(k), G);
            if (t != k * G || barrier_arrivals(t) != t || barrier_aborted(t) || barrier_arrivals(t - 1) >= t ||
                !barrier_aborted(t | kBarrierAbort) || barrier_arrivals(t | kBarrierAbort) != t)
                return 1;
        }""", ["hd_chunks.cuh"])


def test_barrier_word_is_accessed_whole():
    """Acquire and release pair up between accesses of one size only: every
    access to the barrier's word is a 64-bit one."""
    src = open(os.path.join(CSRC, "hd_edit_persist.cu")).read()
    assert re.search(r"unsigned long long arrived;", src)
    uses = re.findall(r"[\w(]*\(&?\w*->arrived\b[^)]*\)", src)
    assert len(uses) >= 4
    for u in uses:
        assert re.match(r".*(atomicAdd\(&ctl->arrived, 1ull\)|atomicOr\(&ctl->arrived, kBarrierAbort\)|"
                        r"ld_acquire64\(&ctl->arrived\))$", u), u
