"""The growth of a build's scratch (csrc/arena_plan.h), compiled for the host:
chunks double from 64 MB to 1 GB and hold what is asked for; where the device
has no room for a chunk, the request alone is tried."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "neural-sparse-cpp_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include "arena_plan.h"
static int fail(const char* what) { return std::printf("%s\n", what), 1; }
int main() {
    const size_t MB = size_t{1} << 20;
    size_t last = 0;
    for (size_t want : {64, 128, 256, 512, 1024, 1024}) {
        last = nsp::arena_chunk(last, MB);
        if (last != want * MB) return fail("growth");
    }
    if (nsp::arena_chunk(64 * MB, 5000 * MB) != 5000 * MB) return fail("large request");
    if (nsp::arena_chunk(5000 * MB, MB) != 1024 * MB) return fail("after a large one");
    char memory;
    size_t room = 0;
    int calls = 0;
    auto allocate = [&](size_t n) -> void* { ++calls; return n <= room ? &memory : nullptr; };
    for (size_t r : {3000 * MB, 100 * MB, 10 * MB, 9 * MB}) {
        room = r;
        calls = 0;
        size_t cap = nsp::arena_chunk(256 * MB, 10 * MB);
        void* p = nsp::arena_allocate(cap, 10 * MB, allocate);
        if ((p != nullptr) != (r >= 10 * MB)) return fail("refused what fits");
        if (p != nullptr && cap != (r >= 512 * MB ? 512 : 10) * MB) return fail("size");
        if (calls > 2) return fail("calls");
    }
    size_t cap = 10 * MB;  // nothing to leave out
    room = calls = 0;
    if (nsp::arena_allocate(cap, 10 * MB, allocate) != nullptr || calls != 1) return fail("exact");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_chunks(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
