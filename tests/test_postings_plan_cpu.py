"""Limits of the exact search's postings (csrc/postings_plan.h), compiled for
the host: a grid-stride walk of a run that ends near 2^31 visits each posting
once and nothing else, and the positions computed past the largest run have an
int32."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "neural-sparse-cpp_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <vector>
#include "postings_plan.h"
int main() {
    // threads of a grid of the widest step the launch takes: 148 * 32 CTAs of 256
    const int64_t step = 148 * 32 * 256;
    const int32_t end = static_cast<int32_t>(nsp::kMaxPostings);
    for (int64_t n : {int64_t{0}, int64_t{1}, int64_t{300}, step - 1, step, 2 * step + 17}) {
        const int32_t lo = static_cast<int32_t>(end - n);
        std::vector<unsigned char> seen(static_cast<size_t>(n), 0);
        bool bad = false;
        for (int64_t first = 0; first < step; ++first)
            nsp::each_posting(lo, end, first, step, [&](int32_t p) {
                if (p < lo || p >= end) bad = true;
                else ++seen[static_cast<size_t>(p - lo)];
            });
        for (unsigned char s : seen) bad |= s != 1;
        if (bad) return std::printf("run of %lld\n", static_cast<long long>(n)), 1;
    }
    if (nsp::kMaxPostings + nsp::kPostingsAhead > 2147483647ll) return std::printf("ahead\n"), 1;
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_positions_near_the_limit(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
