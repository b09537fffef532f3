"""Which terms of an exact index get dense rows (csrc/postings_plan.h), compiled
for the host: the frequent ones, most frequent first, none of few postings, and
no more than a quarter of the free memory holds; none where the allocation
fails."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "neural-sparse-cpp_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <new>
#include <stdexcept>
#include "postings_plan.h"
using nsp::dense_terms;
static int fail(const char* what) { return std::printf("%s\n", what), 1; }
int main() {
    auto starts = [](const std::vector<int32_t>& counts) {
        std::vector<int32_t> s{0};
        for (int32_t c : counts) s.push_back(s.back() + c);
        return s;
    };
    const std::vector<int32_t> want{3, 0, 2, 5};
    // 2,000 docs: from 600 postings on
    const auto s = starts({900, 599, 700, 2000, 0, 600});
    if (dense_terms(s, 2000, 1000, 1u << 30) != want) return fail("by count");
    // room for three rows in a quarter, for none
    if (dense_terms(s, 2000, 1000, 12000) != std::vector<int32_t>{3, 0, 2}) return fail("three");
    if (!dense_terms(s, 2000, 1000, 3999).empty()) return fail("no room");
    // few docs: every term is in a large share of them
    if (!dense_terms(starts({3, 3, 2}), 3, 1000, 1u << 30).empty()) return fail("few postings");
    if (dense_terms(starts({511, 512}), 512, 1000, 1u << 30) != std::vector<int32_t>{1})
        return fail("least count");
    // at most 256 rows, the lowest terms of equal counts
    const auto many = dense_terms(starts(std::vector<int32_t>(300, 5000)), 5000, 1, 1u << 30);
    if (many.size() != 256 || many.back() != 255) return fail("most rows");
    // an allocation that fails
    if (nsp::allocate_dense_rows(7, [](size_t) { throw std::runtime_error("memory"); }) != 0)
        return fail("failed allocation");
    if (nsp::allocate_dense_rows(7, [](size_t) { throw std::bad_alloc(); }) != 0)
        return fail("failed allocation");
    size_t got = 0;
    if (nsp::allocate_dense_rows(7, [&](size_t n) { got = n; }) != 7 || got != 7)
        return fail("allocation");
    if (nsp::allocate_dense_rows(0, [](size_t) { throw std::bad_alloc(); }) != 0) return fail("0");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_dense_terms(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
