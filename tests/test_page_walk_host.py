"""The walk over the pages of a host range (which decides whether a recorded copy may be a kernel), compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "page_walk.h"
#include <set>
#include <stdio.h>
int main() {
    using fnn::every_page;
    const size_t P = 4096;
    // pinned pages 10, 11, 13 (a hole between two registrations), 20
    const std::set<uintptr_t> pinned = {10, 11, 13, 20};
    auto ok = [&](uintptr_t p) { return pinned.count(p / P) == 1; };
    struct { uintptr_t first; size_t bytes; bool want; } cases[] = {
        {10 * P, P, true},          {10 * P, 2 * P, true},          {10 * P + 5, 2 * P - 5, true},
        {10 * P + 5, 2 * P - 4, false}, {11 * P + 100, 2 * P + 1, false},   // both ends pinned, the hole between
        {10 * P, 4 * P, false},     {9 * P + 4095, 2, false},       {13 * P + 4095, 1, true},
        {13 * P + 4095, 2, false},  {20 * P + 1, 1, true},          {20 * P, P + 1, false},
    };
    for (auto &c : cases)
        if (every_page(c.first, c.bytes, P, ok) != c.want) {
            printf("range %zu + %zu\n", (size_t)c.first, c.bytes);
            return 1;
        }
    // one address of the range per page, the first of all included
    std::set<uintptr_t> seen;
    every_page(3 * P + 7, 2 * P, P, [&](uintptr_t p) { seen.insert(p); return true; });
    return seen == std::set<uintptr_t>({3 * P + 7, 4 * P, 5 * P}) ? 0 : 1;
}
"""


def test_every_page_of_a_range_is_asked(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(PROGRAM)
    subprocess.run([os.environ.get("FNN_HOST_CXX", "/usr/bin/g++"), "-std=c++17", "-I",
                    os.path.join(ROOT, "fastnn_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
