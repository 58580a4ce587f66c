"""Where a walk up a tree ends (obvh_b200/csrc/walk_limit.h), on the CPU: at the
root of a sound tree, with an error in a malformed one."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <vector>
#include "walk_limit.h"
using namespace obvh::pipeline;
static const uint32_t kNone = 0xffffffffu;
// the end of the walk from `leaf`, and the levels it took
static Climb walk(const std::vector<uint32_t>& parents, uint32_t internal, uint32_t leaf, uint32_t* levels) {
    uint32_t p = parents[leaf], steps = 0;
    for (;;) {
        const Climb c = climb(p, steps++, internal);
        if (c != Climb::kLevel) {
            *levels = steps - 1;
            return c;
        }
        p = parents[p];
    }
}
int main() {
    int bad = 0;
    for (uint32_t n : {1u, 2u, 3u, 100u}) {  // a chain: the deepest tree of n leaves
        const uint32_t internal = n - 1;
        std::vector<uint32_t> parents(2 * n - 1, kNone);
        for (uint32_t k = 0; k < internal; ++k) {
            parents[internal + k] = k;
            parents[k + 1 < internal ? k + 1 : internal + n - 1] = k;
        }
        uint32_t levels = 0;
        bad += walk(parents, internal, internal + n - 1, &levels) != Climb::kRoot || levels != internal;
        for (uint32_t k = 0; k < internal; ++k) {  // a node that is its own parent, then its child's child
            std::vector<uint32_t> loop = parents;
            loop[k] = k;
            bad += walk(loop, internal, internal + n - 1, &levels) != Climb::kCycle || levels > n;
            loop[k] = internal - 1;
            bad += walk(loop, internal, internal + n - 1, &levels) != Climb::kCycle || levels > n;
            loop[k] = internal;  // a leaf as a parent
            bad += walk(loop, internal, internal + n - 1, &levels) != Climb::kCycle;
        }
    }
    return bad;
}
"""


def test_walks_end_at_the_root_or_with_an_error(tmp_path):
    src = tmp_path / "walk.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "walk"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "obvh_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0

