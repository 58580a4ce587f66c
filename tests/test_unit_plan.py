"""The packed counts of the OBB extents' plan (obvh_b200/csrc/unit_plan.h), on the
CPU: the additions that plan_node makes, for the trees with the most units."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include "unit_plan.h"
using namespace obvh::obbtree;
// a chain of n leaves: internal nodes of 2, 3, ..., n leaves, those of more than 32 listed
static int chain(uint32_t n) {
    const UnitPlan p = unit_plan(n);
    unsigned long long packed = 0;
    unsigned __int128 units = 0;
    for (uint32_t cnt = 33; cnt <= n; ++cnt) {
        const uint32_t own = ((cnt - 1) >> p.unit_shift) + 1;
        packed += (1ull << p.unit_bits) + own;
        units += own;
    }
    const unsigned long long nodes = n > 32 ? n - 32 : 0;
    const bool ok = (packed >> p.unit_bits) == nodes && (packed & ((1ull << p.unit_bits) - 1)) == units;
    if (!ok) std::printf("%u leaves: %llu nodes listed, %llu counted\n", n, nodes, packed >> p.unit_bits);
    return !ok;
}
int main() {
    int bad = 0;
    const uint32_t sizes[] = {1u, 33u, 1000u, 1u << 20, (1u << 21) + 1, 2200000u, 2965820u, 3000000u,
                              (1u << 24) - 1, 1u << 24, (1u << 24) + 1, 1u << 25, (1u << 26) + 7, 1u << 28};
    for (uint32_t n : sizes) bad += chain(n);
    for (uint32_t n = 1; n < (1u << 24); n = 2 * n + 1) bad += unit_plan(n).unit_shift != 9;
    return bad;
}
"""


def test_counts_of_nodes_and_units_never_meet(tmp_path):
    src = tmp_path / "plan.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "plan"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "obvh_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
