// unit_plan.h - how the extents of the larger nodes of any tree are split into
// warp units, and how the running counts of nodes and units share one 64-bit
// word (obb_tree.cu, plan_node).  Host arithmetic only.
#pragma once

#include <cstdint>

namespace obvh {
namespace obbtree {

// Leaves per warp unit, as far as the counts fit (us, 128 / 256 / 512 / 1,024 /
// 2,048: transform of 229,824 triangles 260 / 258 / 260 / 267 / 282, ATRBVH of
// 917,504 2,300 / 2,278 / 2,270 / 2,280 / 2,299; four 1,024s in a row for a
// warp 281 and 2,311).
constexpr uint32_t kUnitShift = 9;

struct UnitPlan {
    uint32_t unit_shift;  // 2^unit_shift leaves per unit
    uint32_t unit_bits;   // the low bits of the word count units, the rest nodes
};

// For a tree of n leaves.  It has fewer than n nodes to list, and the leaf
// counts of its internal nodes add up to less than n (n + 1) / 2 (a tree as
// deep as it has nodes), so it has at most that many 2^unit_shift-ths of units
// and one more per node.  Units of 512 leaves up to 2^24 leaves; beyond, they
// grow with the sum.  (With 32 bits for each count a chain of 2,100,000 leaves
// had more units than its field held: they ran over into the nodes' count.)
constexpr UnitPlan unit_plan(uint32_t n) {
    UnitPlan p{kUnitShift, 64};
    for (uint32_t k = n; k != 0; k >>= 1) --p.unit_bits;
    const uint64_t leaves = static_cast<uint64_t>(n) * (static_cast<uint64_t>(n) + 1) / 2;
    while ((leaves >> p.unit_shift) + n >= (1ull << p.unit_bits)) ++p.unit_shift;
    return p;
}

static_assert(unit_plan(1u << 24).unit_shift == kUnitShift, "512 leaves per unit up to 2^24 leaves");
static_assert(unit_plan(0x7fffffffu).unit_shift < 31, "units within a 32-bit leaf range");

}  // namespace obbtree
}  // namespace obvh
