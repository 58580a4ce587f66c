// walk_limit.h - what a walk from a leaf towards the root does next: one rule
// for a level, the end at the root and a malformed tree.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define OBVH_HOST_DEVICE __host__ __device__
#else
#define OBVH_HOST_DEVICE
#endif

namespace obvh {
namespace pipeline {

enum class Climb : uint32_t {
    kLevel,  // p is an internal node to arrive at
    kRoot,   // the walk has passed the root
    kCycle,  // p is no internal node, or the walk took more levels than the tree has
};

// p: the parent to go to, 0xffffffff above the root; steps: the levels the walk
// has taken; internal: the internal nodes, more than any path is long.
OBVH_HOST_DEVICE constexpr Climb climb(uint32_t p, uint32_t steps, uint32_t internal) {
    return p == 0xffffffffu ? Climb::kRoot : (steps > internal || p >= internal ? Climb::kCycle : Climb::kLevel);
}

}  // namespace pipeline
}  // namespace obvh
