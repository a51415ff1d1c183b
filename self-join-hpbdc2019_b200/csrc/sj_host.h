// Host-side rules of the engine that need no device.
#pragma once
#include <algorithm>
#include <cstdint>

// Host threads that write the keys of a delivered batch of cnt pairs over n point
// ids: one per half a million ids and pairs.  With every core in the team a small
// batch waits for whichever core is busy with something else; but the loop passes
// over all n run offsets however few pairs the batch has, so those count too.
inline int sj_expand_team(uint64_t n, uint64_t cnt, int threads)
{
    return (int)std::min<uint64_t>((uint64_t)std::max(threads, 1), 1 + (n + cnt) / (1u << 19));
}
