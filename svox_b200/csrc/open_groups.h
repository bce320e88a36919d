// How the warps of a block tell each other which group of a sorted log holds a bin's items (see
// render_queue.cuh): the warp whose item is a group's first publishes the group's id in the bin's
// ring of entries, the warps with the group's other items read it there.  Host code too, for the
// test of the rule.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define SVOXB_BOTH __host__ __device__ __forceinline__
#else
#define SVOXB_BOTH inline
#endif

namespace svoxb {

constexpr int kSortedChunks = 4;   // chunks per group of a sorted log
constexpr int kSortedItems = 32 * kSortedChunks;
// A block remembers this many of a bin's last groups.  A warp reads the id of its item's group
// a few instructions after it has taken the item's place, and the block's 24 warps have 24 * 32
// items under way, so as a rule it is among the last 7.  Nothing bounds it, though: a warp may be
// held back while the others fill the bin's next groups, and then finds another group's entry,
// or puts its own in the place of a later one.  So an entry names its group in full.
constexpr int kOpenGroups = 8;

// Entry of the bin's group `number` (0, 1, ...); 0: none yet.
SVOXB_BOTH uint64_t open_group_entry(uint32_t number, int id) {
    return ((uint64_t)(number + 1u) << 32) | (uint32_t)id;
}
SVOXB_BOTH int open_group_place(uint32_t number) { return (int)(number % kOpenGroups); }
SVOXB_BOTH bool open_group_is(uint64_t entry, uint32_t number) {
    return (uint32_t)(entry >> 32) == number + 1u;
}
SVOXB_BOTH int open_group_id(uint64_t entry) { return (int)(uint32_t)entry; }

}  // namespace svoxb
