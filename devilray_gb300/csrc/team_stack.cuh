// team_stack.cuh -- the traversal stack of a team of lanes (team.cuh): the lanes
// carry the same ray, all read the stack, the first one writes it.
//
// No device-only code, so that a host program can run the lanes in any order.
#pragma once

#include "bits.cuh"

namespace dr {

// The next node of the team's ray: the first of the current node's internal
// hits (`hits`, in the ray's octant order; children from `child_base` by `imask`),
// else of the group on top of the stack; the rest of that group goes (back) on
// the stack. Every lane of the warp calls it, `walking` where its team has a ray
// that goes on, with the same values in every lane of a team. True when the ray
// is finished: no node is left or (`full`) the stack holds `limit` entries.
//
// The entries past the shared ones (`over`) are each lane's own copy. The shared
// ones are read by all lanes of a team and written by the first, so the pushes of
// the step before and the pops, and the pops and this step's push, which may
// replace the entry just popped, each have `barrier` between them (all lanes of
// the warp, with memory ordering).
template <int DEPTH, class Entry, class Barrier>
__host__ __device__ __forceinline__ bool team_next_node(bool walking, bool first_lane, uint32_t oct, uint32_t child_base,
                                                        uint32_t imask, uint32_t hits, Entry *stack, Entry *over,
                                                        uint32_t limit, int &sp, uint32_t &node, bool &full,
                                                        Barrier &&barrier)
{
    bool done = false;
    barrier();
    if (walking && hits == 0) {
        if (sp == 0) {
            done = true;
        } else {
            --sp;
            const Entry e = sp < DEPTH ? stack[sp] : over[sp - DEPTH];
            child_base = e.x;
            imask = e.y & 0xffu;
            hits = e.y >> 8;
        }
    }
    barrier();
    if (walking && !done) {
        const uint32_t slot = (uint32_t)lowest_bit(hits) ^ oct;
        const uint32_t rest = hits & (hits - 1u);
        node = child_base + (uint32_t)popcount(imask & ((1u << slot) - 1u));
        if (rest) {
            if ((uint32_t)sp >= limit) {
                done = full = true;
            } else {
                const Entry e{child_base, (rest << 8) | imask};
                if (sp >= DEPTH) over[sp - DEPTH] = e;
                else if (first_lane) stack[sp] = e;
                ++sp;
            }
        }
    }
    return done;
}

}  // namespace dr
