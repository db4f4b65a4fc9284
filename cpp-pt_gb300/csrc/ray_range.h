// How a batch's rays are shared among the warps of a traversal kernel.
#pragma once
#include <cstdint>

#include "bvh.h"

namespace cpppt_gb300 {

// Rays per fetch when `left` rays remain for `nwarps` warps (`share` chunks
// each): kChunk while there are many, down to one for the last ones, so that
// a small batch (or the end of a large one) is spread over all warps.  A warp
// whose rays take different ways through the tree runs the union of their
// steps, and the launch ends with its slowest warp.  Measured (1M-triangle
// soup) against 16 rays a fetch from one CTA per 1024 rays: 1000 shadow rays
// 136 -> 54 us, 30,001 closest-hit rays 194 -> 125 us; the first fetch at half
// the even share 144 us (30,001 rays), at a quarter 171 us, since half the rays
// then wait for a second fetch.  kChunk 8, 16, 24, 32, 48, 64: 1080p at 16 spp
// 92.0, 87.7, 87.2, 86.8, 86.6, 86.5 ms, 1M rays in the 192k-triangle room 336,
// 291, 289, 283, 294, 319 us.
constexpr int kChunk = 32;
CPPPT_HD inline int ray_chunk(int left, int nwarps, int share) {
    const int c = left / (share * nwarps);
    return c < 1 ? 1 : (c > kChunk ? kChunk : c);
}

// Consecutive rays [next, end).  Unsigned: a lane looks up to 32 rays past its
// range and the counter goes up to kChunk a warp past the batch, which for the
// largest batches is past an int.
struct RayRange {
    uint32_t next, end;
};

CPPPT_HD inline uint32_t least(uint32_t a, uint32_t b) { return a < b ? a : b; }

// The range of a fetch of `chunk` rays that found `taken` in the counter, whose
// rays follow the `own` first ones (dealt out without it).
CPPPT_HD inline RayRange fetched_range(int taken, int own, int chunk, int n) {
    const uint32_t next = least((uint32_t)taken + (uint32_t)own, (uint32_t)n);
    return RayRange{next, least(next + (uint32_t)chunk, (uint32_t)n)};
}

// The ray of the r-th lane that wants one, from the range at hand and then
// from the one fetched; false for none.
CPPPT_HD inline bool ray_of(uint32_t r, RayRange at_hand, RayRange fetched, uint32_t& ray) {
    const uint32_t avail = at_hand.end - at_hand.next;
    ray = r < avail ? at_hand.next + r : fetched.next + (r - avail);
    return r < avail || ray < fetched.end;
}

// What is left of the two ranges after `want` lanes took theirs.
CPPPT_HD inline RayRange left_of(uint32_t want, RayRange at_hand, RayRange fetched) {
    const uint32_t avail = at_hand.end - at_hand.next;
    if (want <= avail) return RayRange{at_hand.next + want, at_hand.end};
    return RayRange{least(fetched.next + (want - avail), fetched.end), fetched.end};
}

}  // namespace cpppt_gb300
