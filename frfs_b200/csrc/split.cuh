// Cutting the work of a few long items into parts.
#pragma once
#include <cstdint>

namespace bdgfs {

constexpr int kMaxParts = 16;

// Parts that each of ``total`` items of ``units`` equal units is cut into on
// ``ncta`` CTAs: the number with the smallest (rounds of CTAs) x (units per part
// + what every part repeats, in units: ``once`` uncut, ``again`` for a part), so
// that a few items occupy the SMs and a nearly empty last round costs a part of
// an item's time only.  Cutting needs a slot per part.
__host__ __device__ inline int split_parts(int64_t total, int64_t nslots, int units, int ncta, float once, float again)
{
    int best = 1;
    float cost = 1e30f;
    for (int ns = 1; ns <= (units < kMaxParts ? units : kMaxParts); ++ns) {
        if (ns > 1 && total * ns > nslots) break;
        const float c = float((total * ns + ncta - 1) / ncta) * (float((units + ns - 1) / ns) + (ns > 1 ? again : once));
        if (c < 0.97f * cost) {
            cost = c;
            best = ns;
        }
    }
    return best;
}

}  // namespace bdgfs
