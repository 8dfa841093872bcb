// Cutting the work of a few long items into parts.
//
// An item is ``nb`` equal blocks of work (radii) whose results are rounded and then
// added in order, by its one CTA or, if cut, from a slot per block by the part that
// ends last: an item's result has the same bits whole or cut, wherever it stands
// in a list and however many CTAs run.
#pragma once
#include <cstdint>

namespace bdgfs {

// Items [0, whole) are done whole, the others in ``ns`` parts each.
struct SplitPlan {
    int64_t whole;
    int ns;
};

// Plan for ``total`` items of ``nb`` blocks on ``ncta`` CTAs: full rounds of CTAs are
// left whole; the items of the last, partly filled round (or of a list shorter
// than the CTAs) are cut into the number of parts with the smallest (rounds of
// CTAs) x (blocks per part + what every part repeats, in blocks: ``once`` uncut,
// ``again`` for a part).  A cut item needs ``nb`` of ``nslots`` slots.
__host__ __device__ inline SplitPlan split_plan(int64_t total, int64_t nslots, int nb, int ncta, float once, float again)
{
    const int64_t tail = total % ncta;
    int best = 1;
    float cost = 1e30f;
    for (int ns = 1; tail > 0 && ns <= nb; ++ns) {
        if (ns > 1 && tail * nb > nslots) break;
        const float c = float((tail * ns + ncta - 1) / ncta) * (float((nb + ns - 1) / ns) + (ns > 1 ? again : once));
        if (c < 0.97f * cost) {
            cost = c;
            best = ns;
        }
    }
    return SplitPlan{best > 1 ? total - tail : total, best};
}

// What a launch passes to its kernel: the plan where the host knows the list's length,
// else (ns = 0) what the kernel plans with once it has read the counts.
struct SplitArgs {
    SplitPlan plan;
    int64_t nslots;                 // slots of cut items' blocks, after one per CTA
    int32_t nctas;                  // CTAs that a full round has
    float once, again;
};

__device__ __forceinline__ SplitPlan split_plan(const SplitArgs& s, int64_t total, int nb)
{
    return s.plan.ns > 0 ? s.plan : split_plan(total, s.nslots, nb, s.nctas, s.once, s.again);
}

// Work item -> position in the list, its blocks [b0, b1) of nb, parts of it, and
// its place among the cut items
struct SplitItem {
    int64_t li, cut;
    int b0, b1, ns;
};

__device__ __forceinline__ SplitItem split_item(int64_t item, const SplitPlan& p, int nb)
{
    if (item < p.whole) return SplitItem{item, 0, 0, nb, 1};
    const int64_t k = item - p.whole, cut = k / p.ns;
    const int part = int(k - cut * p.ns);
    return SplitItem{p.whole + cut, cut, nb * part / p.ns, nb * (part + 1) / p.ns, p.ns};
}

__host__ __device__ inline int64_t split_items(int64_t total, const SplitPlan& p)
{
    return p.whole + (total - p.whole) * p.ns;
}

}  // namespace bdgfs
