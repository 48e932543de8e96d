// h3g_few.cuh — a CTA's walk over a tree's levels, for models of at most kFewStates states.
#pragma once

#include "h3g_common.cuh"

namespace h3g {

constexpr int kFewWarps = 16;             // warps of a walking CTA; a lane is a pattern, a warp takes a level's items in turn

// observed state of child d (Topo::kdesc entry) at pattern p: negative if missing or ambiguous, 0 for an internal node
__device__ __forceinline__ int few_state(const Topo& t, int2 d, int p) {
    if (d.y <= -2) return 0;
    return d.y < 0 ? -1 : int(t.states[size_t(d.y) * t.Pp + p]);
}

// The items that one warp of a walk takes: every kFewWarps-th of a level, level after level.
struct FewItem {
    int l, i, end;                            // level, position, the level's end; l == levels: none left
    __device__ __forceinline__ void settle(const int* lv, int levels, int wp) {
        while (i >= end && ++l < levels) { i = end + wp; end = lv[l + 1]; }
    }
    __device__ __forceinline__ void next(const int* lv, int levels, int wp) {
        if (l >= levels) return;
        i += kFewWarps;
        settle(lv, levels, wp);
    }
};

// Runs body(a, b, s0, s1) for every item of every level (lv[0] .. lv[levels]; two descriptors an item), with a barrier after
// each level; states(b, s0, s1) loads the observed states that an item's second descriptor names.  Descriptors are
// loaded two items and states one item ahead, across levels.  `ready` is called once the first are on their way.
template <class States, class Ready, class Body>
__device__ __forceinline__ void few_walk(const int* lv, int levels, const int4* info, int wp, States states, Ready ready, Body body) {
    const int4 none = make_int4(0, -1, 0, -1);
    FewItem at{0, wp, lv[1]};
    at.settle(lv, levels, wp);
    FewItem ahead = at;
    int4 a0 = none, b0 = none, a1 = none, b1 = none;
    int s0 = 0, s1 = 0;
    if (at.l < levels) { a0 = info[2 * at.i]; b0 = info[2 * at.i + 1]; }
    ahead.next(lv, levels, wp);
    if (ahead.l < levels) { a1 = info[2 * ahead.i]; b1 = info[2 * ahead.i + 1]; }
    states(b0, s0, s1);
    ready();
    FewItem far = ahead;
    for (int l = 0; l < levels; ++l) {
        while (at.l == l) {
            int n0, n1;
            int4 a2 = none, b2 = none;
            states(b1, n0, n1);
            far.next(lv, levels, wp);
            if (far.l < levels) { a2 = info[2 * far.i]; b2 = info[2 * far.i + 1]; }
            body(a0, b0, s0, s1);
            at = ahead; ahead = far;
            a0 = a1; b0 = b1; s0 = n0; s1 = n1; a1 = a2; b1 = b2;
        }
        __syncthreads();
    }
}

}  // namespace h3g
