// sph_up.cuh -- the up pass over the GPU-built tree in one launch, shared by
// the two gravity forms (sph_gravity.cu, sph_gravity_theta.cu).
//
// A thread takes a leaf, computes its moments and climbs: at each branch the
// children count themselves in, and the thread that completes the count
// computes the branch and goes on to the branch's parent; the others are done.
// Nothing waits, and a branch sums its children in slot order whoever comes
// last, so the results do not depend on the schedule.  Each tree build sets the
// counts to zero, and a pass leaves them so.
//
// One launch per level left the upper levels to a few warps that each waited
// for memory (N = 1e6, leaf 32: 8 launches, 241 us; N = 2e4: 160 us); the climb
// saves 41 us and 114 us of these.  Host-given trees keep one launch per level: sph_set_tree
// checks them node by node, and a child that no level lists would leave its
// parent's count short for good.
#pragma once

#include "sph_internal.h"

namespace sph {

struct UpNodes {
    const int32_t *T;
    const int32_t *level_nodes;
    const int32_t *level_count;
    const int32_t *parent;  // by data pointer: tree offset, -1 at the root
    int32_t *arrived;       // by data pointer: children done, 0 between passes
    int64_t level_cap;
    int levels;
};

template <class Leaf, class Branch>
__device__ __forceinline__ void up_climb(const UpNodes &u, Leaf &&leaf, Branch &&branch) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = t;
        int l = 0;
        for (; l < u.levels; ++l) {
            const int cnt = u.level_count[l];
            if (r < cnt) break;
            r -= cnt;
        }
        if (l == u.levels) return;
        const int tp = u.level_nodes[(size_t)l * u.level_cap + r];
        if (u.T[tp] == 0) continue;  // a branch: reached from its children
        int dp = u.T[tp + 1];
        leaf(tp, dp);
        for (int p = u.parent[dp]; p >= 0; p = u.parent[dp]) {
            const int pdp = u.T[p + 1];
            int kids = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) kids += u.T[p + 2 + k] != -1;
            __threadfence();  // this node's record before its arrival
            if (atomicAdd(u.arrived + pdp, 1) + 1 != kids) break;
            u.arrived[pdp] = 0;
            __threadfence();  // the other children's records after theirs
            branch(p, pdp);
            dp = pdp;
        }
    }
}

// Launch bound: every node at most once per thread of a full device.
inline int up_blocks(const Tree &tr, int threads) {
    int64_t nodes = 0;
    for (int l = 0; l < tr.n_levels_host; ++l) nodes += tr.level_count_host[l];
    const int64_t b = (nodes + threads - 1) / threads;
    return (int)(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}

inline UpNodes up_nodes(const Tree &tr) {
    return UpNodes{tr.tree, tr.level_nodes, tr.level_count, tr.parent, tr.arrived, tr.level_cap, tr.n_levels_host};
}

}  // namespace sph
