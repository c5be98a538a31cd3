// What scene creation finds out about a caller's BVH, on the host.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <utility>
#include <vector>

#include "../../include/convector_gpu.h"
#include "limits.h"

namespace cvx {

// A pair of nodes that the roots do not reach may hold anything: it is neither
// looked at here nor uploaded, and decides nothing.
struct TreeFacts {
    uint32_t depth = 0;  // roots at depth 1
    std::vector<uint8_t> reached_pairs;
    bool reached(uint32_t pair) const { return reached_pairs[pair] != 0; }
    // Every bound is finite, lo <= hi on each axis and none is -0: the select-form
    // slab test (box_test_sel) gives box_test's bits.
    bool select = false;
    // Besides, every bound is at most kSelectMax in magnitude, every node's bounds
    // are exactly the enclosure of its children's, as the build makes them, and the
    // tree is within the limits of the wide records.
    bool wide = false;
};

// Checks the tree; returns what is wrong with it, or null.
inline const char* check_tree(const cvx_bvh_node* nodes, uint32_t n_nodes, uint32_t n_tris, TreeFacts* out) {
    if (n_nodes < 2 || (n_nodes & 1u)) return "node count must be even and at least 2";
    std::vector<std::pair<uint32_t, uint32_t>> stack{{0u, 1u}, {1u, 1u}};
    out->reached_pairs.assign(n_nodes / 2, 0);
    uint32_t depth = 0;
    size_t visited = 0;
    while (!stack.empty()) {
        auto [i, dep] = stack.back();
        stack.pop_back();
        if (++visited > n_nodes) return "BVH nodes form a cycle";
        depth = dep > depth ? dep : depth;
        out->reached_pairs[i / 2] = 1;
        const cvx_bvh_node& nd = nodes[i];
        if (nd.len == 0) {
            if ((nd.index & 1u) || nd.index + 1 >= n_nodes || nd.index < 2)
                return "internal node child index out of range";
            stack.push_back({nd.index, dep + 1});
            stack.push_back({nd.index + 1, dep + 1});
        } else if ((uint64_t)nd.index + nd.len > n_tris) {
            return "leaf triangle range out of range";
        }
    }
    out->depth = depth;
    bool select = true, bounded = true;
    for (uint32_t i = 0; i < n_nodes && select; i++)
        for (int c = 0; c < 3 && out->reached(i / 2); c++) {
            const float lo = nodes[i].origin[c], hi = nodes[i].far_[c];
            if (!std::isfinite(lo) || !std::isfinite(hi) || !(lo <= hi) || (lo == 0.0f && std::signbit(lo)) ||
                (hi == 0.0f && std::signbit(hi)))
                select = false;
            if (!(std::fabs(lo) <= kSelectMax) || !(std::fabs(hi) <= kSelectMax)) bounded = false;
        }
    bool tight = select && bounded;
    for (uint32_t i = 0; i < n_nodes && tight; i++) {
        if (nodes[i].len != 0 || !out->reached(i / 2)) continue;
        const cvx_bvh_node &c0 = nodes[nodes[i].index], &c1 = nodes[nodes[i].index + 1];
        for (int c = 0; c < 3; c++)
            if (std::min(c0.origin[c], c1.origin[c]) != nodes[i].origin[c] ||
                std::max(c0.far_[c], c1.far_[c]) != nodes[i].far_[c])
                tight = false;
    }
    out->select = select;
    out->wide = tight && depth <= kWideMaxDepth && n_nodes / 2 <= kWideMaxPairs;
    return nullptr;
}

}  // namespace cvx
