// nd_order.cpp -- nested dissection of a grid's unknowns (host).
//
// The Poisson operator of poissonSolver.pyx:41-58 couples a node with its
// four neighbours only, so a grid line of nodes separates what lies on its two
// sides.  The unknowns are split recursively: the line nearest the middle of
// the longer side of the set's bounding box becomes the separator, the nodes
// on its two sides the children.  Node h of the binary tree has the children
// 2h and 2h + 1; an unknown gets the number of the tree node that it belongs
// to (a separator, or a set that is not split any further).
#include <stdint.h>

#include <algorithm>
#include <new>
#include <vector>

#include "oec.h"

namespace {

struct Piece {
    int64_t first, last;  // range of the index array
    int64_t node;
    int depth;
};

}  // namespace

static void dissect(int64_t n, const int32_t *ix, const int32_t *iy, int32_t max_depth, int32_t leaf,
                    int64_t *node_out) {
    std::vector<int32_t> idx((size_t)n), count;
    for (int64_t i = 0; i < n; ++i) idx[(size_t)i] = (int32_t)i;
    std::vector<Piece> todo;
    todo.push_back({0, n, 1, 0});
    while (!todo.empty()) {
        const Piece p = todo.back();
        todo.pop_back();
        int32_t *a = idx.data() + p.first, *b = idx.data() + p.last;
        const int64_t m = p.last - p.first;
        int32_t x0 = ix[*a], x1 = x0, y0 = iy[*a], y1 = y0;
        for (int32_t *k = a; k < b; ++k) {
            x0 = std::min(x0, ix[*k]);
            x1 = std::max(x1, ix[*k]);
            y0 = std::min(y0, iy[*k]);
            y1 = std::max(y1, iy[*k]);
        }
        const int64_t lx = (int64_t)x1 - x0, ly = (int64_t)y1 - y0;
        const bool along_x = lx >= ly;
        const int32_t *c = along_x ? ix : iy;
        const int64_t lo = along_x ? x0 : y0, len = (along_x ? lx : ly) + 1;
        if (p.depth >= max_depth || m <= leaf || len < 3) {
            for (int32_t *k = a; k < b; ++k) node_out[*k] = p.node;
            continue;
        }
        // the line that keeps the larger side smallest, the shorter of two equal ones
        count.assign((size_t)len, 0);
        for (int32_t *k = a; k < b; ++k) ++count[(size_t)(c[*k] - lo)];
        int64_t below = 0, best = -1, best_cost = 0;
        for (int64_t l = 0; l < len; ++l) {
            const int64_t here = count[(size_t)l], above = m - below - here;
            const int64_t cost = 4 * std::max(below, above) + here;
            if (best < 0 || cost < best_cost) {
                best = l;
                best_cost = cost;
            }
            below += here;
        }
        const int32_t cut = (int32_t)(lo + best);
        int32_t *u = std::partition(a, b, [&](int32_t i) { return c[i] < cut; });
        int32_t *v = std::partition(u, b, [&](int32_t i) { return c[i] == cut; });
        for (int32_t *k = u; k < v; ++k) node_out[*k] = p.node;
        if (u > a) todo.push_back({p.first, p.first + (u - a), 2 * p.node, p.depth + 1});
        if (b > v) todo.push_back({p.first + (v - a), p.last, 2 * p.node + 1, p.depth + 1});
    }
}

extern "C" int oec_nd_dissect(int64_t n, const int32_t *ix, const int32_t *iy, int32_t max_depth, int32_t leaf,
                              int64_t *node_out) {
    if (n <= 0 || n > INT32_MAX || !ix || !iy || !node_out || max_depth < 0 || max_depth > 40 || leaf < 1)
        return OEC_ERR_INVALID;
    try {
        dissect(n, ix, iy, max_depth, leaf, node_out);
    } catch (const std::bad_alloc &) {
        return OEC_ERR_HOST;
    }
    return OEC_OK;
}
