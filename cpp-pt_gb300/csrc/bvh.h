// Host-side BVH construction.
//
// Two hierarchies are built for every scene:
//
// 1. RefTopology -- the reference's own binary BVH (BVH::build_node /
//    compute_split, src/primitive/bvh.h:57-216), rebuilt with the same bins,
//    cost, tie order and child order.  It is never traversed on the GPU.  It
//    yields, per triangle, (a) its rank = position in the order
//    BVHNode::intersect visits leaves (bvh.h:33-34, member `right` first), and
//    (b) the box of the innermost internal node above its leaf.  Those two
//    values let any traversal reproduce the reference's closest hit exactly:
//      - the reference reports the smallest t among the triangles it tests,
//        the later-visited (higher rank) one on equal t (triangle.h:55,106);
//      - it tests a triangle iff every ancestor box passes its slab test
//        (aabb.h:19-61), and that test is monotone under box inclusion
//        (every float step -- subtraction, division by the same d, min/max --
//        is monotone), so passing the innermost ancestor box implies
//        passing all of them.
//
// 2. WideBVH -- a binned-SAH BVH collapsed to 4 children per node (the
//    collapse of least total node area), with
//    children boxes quantised to 8 bits relative to the node (64 bytes per
//    node), triangles reordered into its leaves as {a, b-a, c-a} + rank +
//    parent-box index + insertion index (48 bytes).  This is what the GPU
//    traverses.
#pragma once
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define CPPPT_HD __host__ __device__
#else
#define CPPPT_HD
#endif

namespace cpppt_gb300 {

struct Box3 {
    float lo[3], hi[3];
};

struct RefTopology {
    std::vector<int32_t> rank;          // per triangle (insertion index -> DFS rank)
    std::vector<int32_t> leaf_order;    // DFS order of insertion indices
    std::vector<Box3> node_box;         // internal nodes, pre-order
    std::vector<int32_t> node_parent;   // per internal node
    std::vector<int32_t> prim_parent;   // per triangle: internal node holding its leaf (-1: root is a leaf)
};

// Builds the reference topology from per-triangle vertex positions.
// tri_v: 9 floats per triangle (a, b, c).
// n_threads: 0 = all hardware threads, 1 = sequential; the result does not
// depend on it (independent subtrees are built in parallel and joined in
// the reference's pre-order).
RefTopology build_ref_topology(const float* tri_v, int n_tris, int n_threads = 0);

// Compressed 4-wide node, 64 bytes (4 x uint4 on the device):
//   w[0..2] origin p (float bits); w[3] = ex | ey<<8 | ez<<16  (biased float exponents of the
//   per-axis scale s = 2^(e-127)); w[4..7] lo_x[4] lo_y[4] lo_z[4] hi_x[4] (bytes, child c at
//   byte c); w[8..9] hi_y[4] hi_z[4]; w[10..13] child refs; w[14..15] unused.
// A child box is [p + lo*s, p + hi*s].  Empty slots have lo = 255, hi = 0.
// Child ref: bit 31 clear -> internal node index; bit 31 set -> leaf with
// (ref >> 27 & 15) + 1 triangles starting at (ref & 0x7ffffff).
struct WideNode {
    uint32_t w[16];
};

struct WideBVH {
    std::vector<WideNode> nodes;      // breadth-first order, root at 0
    std::vector<int32_t> tri_order;   // leaf order -> insertion index
    int max_depth = 0;                // in wide nodes
    int max_leaf = 0;
    float inflate = 0.0f;             // absolute box inflation used
};

// tri_v as above.  max_leaf <= 16.
WideBVH build_wide_bvh(const float* tri_v, int n_tris, int max_leaf = 4, int n_threads = 0);

// The collapse of a binary tree into 4-wide nodes that visits least: a ray
// visits a node with a probability about its box's area, and which leaves it
// tests does not depend on the grouping, so the sum of the wide nodes' areas
// is minimised, bottom-up.  cost[j - 1] of a subtree is the least sum with
// which it can stand as at most j children of one wide node: a leaf costs
// nothing, an inner node either becomes one child (its area and the best
// split of 4 slots between its two sides) or is dissolved, its slots split
// between its sides.  (The dynamic program of Ylitie, Karras and Laine 2017,
// "Efficient incoherent ray traversal on GPUs through compressed wide BVHs",
// for leaves that stay as they are.)  Against opening the child of largest area first: 1M
// triangle soup 21 % fewer nodes and 4 % less area, closest hit of 1.8M rays
// 851 -> 754 us, any hit 601 -> 578; 192k-triangle room any hit 138 -> 124.
//
// l, r: costs of the sides; returns the choices for collapse_children.
CPPPT_HD inline uint32_t collapse_cost(float area, const float l[3], const float r[3], float cost[3]) {
    const float d2 = l[0] + r[0];
    const float d3l = l[0] + r[1], d3r = l[1] + r[0];
    const float d4a = l[0] + r[2], d4b = l[1] + r[1], d4c = l[2] + r[0];
    float d4 = d4a;
    uint32_t four = 1;  // slots of the left side
    if (d4b < d4) { d4 = d4b; four = 2; }
    if (d4c < d4) { d4 = d4c; four = 3; }
    cost[0] = area + d4;
    const uint32_t two = d2 < cost[0] ? 1 : 0;  // 0: one child
    cost[1] = two ? d2 : cost[0];
    const float d3 = d3r < d3l ? d3r : d3l;
    const uint32_t three = d3 < cost[1] ? (d3r < d3l ? 2 : 1) : 0;  // 0: as with two slots
    cost[2] = three ? d3 : cost[1];
    return four | three << 2 | two << 4;
}

// Children of the wide node at inner node `root`: at most 4 nodes to ch, left
// to right.  left(i) < 0: leaf; choice(i): collapse_cost's result.
template <class Left, class Right, class Choice>
CPPPT_HD inline int collapse_children(int32_t root, Left left, Right right, Choice choice, int32_t ch[4]) {
    int32_t node[4];  // pending subtrees, and their slots
    uint32_t slots[4];
    int top = 0, nc = 0;
    const uint32_t four = choice(root) & 3;
    node[top] = right(root); slots[top++] = 4 - four;
    node[top] = left(root); slots[top++] = four;
    while (top > 0) {
        const int32_t i = node[--top];
        uint32_t j = slots[top];
        if (left(i) >= 0) {
            const uint32_t c = choice(i), three = c >> 2 & 3, two = c >> 4 & 1;
            if (j == 3 && three == 0) j = 2;
            if (j == 2 && two == 0) j = 1;
            if (j > 1) {
                const uint32_t k = j == 3 ? three : 1;
                node[top] = right(i); slots[top++] = j - k;
                node[top] = left(i); slots[top++] = k;
                continue;
            }
        }
        ch[nc++] = i;
    }
    return nc;
}

// Children of the wide node at inner node `root` when the child of largest
// area is opened first.
template <class Left, class Right, class Area>
CPPPT_HD inline int collapse_largest(int32_t root, Left left, Right right, Area area, int32_t ch[4]) {
    int nc = 2;
    ch[0] = left(root);
    ch[1] = right(root);
    while (nc < 4) {
        int pick = -1;
        float best = -1.0f;
        for (int i = 0; i < nc; i++)
            if (left(ch[i]) >= 0 && area(ch[i]) > best) {
                best = area(ch[i]);
                pick = i;
            }
        if (pick < 0) break;
        const int32_t c = ch[pick];
        ch[pick] = left(c);
        ch[nc++] = right(c);
    }
    return nc;
}

// The deepest tree whose walk the traversal's stack (64 entries) holds.  A
// scene is accepted if the largest-first collapse is no deeper; where the
// cheapest one is, the largest-first one is the tree (a scale-3 chain of 19
// clusters of 4000 triangles: 21 and 19).  Both depths are known before the
// nodes are written.
constexpr int kMaxWideDepth = 20;
// Record of a node: collapse_cost's choices, and above them the depth of the
// largest-first collapse from it.
constexpr int kDepthShift = 8;

constexpr uint32_t kLeafBit = 0x80000000u;
inline uint32_t make_leaf_ref(uint32_t start, uint32_t count) {
    return kLeafBit | ((count - 1u) << 27) | start;
}

}  // namespace cpppt_gb300
