// Host-side acceleration-structure builder: binned SAH binary BVH collapsed
// into the 8-wide quantised layout of ar_types.h.
//
// Replaces BLASAccel::build / TLAS::build (src/accel/bvh.rs:326-411).  The
// reference builds a binary full-sweep SAH tree for a scalar CPU traversal;
// here the tree is re-shaped for the GPU (8 children per 80-byte node, leaves
// of at most 3 primitives, octant-ordered slots).  Closest-hit results do not
// depend on tree shape except for exact ties in t.
#pragma once
#include <cstdint>
#include <vector>
#include "ar_types.h"

namespace ar {

struct PrimBox {
    float mn[3], mx[3];
};

struct BuildOptions {
    uint32_t max_leaf = 3;  // 1..4
    uint32_t bins = 32;
    uint32_t threads = 0;   // 0: all hardware threads
    uint32_t width = 8;     // children per wide node, 2..8
    float node_cost = 0.5f; // SAH: a node visit relative to one triangle test
};

struct WideBuild {
    std::vector<WideNode> nodes;      // nodes[0] is the root; child_base/tri_base are build-local
    std::vector<uint32_t> prim_order; // leaf-order primitive ids (tri_base indexes this)
    uint32_t depth = 0;               // number of wide levels
};

// The scene's geometry buffer: nodes, then triangles, then instances, each
// section starting at a multiple of its record size from the buffer's start, so
// that a 32-bit link counts records from there: links reach 206 GB of triangles and
// 275 GB of instances, more than a GPU holds (counting 16-byte words in their
// place, they reached 64 GiB; 16M rays on the 1M-triangle soup 17.59 -> 17.77 ms).
struct GeomLayout {
    uint32_t first_tri, first_inst;  // in their records, from the start
    uint64_t bytes;
    bool fits;  // every link is below 2^32
};
inline GeomLayout geom_layout(uint64_t nodes, uint64_t tris, uint64_t instances) {
    const auto records = [](uint64_t end, uint64_t record) { return (end + record - 1) / record; };
    const uint64_t t = records(nodes * sizeof(WideNode), sizeof(TriRecord));
    const uint64_t i = records((t + tris) * sizeof(TriRecord), sizeof(InstanceRecord));
    const uint64_t most = UINT32_MAX;
    return {uint32_t(t), uint32_t(i), (i + instances) * sizeof(InstanceRecord),
            nodes <= most && t + tris <= most && i + instances <= most};
}

// Builds the wide BVH over `boxes`.  An empty input yields an empty build.
WideBuild build_wide_bvh(const std::vector<PrimBox>& boxes, const BuildOptions& opts);

}  // namespace ar
