// Four-wide tree over a payload's binary BVH, built on the host at scene
// upload (wide_bvh.cpp) and walked by trace_any4 and trace_closest4
// (traverse.cuh).
//
// A wide node stands for a binary inner node P and holds up to four entries:
// for each child C of P, C's two children when C is an inner node whose box
// contains theirs (C is "expanded"), else C itself.  Entries are kept in
// the binary tree's order (left child's side first), so a traversal that
// orders them by the ray's sign on P's and C's split axes visits leaves in
// exactly the order of the binary traversal (noor/cuda/bvh.cuh:193-234).
// Skipping C's own slab test changes no outcome: for a ray whose direction
// components lie within 1e-18 .. 1e18 and whose origin within 1e12
// (wide_degenerate in traverse.cuh), the slab test's per-axis intervals are
// monotone in the box bounds, so a box inside C can only pass where C passes;
// other rays walk the binary tree below that point, node by node.
//
// Entries whose slab test the binary traversal runs against a ray that may
// differ from the one at P's visit (an entry without instance bits under a
// top-level node, where an earlier sibling may have left an object-space
// ray; anything under an inner node whose subtree holds instance or light
// nodes) are deferred: pushed untested, in order, and tested when taken,
// against the ray of that moment, as the binary traversal does.
//
// On the device (pack_wide_tree) a wide node's test only filters: it is one
// fused multiply-add per plane, widened by a bound on its rounding.  What it
// lets through too much is caught by the exact slab test of the binary node:
// a ref is tested exactly when it is taken, with the distance of that moment,
// and a triangle leaf when one of its triangles is hit, with the distance of
// the moment the leaf was taken.  An inner entry passed in error only leads
// to boxes inside it, which miss whenever it misses (an inner node whose
// children stick out of its box is kept as a ref and so tested exactly), and
// closest hit's shrinking distance is covered the same way.
// Trees with deferred entries keep the binary closest hit.
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

namespace nb {

// stack and child-slot words
constexpr uint32_t kWRef = 0x80000000u;       // a binary node (else the index of a wide node)
constexpr uint32_t kWUntested = 0x40000000u;  // with kWRef: its box is tested when it is taken
constexpr uint32_t kWIndex = 0x1FFFFFFFu;
constexpr uint32_t kWNone = 0xFFFFFFFFu;
// device words only: a triangle leaf, kWRef | kWLeaf without kWUntested,
// count - 1 in bits 26-28, first triangle below; an instance whose transform
// is the identity and whose box holds its tree's, kWInstance | transform
constexpr uint32_t kWLeaf = 0x20000000u;
constexpr uint32_t kWLeafShift = 26;
constexpr uint32_t kWLeafMaxCount = 8;
constexpr uint32_t kWLeafStart = (1u << kWLeafShift) - 1u;
constexpr uint32_t kWInstance = kWRef | kWUntested;
// Whether kWRef words can name the nodes of a tree: what build_wide_tree asks of
// it, and what the walks of the binary tree by such words (trace_closest4 and
// trace_any4, `binary`) do, whose words of larger indices would read as leaves
// and instances
constexpr bool ref_words_fit(size_t num_nodes) { return num_nodes < kWIndex; }
// deepest stack a tree may need to be used (words per thread)
constexpr int kWideMaxStack = 96;
// meta[0] bits; the split axes of P, the left and the right child at bits
// 4, 6 and 8
constexpr uint32_t kW4World = 1u;    // P resets the ray to world space (a top-level node)
constexpr uint32_t kW4ExpandL = 2u;  // slots 0, 1 hold the left child's children
constexpr uint32_t kW4ExpandR = 4u;  // slots 2, 3 hold the right child's children

// 128 bytes: the four entry boxes as structure of arrays, the entry words,
// and meta = {flags and axes, 0, 0, 0}
struct WideNodeHost {
    float lo[3][4];
    float hi[3][4];
    uint32_t child[4];
    uint32_t meta[4];
};
static_assert(sizeof(WideNodeHost) == 128, "wide node layout");

struct WideTree {
    std::vector<WideNodeHost> nodes;
    std::vector<uint32_t> map;  // binary inner node -> its wide node (kWNone where there is none)
    std::vector<uint32_t> node; // wide node -> its binary inner node
    uint32_t root = 0;          // the binary root the tree was built from
    int stack_need = 0;         // the deepest stack trace_any4 / trace_closest4 can reach
    int binary_need = 0;        // ... and the binary traversal
    bool closest = false;       // trace_closest4 may use the tree
};

// Collapse the binary tree (8 words per node: min.xyz, w0, max.xyz, w1, as
// the payload's two uint4 arrays interleaved) reachable from `root`.
// Returns false, with the reason in *why, when the tree has a cycle, a NaN
// box bound, more nodes than the stack words can address or a deeper stack
// than `max_stack`; trace_any4 is then not used for the scene.
bool build_wide_tree(const uint32_t* nodes8, size_t nn, uint32_t root, int max_stack, WideTree& out,
                     std::string* why);

// The tree as the device walks it.  A node keeps the layout above with its
// own words: child may be a kWLeaf or kWInstance word; the box of an empty
// slot is inside out and that of a deferred entry unbounded (its words need
// no kWUntested: every ref is tested when it is taken); meta[0] holds
// kW4World and meta[1] three bits per ray octant o (bit a: direction
// component a <= 0) at 3 * o: bit 0 swaps slots 0 and 1, bit 1 slots 2 and 3,
// bit 2 the two pairs, in that order, to put the entries into the binary
// traversal's order.
struct WideTreeDev {
    std::vector<WideNodeHost> nodes;
    std::vector<uint32_t> leaf_of;      // first triangle -> binary node, for the leaves that words name
    std::vector<uint32_t> inst_root;    // transform -> the word of its tree, for kWInstance words
    uint32_t root_word = 0;             // where a traversal starts
    float reach = 0.0f;                 // the largest coordinate of an entry box
};
// coordinates of the traversal's error bounds
constexpr float kWideMaxCoord = 1e12f;
// A leaf that a word cannot hold (more than kWLeafMaxCount triangles, a start
// beyond kWLeafStart, a first triangle that another leaf shares) stays a
// ref, as does an instance whose transform leads to two trees.
// ident: bit i of word i / 32 set where transform i is exactly the identity.
// False where the traversal's error bounds do not hold (a coordinate beyond
// kWideMaxCoord).
bool pack_wide_tree(const uint32_t* nodes8, WideTree& tree, size_t num_tris, const std::vector<uint32_t>& ident,
                    WideTreeDev& out);

}  // namespace nb
