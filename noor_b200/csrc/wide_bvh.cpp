// Host collapse of a payload's binary BVH into the four-wide any-hit tree
// (layout and rules in wide_bvh.h).
#include "wide_bvh.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "host_threads.h"
#include "noor_b200.h"

namespace nb {

namespace {

constexpr uint32_t kKindMask =
    NOOR_LIGHT_NODE_MASK | NOOR_MESH_INSTANCE_MASK | NOOR_MESH_LEAF_MASK | NOOR_TRI_LEAF_MASK;

enum Kind : uint8_t { kInner, kLight, kInstance, kMeshLeaf, kTriLeaf };

struct Tree {
    const uint32_t* w;
    size_t nn;
    uint32_t w0(uint32_t n) const { return w[8 * (size_t)n + 3]; }
    uint32_t w1(uint32_t n) const { return w[8 * (size_t)n + 7]; }
    float lo(uint32_t n, int a) const { return bits(w[8 * (size_t)n + a]); }
    float hi(uint32_t n, int a) const { return bits(w[8 * (size_t)n + 4 + a]); }
    static float bits(uint32_t u) {
        float f;
        std::memcpy(&f, &u, 4);
        return f;
    }
    // the node kinds in the order the traversal tells them apart
    Kind kind(uint32_t n) const {
        const uint32_t f = w1(n);
        if (!(f & kKindMask)) return kInner;
        if (f & NOOR_LIGHT_NODE_MASK) return kLight;
        if (f & NOOR_MESH_INSTANCE_MASK) return kInstance;
        if (f & NOOR_MESH_LEAF_MASK) return kMeshLeaf;
        return kTriLeaf;
    }
    // the traversal resets the ray to world space on taking this node
    bool world(uint32_t n) const { return (w1(n) & NOOR_MESH_NODE_MASK) != 0u; }
    uint32_t axis(uint32_t n) const { return w1(n) & NOOR_AXIS_MASK; }
    uint32_t count(uint32_t n) const { return w1(n) & NOOR_COUNT_MASK; }
    bool nan_box(uint32_t n) const {
        for (int a = 0; a < 3; ++a)
            if (std::isnan(lo(n, a)) || std::isnan(hi(n, a))) return true;
        return false;
    }
    bool contains(uint32_t c, uint32_t g) const {
        for (int a = 0; a < 3; ++a)
            if (!(lo(g, a) >= lo(c, a) && hi(g, a) <= hi(c, a))) return false;
        return true;
    }
    // the i-th successor the traversal can take from n (i < num_succ)
    uint32_t num_succ(uint32_t n) const {
        switch (kind(n)) {
            case kInner: return 2;
            case kInstance: return 1;
            case kMeshLeaf: return count(n);
            default: return 0;
        }
    }
    uint32_t succ(uint32_t n, uint32_t i) const {
        switch (kind(n)) {
            case kInner: return i == 0 ? n + 1 : w0(n);
            case kInstance: return w0(n);
            default: return n + 1 + i;
        }
    }
};

}  // namespace

bool build_wide_tree(const uint32_t* nodes8, size_t nn, uint32_t root, int max_stack, WideTree& out,
                     std::string* why) {
    out = WideTree{};
    auto fail = [&](const char* m) {
        if (why) *why = m;
        out = WideTree{};
        return false;
    };
    if (nn == 0 || !ref_words_fit(nn) || root >= nn) return fail("node count or root out of range");
    const Tree T{nodes8, nn};

    // every node the traversal can reach, in post order (successors first),
    // with cycles refused; pure = no instance, mesh or light node in the
    // subtree, so the ray cannot change while the subtree is walked
    std::vector<uint8_t> state(nn, 0);  // 0 new, 1 on the path, 2 done
    std::vector<uint8_t> pure(nn, 0);
    std::vector<uint32_t> post;
    post.reserve(nn);
    {
        std::vector<std::pair<uint32_t, uint32_t>> path;  // node, next successor
        path.emplace_back(root, 0u);
        state[root] = 1;
        while (!path.empty()) {
            auto& top = path.back();
            const uint32_t n = top.first;
            if (top.second < T.num_succ(n)) {
                const uint32_t s = T.succ(n, top.second++);
                if (s >= nn) return fail("successor out of range");
                if (state[s] == 1) return fail("the tree has a cycle");
                if (state[s] == 0) {
                    state[s] = 1;
                    path.emplace_back(s, 0u);
                }
                continue;
            }
            if (T.nan_box(n)) return fail("NaN box bound");
            const Kind k = T.kind(n);
            bool p = !T.world(n) && k != kLight && k != kInstance && k != kMeshLeaf;
            if (p && k == kInner) p = pure[n + 1] && pure[T.w0(n)];
            pure[n] = p ? 1 : 0;
            state[n] = 2;
            post.push_back(n);
            path.pop_back();
        }
    }

    out.map.assign(nn, kWNone);
    out.nodes.reserve(nn / 4);
    out.node.reserve(nn / 4);
    std::vector<uint32_t> work;
    bool deferred = false;
    auto get_wide = [&](uint32_t n) -> uint32_t {
        if (out.map[n] == kWNone) {
            out.map[n] = (uint32_t)out.nodes.size();
            out.nodes.emplace_back();
            out.node.push_back(n);
            work.push_back(n);
        }
        return out.map[n];
    };
    // inner nodes taken from refs: the root, mesh-leaf members, instance roots
    if (T.kind(root) == kInner) get_wide(root);
    for (uint32_t n : post) {
        const Kind k = T.kind(n);
        if (k != kMeshLeaf && k != kInstance) continue;
        for (uint32_t i = 0; i < T.num_succ(n); ++i)
            if (T.kind(T.succ(n, i)) == kInner) get_wide(T.succ(n, i));
    }
    while (!work.empty()) {
        const uint32_t P = work.back();
        work.pop_back();
        const bool world = T.world(P);
        // whether the binary traversal tests x against the ray of P's visit
        auto testable = [&](uint32_t x) { return world ? T.world(x) : (bool)pure[P]; };
        auto entry = [&](uint32_t x) -> uint32_t {
            if (!testable(x)) {
                deferred = true;
                if (T.kind(x) == kInner) get_wide(x);
                return kWRef | kWUntested | x;
            }
            if (T.kind(x) == kInner) return get_wide(x);
            return kWRef | x;
        };
        WideNodeHost h;
        std::memset(&h, 0, sizeof(h));
        uint32_t flags = (world ? kW4World : 0u) | (T.axis(P) << 4);
        const uint32_t cs[2] = {P + 1, T.w0(P)};
        for (int c = 0; c < 2; ++c) {
            const uint32_t C = cs[c];
            uint32_t slot_nodes[2] = {C, kWNone};
            bool expand = false;
            if (T.kind(C) == kInner && testable(C)) {
                const uint32_t g0 = C + 1, g1 = T.w0(C);
                expand = testable(g0) && testable(g1) && T.contains(C, g0) && T.contains(C, g1);
                if (expand) {
                    slot_nodes[0] = g0;
                    slot_nodes[1] = g1;
                    flags |= (c == 0 ? kW4ExpandL : kW4ExpandR) | (T.axis(C) << (c == 0 ? 6 : 8));
                }
            }
            for (int j = 0; j < 2; ++j) {
                const int s = 2 * c + j;
                const uint32_t x = slot_nodes[j];
                if (x == kWNone) {
                    h.child[s] = kWNone;
                    continue;
                }
                // entry() may grow out.nodes: write through the index afterwards
                h.child[s] = entry(x);
                for (int a = 0; a < 3; ++a) {
                    h.lo[a][s] = T.lo(x, a);
                    h.hi[a][s] = T.hi(x, a);
                }
            }
        }
        h.meta[0] = flags;
        out.nodes[out.map[P]] = h;
    }

    // deepest stack: a wide node with k entries pushes k - 1 of them before
    // taking the first, a mesh leaf of n members pushes n - 1, and below a
    // ray that may not skip boxes inner nodes are walked one by one (one push
    // each); the larger of the two counts
    std::vector<int> need(nn, 0);
    for (uint32_t n : post) {
        int v = 0;
        switch (T.kind(n)) {
            case kInner:
                if (out.map[n] != kWNone) {
                    const WideNodeHost& h = out.nodes[out.map[n]];
                    int k = 0, m = 0;
                    for (int s = 0; s < 4; ++s) {
                        if (h.child[s] == kWNone) continue;
                        ++k;
                        // the entry's binary node: the ref's, else slot s's (the
                        // left or right child, or one of their children)
                        uint32_t bx = (h.child[s] & kWRef) ? (h.child[s] & kWIndex) : kWNone;
                        if (bx == kWNone) {
                            const uint32_t C = s < 2 ? n + 1 : T.w0(n);
                            const bool ex = (h.meta[0] & (s < 2 ? kW4ExpandL : kW4ExpandR)) != 0u;
                            bx = !ex ? C : ((s & 1) ? T.w0(C) : C + 1);
                        }
                        m = std::max(m, need[bx]);
                    }
                    v = (k > 0 ? k - 1 : 0) + m;
                }
                v = std::max(v, 1 + std::max(need[n + 1], need[T.w0(n)]));
                break;
            case kMeshLeaf: {
                const uint32_t cnt = T.count(n);
                int m = 0;
                for (uint32_t i = 1; i <= cnt; ++i) m = std::max(m, need[n + i]);
                v = cnt ? (int)cnt - 1 + m : 0;
                break;
            }
            case kInstance: v = need[T.w0(n)]; break;
            default: break;
        }
        need[n] = v;
    }
    out.stack_need = need[root];
    out.root = root;
    // the binary traversal's stack: one push per inner node, n - 1 per mesh
    // leaf of n members
    for (uint32_t n : post) {
        int v = 0;
        for (uint32_t i = 0; i < T.num_succ(n); ++i) v = std::max(v, need[T.succ(n, i)]);
        if (T.kind(n) == kInner) v += 1;
        if (T.kind(n) == kMeshLeaf && T.count(n)) v += (int)T.count(n) - 1;
        need[n] = v;
    }
    out.binary_need = need[root];
    if (out.stack_need > max_stack) return fail("the four-wide traversal needs a deeper stack than allowed");
    // closest hit re-tests every binary node when it is taken and relies on
    // each entry box being tested against the ray of its parent's visit: no
    // deferred entries
    out.closest = !deferred;
    return true;
}

bool pack_wide_tree(const uint32_t* nodes8, WideTree& tree, size_t num_tris, const std::vector<uint32_t>& ident,
                    WideTreeDev& out) {
    out = WideTreeDev{};
    const Tree T{nodes8, tree.map.size()};
    const size_t n = tree.nodes.size(), ni = 32 * ident.size();
    out.leaf_of.assign(std::max<size_t>(num_tris, 1), kWNone);
    out.inst_root.assign(std::max<size_t>(ni, 1), kWNone);
    auto leaf_fits = [&](uint32_t x) {
        const uint32_t cnt = T.w1(x) & NOOR_TRI_COUNT_MASK;
        return T.kind(x) == kTriLeaf && cnt >= 1 && cnt <= kWLeafMaxCount && T.w0(x) <= kWLeafStart &&
               T.w0(x) < num_tris;
    };
    auto claim_leaf = [&](uint32_t x) {
        if (leaf_fits(x) && out.leaf_of[T.w0(x)] == kWNone) out.leaf_of[T.w0(x)] = x;
    };
    // the instance node an entry leads to: itself, or the only member of a
    // mesh leaf whose box holds it; kWNone where there is none
    auto instance_of = [&](uint32_t x) {
        if (T.kind(x) == kMeshLeaf && T.count(x) == 1 && T.contains(x, x + 1)) x = x + 1;
        return T.kind(x) == kInstance ? x : kWNone;
    };
    auto transform = [&](uint32_t x) { return T.w1(x) & NOOR_TRANS_MASK; };
    // the transform is the identity, and the box holds the tree's: the boxes
    // of the tree are tested against the same ray as the instance's, and one
    // that passes is inside it
    auto same_space = [&](uint32_t x) {
        const uint32_t t = transform(x);
        return t < ni && t <= kWIndex && ((ident[t / 32] >> (t % 32)) & 1u) && T.contains(x, T.w0(x));
    };
    // an inner node whose children stick out of its box is tested exactly
    auto inner_word = [&](uint32_t x) {
        const uint32_t w = tree.map[x];
        return w != kWNone && T.contains(x, x + 1) && T.contains(x, T.w0(x)) ? w : kWRef | x;
    };
    auto tree_word = [&](uint32_t x) -> uint32_t {
        if (T.kind(x) == kInner) return inner_word(x);
        if (leaf_fits(x) && out.leaf_of[T.w0(x)] == x)
            return kWRef | kWLeaf | ((T.w1(x) & NOOR_TRI_COUNT_MASK) - 1u) << kWLeafShift | T.w0(x);
        const uint32_t i = instance_of(x);
        if (i != kWNone && same_space(i) && out.inst_root[transform(i)] != kWNone) return kWInstance | transform(i);
        return kWRef | x;
    };
    float reach = 0.0f;
    std::vector<uint32_t> inst;
    auto see_entry = [&](uint32_t x) {
        claim_leaf(x);
        const uint32_t i = instance_of(x);
        if (i == kWNone || !same_space(i)) return;
        claim_leaf(T.w0(i));
        inst.push_back(i);
    };
    see_entry(tree.root);
    for (const WideNodeHost& h : tree.nodes)
        for (int s = 0; s < 4; ++s) {
            if (h.child[s] == kWNone) continue;
            for (int a = 0; a < 3; ++a) reach = std::max(reach, std::max(std::fabs(h.lo[a][s]), std::fabs(h.hi[a][s])));
            if ((h.child[s] & (kWRef | kWUntested)) == kWRef) see_entry(h.child[s] & kWIndex);
        }
    if (!(reach <= kWideMaxCoord)) return false;
    out.reach = reach;
    // one tree per transform
    std::vector<uint32_t> root_of(out.inst_root.size(), kWNone);
    for (uint32_t i : inst) {
        uint32_t& r = root_of[transform(i)];
        r = r == kWNone || r == T.w0(i) ? T.w0(i) : kWRef;
    }
    for (size_t t = 0; t < root_of.size(); ++t) {
        if (root_of[t] == kWNone || root_of[t] == kWRef) continue;
        // trees of instances inside instances are taken as refs
        const uint32_t r = root_of[t];
        out.inst_root[t] = T.kind(r) == kInner ? inner_word(r) : (T.kind(r) == kTriLeaf ? tree_word(r) : kWRef | r);
    }
    out.root_word = tree_word(tree.root);
    out.nodes.swap(tree.nodes);
    nbh::parallel_ranges(n, 2048, 16, [&](size_t b, size_t e) {
        for (size_t i = b; i < e; ++i) {
            WideNodeHost& h = out.nodes[i];
            for (int s = 0; s < 4; ++s) {
                const uint32_t w = h.child[s];
                const bool none = w == kWNone, deferred = !none && (w & (kWRef | kWUntested)) == (kWRef | kWUntested);
                for (int a = 0; a < 3; ++a) {
                    // a box of the tree's that is inside out (the slab test can still pass
                    // it) gets the box around it
                    const float lo = std::min(h.lo[a][s], h.hi[a][s]), hi = std::max(h.lo[a][s], h.hi[a][s]);
                    h.lo[a][s] = none ? 3.4e38f : (deferred ? -3.4e38f : lo);
                    h.hi[a][s] = none ? -3.4e38f : (deferred ? 3.4e38f : hi);
                }
                if (none) continue;
                if (!(w & kWRef))
                    h.child[s] = inner_word(tree.node[w]);
                else
                    h.child[s] = deferred ? kWRef | (w & kWIndex) : tree_word(w & kWIndex);
            }
            const uint32_t f = h.meta[0];
            uint32_t flips = 0;
            for (uint32_t o = 0; o < 8; ++o) {
                uint32_t k = (o >> ((f >> 4) & 3u)) & 1u ? 4u : 0u;
                if ((f & kW4ExpandL) && ((o >> ((f >> 6) & 3u)) & 1u)) k |= 1u;
                if ((f & kW4ExpandR) && ((o >> ((f >> 8) & 3u)) & 1u)) k |= 2u;
                flips |= k << (3 * o);
            }
            h.meta[0] = f & kW4World;
            h.meta[1] = flips;
            h.meta[2] = h.meta[3] = 0;
        }
    });
    return true;
}

}  // namespace nb

#include "host_common.h"

extern "C" int noor_wide_tree_info(const noor_payload* payload, uint32_t root, uint32_t* num_wide,
                                   uint32_t* num_expanded, uint32_t* stack_need, uint32_t* closest) {
    if (!payload || !payload->bvh_min_right_start || !payload->bvh_max_axis_count || !num_wide || !num_expanded ||
        !stack_need || !closest || root >= payload->num_bvh_nodes)
        return set_error(NOOR_ERR_INVALID, "noor_wide_tree_info: bad argument");
    const size_t nn = payload->num_bvh_nodes;
    std::vector<uint32_t> w(8 * nn);
    for (size_t i = 0; i < nn; ++i) {
        std::memcpy(&w[8 * i], payload->bvh_min_right_start + 4 * i, 16);
        std::memcpy(&w[8 * i + 4], payload->bvh_max_axis_count + 4 * i, 16);
    }
    nb::WideTree t;
    std::string why;
    if (!nb::build_wide_tree(w.data(), nn, root, nb::kWideMaxStack, t, &why))
        return set_error(NOOR_ERR_UNSUPPORTED, "four-wide tree: " + why);
    uint32_t ex = 0;
    for (const nb::WideNodeHost& h : t.nodes)
        ex += ((h.meta[0] & nb::kW4ExpandL) ? 1u : 0u) + ((h.meta[0] & nb::kW4ExpandR) ? 1u : 0u);
    *num_wide = (uint32_t)t.nodes.size();
    *num_expanded = ex;
    *stack_need = (uint32_t)t.stack_need;
    *closest = t.closest ? 1u : 0u;
    clear_error();
    return NOOR_OK;
}
