// fmm_build.cuh -- the reference octree and its interaction lists built on the device.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gx {

constexpr int kKeyLevels = 21;  // octant levels a 63-bit path key resolves
constexpr int kBboxBlocks = 296;

// Tree topology from the bodies (layout of fmm_tree.hpp).  Capacity is the number of node
// slots allocated; hdr receives {n_nodes, n_levels, overflow} where overflow is 1 when a
// node below kKeyLevels still has to split (the host builder takes such trees) and 2 when
// the node slots ran out.
struct TreeBuildArgs {
    int32_t n;
    const double* x;
    const double* y;
    const double* z;
    double softening;
    int64_t cap;
    int max_depth;
    int32_t capacity;
    double* part;     // bbox partials, 6 * kBboxBlocks
    double* root;     // cx, cy, cz, hw
    uint64_t* keys;   // n, then sorted in place through keys_alt
    uint64_t* keys_alt;
    int32_t* idx;     // n
    int32_t* perm;    // n: bodies in tree order
    int32_t* beg;     // capacity each
    int32_t* end;
    int32_t* child;
    double* cx;
    double* cy;
    double* cz;
    double* hw;
    int32_t* level_off;  // kKeyLevels + 3
    int32_t* hdr;        // 3
    // Levels of the key that the sort orders (0: all kKeyLevels).  Fewer levels take fewer
    // radix passes; a tree that would split a node at that depth sets hdr[2] bit 2 instead
    // (the caller rebuilds with more levels).
    int key_levels;
};
size_t tree_build_temp_bytes(int32_t n, int64_t cap);
cudaError_t launch_tree_build(const TreeBuildArgs& t, void* temp, size_t temp_bytes, int sms, cudaStream_t st);
// After a successful build: bodies of every leaf in ascending index order in t.perm
// (uses t.idx as scratch).
cudaError_t launch_tree_leaf_order(const TreeBuildArgs& t, int32_t n_nodes, void* temp, size_t temp_bytes,
                                   cudaStream_t st);

// What the list walk reads of a node, packed (48 B: three 16-byte loads).
struct __align__(16) WalkNode {
    double cx, cy, cz, hw;
    int32_t child;  // first child, -1 for a leaf
    int32_t mask;   // bit c set when child c has mass > 0
    int32_t leaf;   // ordinal among the leaves with mass > 0 (leaves only)
    int32_t count;  // bodies
};

// Counters of the list passes, zeroed before them.
struct ListCounters {
    unsigned long long far, near;              // list entries
    unsigned long long chunks;                 // far-list chunks (work items) reserved
    unsigned long long slots;                  // partial sums of leaves with several chunks
    unsigned long long far_pairs, near_pairs;  // (body, far node) and (body, body) pairs
    unsigned long long segs;                   // segments of long near lists reserved
    int ticket, n_long, n_slow;
    int leaves;                                // leaves with mass > 0
};
constexpr int kNearSeg = 512;  // entries of a segment of a long near list
constexpr int kWalkStackSlots = 1024;  // entries a walk's stack may hold

// Leaves with mass > 0 (depth-first) and their near / far lists, after the node moments.
struct TreeListArgs {
    int32_t n;
    int32_t n_nodes;
    const int32_t* beg;
    const int32_t* end;
    const int32_t* child;
    const int32_t* perm;
    const double* cx;
    const double* cy;
    const double* cz;
    const double* hw;
    const double* rec;  // node records (mass at slot 3)
    // Optional (capacity mode): the bodies' masses and, filled by launch_tree_massive, the
    // number of bodies with mass > 0 before each tree position (n + 1).  With all masses
    // finite and >= 0 a node's mass is > 0 exactly when its range holds such a body, so the
    // lists then need no node records and can be built while the moments are computed.
    const double* m;
    int32_t* mprefix;
    WalkNode* wn;       // n_nodes, filled before the walk
    double theta;
    int walk_stack;     // at most kWalkStackSlots: where a walk's stack counts as overflowing
    int64_t t_begin, t_end;
    // body-position scratch, n + 1 each
    int64_t* mark;   // bodies of leaves with mass > 0: 1 in the high word, the leaf's first also in the low
    int64_t* place;  // its exclusive scan: place among those bodies, leaves before
    // leaves, n_nodes + 1 each
    int32_t* leaf_off;
    int32_t* leaf_part;  // n
    int32_t* leaf_node;
    int32_t* node_leaf;  // n_nodes
    // Lists of leaf l (n_nodes entries each): near leaves near_leaf[near_beg .. near_end), their
    // bodies near_src, far chunks far_nch, first partial-sum slot (far_nch > 1) far_slot.
    int32_t* near_beg;
    int32_t* near_end;
    int32_t* near_src;
    int32_t* far_nch;
    int64_t* far_slot;
    ListCounters* counters;
    // far_cap chunks of kM2PChunk far nodes, each with its work item of the same number
    // (M2PItem); a leaf's chunks are numbered in walk order but lie anywhere in the pool
    int32_t* far_node;
    void* items;
    int32_t* near_leaf;  // near_cap leaf ordinals
    // near lists too long for a warp's buffer: linked segments of unsorted ordinals, then the
    // leaves that have them; and leaves whose walk overflowed its stack
    int32_t* seg_near;   // seg_cap * kNearSeg
    int32_t* seg_next;   // seg_cap
    int32_t* seg_count;  // seg_cap
    int32_t* long_leaf;  // n_nodes each
    int32_t* long_head;
    int32_t* long_near;
    int32_t* slow_leaf;
    // Capacity mode (nullable cnt_nodes / overflow): n_nodes is the capacity of the node
    // arrays and the count is read on the device (cnt_nodes = the topology build's header
    // {nodes, levels, flags}; a flag leaves no nodes); pool_check marks an overflow when a total
    // exceeds its pool (and records the largest totals seen in need, with a sticky copy of the
    // flag), and everything after the lists is skipped.
    const int32_t* cnt_nodes;
    int* overflow;
    int* overflow_sticky;
    unsigned long long* need;  // kNeed: {nodes, chunks, near, slots, tree levels, segments}
    // pools (in both modes; writes past them are left out and the totals tell): chunks,
    // entries, segments, slots
    int64_t far_cap, near_cap, seg_cap, slot_cap;
};
constexpr int kNeed = 6;
// Where the scan leaves the number of leaves (device memory).
__host__ __device__ inline const int32_t* leaf_count_of(const TreeListArgs& a) {
    return reinterpret_cast<const int32_t*>(a.place + a.n);
}
size_t tree_list_temp_bytes(int32_t n, int32_t n_nodes);
// Leaf compaction and the lists with their far-field work items (kernels read the number of leaves
// on the device; sizes become known on the host, when it wants them, from the counters).
cudaError_t launch_tree_lists(const TreeListArgs& a, void* temp, size_t temp_bytes, int sms, cudaStream_t st);
// The near lists one after the other in leaf order: leaf l's, from near_beg[l] of near_leaf on, to
// out[off[l] .. off[l + 1]).
cudaError_t launch_near_gather(int32_t n_leaves, const int32_t* near_beg, const int32_t* near_leaf, const int32_t* off,
                               int32_t* out, cudaStream_t st);
// mprefix from the masses (a.m, a.perm); a mass < 0 or NaN marks an overflow with bit 1 of
// the sticky word (the caller then evaluates through the host-read path).  temp: scan scratch
// for n + 1 ints.
cudaError_t launch_tree_massive(const TreeListArgs& a, void* temp, size_t temp_bytes, cudaStream_t st);
// Capacity mode: after the lists, the overflow check of the pools (and of the topology build's
// header tree_hdr).
cudaError_t launch_pool_check(const TreeListArgs& a, const int32_t* tree_hdr, cudaStream_t st);
// The far-field items reordered by decreasing cost (targets x nodes) into out, completed with
// their leaves' chunk counts and partial-sum slots.
struct M2PItem;
size_t item_order_temp_bytes(int32_t n_items);
// n_items is the length of the arrays; n_real (nullable: all) the items on the device.
cudaError_t launch_item_order(const TreeListArgs& a, int32_t n_items, const unsigned long long* n_real,
                              const int* overflow, uint32_t* cost, uint32_t* cost_alt, int32_t* idx, int32_t* idx_alt,
                              void* temp, size_t temp_bytes, M2PItem* out, int sms, cudaStream_t st);

}  // namespace gx
