// fmm_build.cu -- the reference octree (FastMultipoleSolver::build,
// cpp/fmm/fmm_solver.cpp:48-98) and its interaction lists (:228-277) built on the device.
//
// The reference inserts bodies one at a time; a leaf splits when it would hold more than
// leaf_capacity bodies below max_depth (:133-155).  The resulting tree is the recursive
// 8-way partition in which exactly the nodes with more than leaf_capacity bodies above
// max_depth are split.  A body's octant at every level depends only on its position and on
// the cell centres along its path, which follow the reference's recurrence
// (child centre = centre +- half_width * 0.5, :111-131; octant by >=, :104-109).  So:
//   1. root cell from the bounding box (:62-85);
//   2. every body's path as a 63-bit key, 3 bits per level, level 0 in the top bits;
//   3. a stable radix sort of (key, body): depth-first tree order;
//   4. the octants that a sorted body has in common with its neighbour and with the body
//      leaf_capacity places on tell at which levels it starts a node that splits; counts per
//      level and block of bodies number the nodes, and eight lanes per node find its children;
//   5. one warp per leaf sorts the leaf's bodies into ascending index order, the order
//      the reference's sums run in.
// Nodes are numbered breadth-first.  Trees that need a split below level 21 (more than
// leaf_capacity nearly coincident bodies) are reported back for the host builder.
//
// Lists: every leaf with mass > 0 is walked once with the reference's tests (mass > 0,
// well_separated, leaf) by one warp over a shared-memory stack; far nodes go straight into
// chunks of a pool (one far-field work item each), near leaves into a buffer that is sorted into the
// reference's depth-first order.
#include "fmm_build.cuh"
#include "fmm.cuh"
#include "gx_device.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <atomic>
#include <cfloat>

namespace gx {
namespace {

constexpr int kBboxThreads = 256;
constexpr int kWalkThreads = 128;  // 4 warps, one leaf each
// Slots of a warp's shared buffer: its stack grows from the bottom (up to kWalkStack), the near
// leaves it has met from the top (up to kWalkNear).  4 x 1152 x 4 B = 18 KiB per block, plus the
// 1 KiB the runtime reserves: 8 blocks (32 warps, the count __launch_bounds__(kWalkThreads, 8)
// sizes the registers for) take 152 KiB, inside the 70% shared-memory carveout asked for; the
// rest of the SM's unified memory stays L1 for the node-record loads.
constexpr int kWalkSlots = 1152;
constexpr int kWalkStack = 1024;
constexpr int kWalkNear = 512;
static_assert(kWalkNear == kNearSeg, "a full buffer is one segment");
static_assert(kWalkStack == kWalkStackSlots, "the host's bound of the stack");
constexpr int kStack = 7 * (kKeyLevels + 1) + 8;

__global__ void __launch_bounds__(kBboxThreads) bbox_partial_kernel(const TreeBuildArgs t) {
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int i = blockIdx.x * kBboxThreads + threadIdx.x; i < t.n; i += gridDim.x * kBboxThreads) {
        const double v[3] = {t.x[i], t.y[i], t.z[i]};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = fmin(lo[c], v[c]);
            hi[c] = fmax(hi[c], v[c]);
        }
    }
    __shared__ double s[6][kBboxThreads / 32];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = warp_min(lo[c]);
        hi[c] = warp_max(hi[c]);
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int c = 0; c < 3; ++c) {
            s[c][w] = lo[c];
            s[3 + c][w] = hi[c];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = s[threadIdx.x][0];
        for (int k = 1; k < kBboxThreads / 32; ++k) v = threadIdx.x < 3 ? fmin(v, s[threadIdx.x][k]) : fmax(v, s[threadIdx.x][k]);
        t.part[blockIdx.x * 6 + threadIdx.x] = v;
    }
}

__device__ __forceinline__ int octant_of(double x, double y, double z, double cx, double cy, double cz) {
    return (x >= cx ? 1 : 0) + (y >= cy ? 2 : 0) + (z >= cz ? 4 : 0);
}

// Child centre (subdivide, fmm_solver.cpp:111-131): centre + sign * (half_width * 0.5).
__device__ __forceinline__ double child_centre(double c, double chw, bool up) { return dadd(c, up ? chw : -chw); }

// Root cell (fmm_solver.cpp:62-85) from the partial extrema -- every block reduces them for itself
// (minima and maxima do not depend on the order), block 0 stores it -- and the path keys.  Block 0
// also clears the build's flags and the ticket of split_count_kernel.
__global__ void __launch_bounds__(kBboxThreads) keys_kernel(const TreeBuildArgs t, int blocks, int* ticket) {
    __shared__ double s[6][kBboxThreads / 32];
    __shared__ double s_root[4];
    double lo[3] = {DBL_MAX, DBL_MAX, DBL_MAX}, hi[3] = {-DBL_MAX, -DBL_MAX, -DBL_MAX};
    for (int b = threadIdx.x; b < blocks; b += kBboxThreads)
        for (int c = 0; c < 3; ++c) {
            lo[c] = fmin(lo[c], t.part[b * 6 + c]);
            hi[c] = fmax(hi[c], t.part[b * 6 + 3 + c]);
        }
    for (int c = 0; c < 3; ++c) {
        lo[c] = warp_min(lo[c]);
        hi[c] = warp_max(hi[c]);
    }
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int c = 0; c < 3; ++c) {
            s[c][w] = lo[c];
            s[3 + c][w] = hi[c];
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int c = 0; c < 3; ++c)
            for (int k = 1; k < kBboxThreads / 32; ++k) {
                s[c][0] = fmin(s[c][0], s[c][k]);
                s[3 + c][0] = fmax(s[3 + c][0], s[3 + c][k]);
            }
        for (int c = 0; c < 3; ++c) s_root[c] = dmul(dadd(s[c][0], s[3 + c][0]), 0.5);
        double hw = dmul(0.5, fmax(fmax(dsub(s[3][0], s[0][0]), dsub(s[4][0], s[1][0])), dsub(s[5][0], s[2][0])));
        hw = fmax(hw, dadd(t.softening, 1.0e-6));
        s_root[3] = dmul(hw, 1.0001);
        if (blockIdx.x == 0) {
            for (int c = 0; c < 4; ++c) t.root[c] = s_root[c];
            for (int c = 0; c < 3; ++c) t.hdr[c] = 0;
            *ticket = 0;
        }
    }
    __syncthreads();
    for (int i = blockIdx.x * kBboxThreads + threadIdx.x; i < t.n; i += gridDim.x * kBboxThreads) {
        const double x = t.x[i], y = t.y[i], z = t.z[i];
        double cx = s_root[0], cy = s_root[1], cz = s_root[2], hw = s_root[3];
        uint64_t key = 0;
        for (int l = 0; l < kKeyLevels; ++l) {
            const int o = octant_of(x, y, z, cx, cy, cz);
            key |= (uint64_t)o << (3 * (kKeyLevels - 1 - l));
            const double chw = dmul(hw, 0.5);
            cx = child_centre(cx, chw, o & 1);
            cy = child_centre(cy, chw, o & 2);
            cz = child_centre(cz, chw, o & 4);
            hw = chw;
        }
        t.keys[i] = key;
        t.idx[i] = i;
    }
}

// First position p in [b, e) whose octant at shift sh is >= o (octants are non-decreasing
// in a cell's sorted range).
__device__ __forceinline__ int lower_octant(const uint64_t* keys, int b, int e, int sh, int o) {
    while (b < e) {
        const int mid = (b + e) >> 1;
        if ((int)((keys[mid] >> sh) & 7) < o) b = mid + 1;
        else e = mid;
    }
    return b;
}

// The topology in parallel from the sorted path keys.  A node at depth L is a key prefix of
// L octants (key >> 3 (kKeyLevels - L)); it splits when it holds more than cap bodies and
// L < max_depth, and a splitting node's 8 children (all of them, empty ones included) are
// the nodes of depth L + 1.  Nodes are numbered breadth-first with children in octant order,
// i.e. level by level in key-prefix order, so a node's number follows from counts alone.  Sorted
// body i is the first of a splitting prefix for the depths [lo, hi] where lo - 1 octants are common
// to it and body i - 1, and hi octants to it and body i + cap (SplitRange), so
//   split_count_kernel counts the splitting prefixes per depth and block of bodies, and its last
//   block scans the counts: S_L, level_off[L + 1] = level_off[L] + 8 S_(L-1) (level_off[0] = 0,
//   level_off[1] = 1), and each block's first rank of every depth;
//   split_emit_kernel ranks them by ballots and lists them in (depth, key) order with their own
//   node's number, which the rank of their parent's prefix gives;
//   tree_children_kernel writes the children's records, from level_off[L + 1] + 8 rank on.
// Latency-bound, so what counts is launches and dependent loads: N = 65,536 leaf 64 30 us for the
// three, N = 1000 26 and N = 2^20 leaf 16 52, against 62, 45 and 130 us with a flag per body
// and depth, a scan of all of them (22 M at N = 2^20) and binary searches over whole prefixes.
// A node's centre is the reference's recurrence (subdivide, fmm_solver.cpp:111-131) walked
// from the root along its prefix -- the same operations in the same order as building level
// by level, so the same bits.  A prefix of depth kKeyLevels that would still split needs a
// deeper key: hdr[2] bit 0 hands the tree to the host builder.  When the sort ordered only
// the first key_levels levels, a prefix of that depth that would split sets hdr[2] bit 2
// instead (the build stops there; the caller redoes it with all levels).

__device__ __forceinline__ uint64_t key_prefix(uint64_t key, int L) {
    const int sh = 3 * (kKeyLevels - L);
    return sh >= 64 ? 0 : key >> sh;
}

// Leading octants that two keys have in common.
__device__ __forceinline__ int common_levels(uint64_t p, uint64_t q) {
    return p == q ? kKeyLevels : (__clzll((long long)(p ^ q)) - 1) / 3;
}

// Depths at which sorted body i starts a splitting prefix (hi < lo: none).  flags: what the build
// cannot do, as hdr[2] bits -- a prefix of all kKeyLevels that would split (1), or one at a depth
// whose children the sort has not ordered (4).
struct SplitRange {
    int lo, hi, flags;
    __device__ __forceinline__ SplitRange(const TreeBuildArgs& t, const uint64_t* keys, int i) : lo(0), hi(-1), flags(0) {
        if (i >= t.n || (int64_t)i + t.cap >= (int64_t)t.n) return;
        const int sorted = t.key_levels > 0 ? t.key_levels : kKeyLevels;  // levels the sort ordered
        const int lmax = min(t.max_depth, kKeyLevels + 1);
        const uint64_t key = keys[i];
        if (i > 0) lo = common_levels(key, keys[i - 1]) + 1;
        hi = min(common_levels(key, keys[i + t.cap]), lmax - 1);
        if (lo <= kKeyLevels && hi >= kKeyLevels) flags |= 1;
        hi = min(hi, kKeyLevels - 1);
        if (lo <= hi && hi >= sorted) flags |= 4;
        hi = min(hi, sorted - 1);
    }
};

// Depths in which any body of a warp starts a splitting prefix (hi < lo: none).
__device__ __forceinline__ int2 warp_depths(const SplitRange& r) {
    const bool any = r.lo <= r.hi;
    return make_int2(__reduce_min_sync(0xffffffffu, any ? r.lo : kKeyLevels),
                     __reduce_max_sync(0xffffffffu, any ? r.hi : -1));
}

constexpr int kTopoThreads = 256;
constexpr int kTopoPer = 4;                                   // bodies per thread
constexpr int kTopoBodies = kTopoThreads * kTopoPer;          // ... and per block
constexpr int kTopoGroups = kTopoBodies / 32;                 // groups of 32 bodies (one ballot each)
static_assert(kTopoGroups == 32, "a warp scans the groups of a block");

// What split_count_kernel leaves for the other two: start[L] = splitting prefixes above depth L
// (start[kKeyLevels]: all), first[L * blocks + b] = rank at depth L of block b's first.
struct Topology {
    int* ticket;
    int* start;  // kKeyLevels + 1
    int* first;  // kKeyLevels * blocks
    int2* split; // (first body, node) in (depth, key) order
    int blocks;
    int split_cap;
};

__global__ void __launch_bounds__(kTopoThreads) split_count_kernel(const TreeBuildArgs t, const uint64_t* keys,
                                                                   const Topology p) {
    __shared__ int s_cnt[kKeyLevels][kTopoGroups];
    __shared__ int s_total[kKeyLevels];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (int k = tid; k < kKeyLevels * kTopoGroups; k += kTopoThreads) (&s_cnt[0][0])[k] = 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kTopoPer; ++u) {
        const SplitRange r(t, keys, blockIdx.x * kTopoBodies + u * kTopoThreads + tid);
        if (r.flags) atomicOr(&t.hdr[2], r.flags);
        const int2 d = warp_depths(r);
        for (int L = d.x; L <= d.y; ++L) {
            const unsigned m = __ballot_sync(0xffffffffu, r.lo <= L && L <= r.hi);
            if (lane == 0) s_cnt[L][u * (kTopoThreads / 32) + w] = __popc(m);
        }
    }
    __syncthreads();
    for (int L = w; L < kKeyLevels; L += kTopoThreads / 32) {
        const int c = __reduce_add_sync(0xffffffffu, s_cnt[L][lane]);
        if (lane == 0) p.first[(size_t)L * p.blocks + blockIdx.x] = c;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(p.ticket, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last block: exclusive scans over the blocks, a warp per depth
    for (int L = w; L < kKeyLevels; L += kTopoThreads / 32) {
        int* const f = p.first + (size_t)L * p.blocks;
        int carry = 0;
#pragma unroll 4
        for (int b = lane; b - lane < p.blocks; b += 32) {
            const int c = b < p.blocks ? __ldcg(f + b) : 0;
            int run = c;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= o) run += y;
            }
            if (b < p.blocks) f[b] = carry + run - c;
            carry += __shfl_sync(0xffffffffu, run, 31);
        }
        if (lane == 0) s_total[L] = carry;
    }
    __syncthreads();
    if (w != 0) return;
    // lane L: depth L; S_L = 0 ends the tree
    const int c = lane < kKeyLevels ? s_total[lane] : 0;
    int64_t run = c;
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += y;
    }
    if (lane <= kKeyLevels) p.start[lane] = (int)(run - c);
    const int deep = __ffs(__ballot_sync(0xffffffffu, c == 0)) - 1;  // depths with splitting nodes
    const int64_t off = 1 + 8 * run;
    const int32_t off32 = off <= 0x7fffffffLL ? (int32_t)off : 0x7fffffff;
    if (lane < deep) t.level_off[lane + 2] = off32;
    if (lane == deep) {  // run: all of them
        t.level_off[0] = 0;
        t.level_off[1] = 1;
        t.level_off[deep + 2] = off32;
        t.hdr[0] = off32;
        t.hdr[1] = deep + 1;
        if (off > t.capacity) atomicOr(&t.hdr[2], 2);
    }
}

// The splitting nodes in (depth, key) order; every node starts as a leaf (child -1); the root's record.
__global__ void __launch_bounds__(kTopoThreads) split_emit_kernel(const TreeBuildArgs t, const uint64_t* keys,
                                                                  const Topology p) {
    __shared__ int s_cnt[kKeyLevels][kTopoGroups];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    SplitRange r[kTopoPer] = {{t, keys, (int)blockIdx.x * kTopoBodies + tid},
                              {t, keys, (int)blockIdx.x * kTopoBodies + kTopoThreads + tid},
                              {t, keys, (int)blockIdx.x * kTopoBodies + 2 * kTopoThreads + tid},
                              {t, keys, (int)blockIdx.x * kTopoBodies + 3 * kTopoThreads + tid}};
    for (int k = tid; k < kKeyLevels * kTopoGroups; k += kTopoThreads) (&s_cnt[0][0])[k] = 0;
    __syncthreads();
    int2 d[kTopoPer];
#pragma unroll
    for (int u = 0; u < kTopoPer; ++u) {
        d[u] = warp_depths(r[u]);
        for (int L = d[u].x; L <= d[u].y; ++L) {
            const unsigned m = __ballot_sync(0xffffffffu, r[u].lo <= L && L <= r[u].hi);
            if (lane == 0) s_cnt[L][u * (kTopoThreads / 32) + w] = __popc(m);
        }
    }
    __syncthreads();
    for (int L = w; L < kKeyLevels; L += kTopoThreads / 32) {  // rank of each group's first
        const int c = s_cnt[L][lane];
        int run = c;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += y;
        }
        s_cnt[L][lane] = p.first[(size_t)L * p.blocks + blockIdx.x] + run - c;
    }
    __syncthreads();
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int u = 0; u < kTopoPer; ++u) {
        const int i = blockIdx.x * kTopoBodies + u * kTopoThreads + tid;
        const int g = u * (kTopoThreads / 32) + w;
        // splitting prefixes one depth up that start at or before body i
        int parents = d[u].x > 0 && d[u].x < kKeyLevels ? s_cnt[d[u].x - 1][g] : 0;
        for (int L = d[u].x; L <= d[u].y; ++L) {
            const bool mine = r[u].lo <= L && L <= r[u].hi;
            const unsigned m = __ballot_sync(0xffffffffu, mine);
            const int rank = s_cnt[L][g] + __popc(m & below);
            if (mine) {
                const int e = p.start[L] + rank;
                int self = 0;
                if (L > 0) self = t.level_off[L] + 8 * (parents - 1) + (int)((keys[i] >> (3 * (kKeyLevels - L))) & 7);
                if (e < p.split_cap) p.split[e] = make_int2(i, self);
            }
            parents = rank + (mine ? 1 : 0);
        }
    }
    const int nodes = min(t.hdr[0], t.capacity);
    for (int k = blockIdx.x * kTopoThreads + tid; k < nodes; k += gridDim.x * kTopoThreads) t.child[k] = -1;
    if (blockIdx.x == 0 && tid == 0) {
        t.beg[0] = 0;
        t.end[0] = t.n;
        t.cx[0] = t.root[0];
        t.cy[0] = t.root[1];
        t.cz[0] = t.root[2];
        t.hw[0] = t.root[3];
    }
}

// Eight lanes per splitting node: its end by a search with eight probes a round, each child's first
// body by binary search on the octant inside the node's range, and the children's records, their
// centres by the reference's recurrence walked from the root along the path.
__global__ void __launch_bounds__(256) tree_children_kernel(const TreeBuildArgs t, const uint64_t* keys, const Topology p) {
    if (t.hdr[2] & 2) return;
    __shared__ int s_start[kKeyLevels + 1];
    if (threadIdx.x <= kKeyLevels) s_start[threadIdx.x] = p.start[threadIdx.x];
    __syncthreads();
    const int total = min(s_start[kKeyLevels], p.split_cap);
    const int lane = threadIdx.x & 31, c = lane & 7;
    const unsigned group = 0xffu << (lane & 24);
    for (int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x; q < 8 * (int64_t)total; q += (int64_t)gridDim.x * 256) {
        const int k = (int)(q >> 3);
        int L = 0;
        while (L < kKeyLevels - 1 && s_start[L + 1] <= k) ++L;
        const int2 sp = p.split[k];
        const int i = sp.x;
        const uint64_t key = keys[i], prefix = key_prefix(key, L);
        // bodies i .. i + cap share the prefix; keys[lo - 1] has it, keys[hi] (if any) has not
        int lo = i + (int)t.cap + 1, hi = t.n;
        while (lo < hi) {
            const int step = (hi - lo + 7) >> 3;
            const int64_t at = lo + (int64_t)c * step;
            const bool same = at < hi && key_prefix(keys[at], L) == prefix;
            const int m = __popc(__ballot_sync(group, same) & group);
            if (m == 0) break;
            hi = (int)min((int64_t)hi, lo + (int64_t)m * step);
            lo += (m - 1) * step + 1;
        }
        const int e = lo;
        const int sh = 3 * (kKeyLevels - 1 - L);
        const int cb = c == 0 ? i : lower_octant(keys, i, e, sh, c);
        __syncwarp(group);
        const int next = __shfl_sync(group, cb, (lane & 24) | ((c + 1) & 7));
        const int ce = c == 7 ? e : next;
        double cx = t.root[0], cy = t.root[1], cz = t.root[2], hw = t.root[3];
        for (int d = 0; d < L; ++d) {
            const int o = (int)((key >> (3 * (kKeyLevels - 1 - d))) & 7);
            hw = dmul(hw, 0.5);
            cx = child_centre(cx, hw, o & 1);
            cy = child_centre(cy, hw, o & 2);
            cz = child_centre(cz, hw, o & 4);
        }
        const double chw = dmul(hw, 0.5);
        const int c0 = t.level_off[L + 1] + 8 * (k - s_start[L]);
        if (c == 0) t.child[sp.y] = c0;
        t.beg[c0 + c] = cb;
        t.end[c0 + c] = ce;
        t.cx[c0 + c] = child_centre(cx, chw, c & 1);
        t.cy[c0 + c] = child_centre(cy, chw, c & 2);
        t.cz[c0 + c] = child_centre(cz, chw, c & 4);
        t.hw[c0 + c] = chw;
    }
}

__global__ void __launch_bounds__(256) gather_perm_kernel(const int32_t* idx_sorted, int32_t* perm, int n) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) perm[i] = idx_sorted[i];
}

// Leaf order: one warp per leaf puts the leaf's bodies in ascending index order (the
// reference's particle_indices order): each body's new place is the number of smaller
// indices in the leaf, written to t.idx and copied back.
__global__ void __launch_bounds__(256) leaf_sort_kernel(const TreeBuildArgs t, int n_nodes) {
    const int w = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (t.hdr[2] != 0 || w >= min(n_nodes, t.hdr[0]) || t.child[w] >= 0) return;
    const int b = t.beg[w], e = t.end[w];
    if (e - b < 2) return;
    for (int i = b + lane; i < e; i += 32) {
        const int v = t.perm[i];
        int r = 0;
        for (int q = b; q < e; ++q) r += t.perm[q] < v;
        t.idx[b + r] = v;
    }
    __syncwarp();
    for (int i = b + lane; i < e; i += 32) t.perm[i] = t.idx[i];
}

__device__ __forceinline__ double node_mass(const double* rec, int k) { return rec[(size_t)k * kFmmRec + kRecMass]; }

// Nodes of the tree: the count on the device when the host did not read it (a.n_nodes is
// then the capacity of the node arrays).
__device__ __forceinline__ int list_nodes(const TreeListArgs& a) {
    if (!a.cnt_nodes) return a.n_nodes;
    return a.cnt_nodes[2] ? 0 : min(a.cnt_nodes[0], a.n_nodes);  // header {nodes, levels, flags}
}

// Node k has mass > 0: from the massive-body counts when given, else from its record.
__device__ __forceinline__ bool node_massive(const TreeListArgs& a, int k) {
    if (a.mprefix) return a.mprefix[a.end[k]] > a.mprefix[a.beg[k]];
    return node_mass(a.rec, k) > 0.0;
}

// mflag[k] = body at tree position k has mass > 0 (k < n), mflag[n] = 0; a mass < 0 or NaN
// (whose node sums the counts cannot stand for) raises the overflow words.
__global__ void __launch_bounds__(256) massive_flags_kernel(const TreeListArgs a, int32_t* mflag) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k > a.n) return;
    if (k == a.n) {
        mflag[k] = 0;
        return;
    }
    const double mk = a.m[a.perm[k]];
    mflag[k] = mk > 0.0 ? 1 : 0;
    if (!(mk >= 0.0)) {
        if (a.overflow) *a.overflow = 1;
        if (a.overflow_sticky) atomicOr(a.overflow_sticky, 3);
    }
}

// Leaves with mass > 0 (the low word of the marks' total).
__device__ __forceinline__ int leaf_count(const TreeListArgs& a) { return *leaf_count_of(a); }

// Marks the body positions of every leaf with mass > 0 (high word) and the first of each (low
// word), eight lanes per node; one scan of both words then gives a leaf's number and its place.
__global__ void __launch_bounds__(256) leaf_mark_kernel(const TreeListArgs a) {
    const int q = blockIdx.x * 256 + threadIdx.x, k = q >> 3;
    if (k >= list_nodes(a) || a.child[k] >= 0 || !node_massive(a, k)) return;
    const int b = a.beg[k], e = a.end[k];
    for (int p = b + (q & 7); p < e; p += 8) a.mark[p] = (1ll << 32) | (p == b ? 1 : 0);
}

// Thread k: leaf k's tables and node k's walk record, and the slot of the body at position k.
// N = 65,536 leaf 64: 18 us with the marks and the scan, against 48 us with a thread per leaf
// copying its bodies, two scans and a pass of its own for the records.
__global__ void __launch_bounds__(256) leaf_emit_kernel(const TreeListArgs a) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k == 0) a.counters->leaves = leaf_count(a);
    if (k < a.n && a.mark[k] != 0) a.leaf_part[(int)(a.place[k] >> 32)] = a.perm[k];
    if (k >= list_nodes(a)) return;
    const int b = a.beg[k], e = a.end[k];
    WalkNode w;
    w.cx = a.cx[k];
    w.cy = a.cy[k];
    w.cz = a.cz[k];
    w.hw = a.hw[k];
    w.child = a.child[k];
    w.count = e - b;
    w.leaf = -1;
    w.mask = 0;
    if (w.child < 0 && node_massive(a, k)) {
        const int64_t at = a.place[b];
        const int o = (int)(at & 0xffffffffll);
        w.leaf = o;
        a.leaf_node[o] = k;
        a.node_leaf[k] = o;
        a.leaf_off[o] = (int)(at >> 32);
        a.leaf_off[o + 1] = (int)(a.place[e] >> 32);
    }
    if (w.child >= 0)
        for (int c = 0; c < 8; ++c) w.mask |= (node_massive(a, w.child + c) ? 1 : 0) << c;
    a.wn[k] = w;
}

// well_separated (fmm_solver.cpp:228-241): 2 (hw_t + hw_s) / dist < theta, dist != 0, with
// the reference's operations.  The reference's quotient is within 1.5 ulp of the exact
// num / sqrt(r2), so wherever (hw_t + hw_s)^2 and theta^2 r2 / 4 (each within a few ulp) differ by
// more than 1e-12 relative the squares give the same answer without the square root and the
// division; only near-ties take the reference's own operations.  So do all nodes of a tree whose
// extent or theta could make the squares overflow or underflow (SeparationTest::squares).
struct SeparationTest {
    double theta, lo, hi;  // theta^2 / 4 times 1 -+ 1e-12
    bool squares;
    __device__ __forceinline__ SeparationTest(double th, double root_hw) : theta(th) {
        const double q = dmul(dmul(th, th), 0.25);
        lo = dmul(q, 1.0 - 1e-12);
        hi = dmul(q, 1.0 + 1e-12);
        // cells are at least root_hw 2^-32 wide (max_depth bounds the tree on the device at 21)
        squares = th > 1e-50 && th < 1e50 && root_hw > 1e-60 && root_hw < 1e60;
    }
    __device__ __forceinline__ bool operator()(const WalkNode& T, const WalkNode& S) const {
        const double dx = dsub(S.cx, T.cx), dy = dsub(S.cy, T.cy), dz = dsub(S.cz, T.cz);
        const double r2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
        const double w = dadd(T.hw, S.hw);
        if (squares) {
            const double w2 = dmul(w, w);
            if (w2 < dmul(lo, r2)) return true;
            if (w2 > dmul(hi, r2)) return false;
        }
        if (r2 == 0.0) return false;  // dist == 0
        return __ddiv_rn(dmul(2.0, w), __dsqrt_rn(r2)) < theta;
    }
};

__device__ __forceinline__ WalkNode load_walk_node(const WalkNode* wn, int s) {
    WalkNode r;
    const double2* q = reinterpret_cast<const double2*>(wn + s);
    const double2 a0 = q[0], a1 = q[1];
    const int4 a2 = *reinterpret_cast<const int4*>(q + 2);
    r.cx = a0.x; r.cy = a0.y; r.cz = a1.x; r.hw = a1.y;
    r.child = a2.x; r.mask = a2.y; r.leaf = a2.z; r.count = a2.w;
    return r;
}

// One warp sorts n <= 32 K distinct values of src (shared memory, any order) ascending into dst,
// by way of the 32 K words of tmp (shared, apart from src): a bitonic network in registers, K
// neighbours per lane, its compare-exchanges across lanes by shuffle.
template <int K>
__device__ __forceinline__ void warp_sort(const uint32_t* src, uint32_t* tmp, int n, int lane, int32_t* dst) {
    uint32_t v[K];
#pragma unroll
    for (int r = 0; r < K; ++r) v[r] = r * 32 + lane < n ? src[r * 32 + lane] : 0xffffffffu;
    auto exchange = [](uint32_t& x, uint32_t& y, bool up) {  // x before y
        const uint32_t lo = min(x, y), hi = max(x, y);
        x = up ? lo : hi;
        y = up ? hi : lo;
    };
    // runs of up to K inside a lane
    if constexpr (K > 1) {
#pragma unroll
        for (int k = 2; k <= K; k <<= 1)
#pragma unroll
            for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
                for (int r = 0; r < K; ++r)
                    if ((r & j) == 0) exchange(v[r], v[r | j], k < K ? (r & k) == 0 : (lane & 1) == 0);
    }
    for (int k = 2; k <= 32; k <<= 1) {  // runs of k lanes
        const bool up = (lane & k) == 0;
        for (int j = k >> 1; j > 0; j >>= 1) {
            const bool low = (lane & j) == 0;
#pragma unroll
            for (int r = 0; r < K; ++r) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, v[r], j);
                v[r] = low == up ? min(v[r], o) : max(v[r], o);
            }
        }
        if constexpr (K > 1) {
#pragma unroll
            for (int j = K >> 1; j > 0; j >>= 1)
#pragma unroll
                for (int r = 0; r < K; ++r)
                    if ((r & j) == 0) exchange(v[r], v[r | j], up);
        }
    }
    if (K == 1) {
        if (lane < n) dst[lane] = (int32_t)v[0];
        return;
    }
#pragma unroll
    for (int r = 0; r < K; ++r) tmp[lane * K + r] = v[r];
    __syncwarp();
    for (int i = lane; i < n; i += 32) dst[i] = (int32_t)tmp[i];
    __syncwarp();
}

// The far list of one leaf in the making (uniform over the warp): chunks are reserved as they are
// needed, the full ones entered as work items.
struct FarChunks {
    int leaf;
    bool wanted;               // the leaf has a target in range
    int64_t chunk = -1;        // current chunk
    int fill = kM2PChunk;      // entries in it (full: the next entry opens a chunk)
    int nch = 0;
    int count = 0;             // entries met

    __device__ __forceinline__ void close(const TreeListArgs& a, int lane) {
        if (chunk < 0) return;
        if (lane == 0 && chunk < a.far_cap) {
            M2PItem it;
            it.leaf = leaf;
            it.chunk = nch;
            it.nchunks = 0;  // entered with the item order, like scratch
            it.count = fill;
            it.fb = chunk * kM2PChunk;
            it.scratch = 0;
            ((M2PItem*)a.items)[chunk] = it;
        }
        ++nch;
    }
    // Lanes of mask m append their node s, in lane order.
    __device__ __forceinline__ void append(const TreeListArgs& a, unsigned m, int lane, int s) {
        if (m == 0) return;
        const int k = __popc(m), pos = fill + __popc(m & ((1u << lane) - 1u));
        count += k;
        if (!wanted) return;
        int64_t next = chunk;
        if (fill + k > kM2PChunk) {
            unsigned long long c = 0;
            if (lane == 0) c = atomicAdd(&a.counters->chunks, 1ull);
            next = (int64_t)__shfl_sync(0xffffffffu, c, 0);
        }
        if (m >> lane & 1u) {
            const int64_t c = pos < kM2PChunk ? chunk : next;
            if (c < a.far_cap) a.far_node[c * kM2PChunk + (pos & (kM2PChunk - 1))] = s;
        }
        if (fill + k > kM2PChunk) {
            const int left = fill + k - kM2PChunk;
            fill = kM2PChunk;
            close(a, lane);
            chunk = next;
            fill = left;
        } else {
            fill += k;
        }
    }
};
static_assert((kM2PChunk & (kM2PChunk - 1)) == 0, "positions wrap by mask");

__device__ __forceinline__ bool leaf_in_range(const TreeListArgs& a, int tb, int te, int lane) {
    if (a.t_begin <= 0 && a.t_end >= a.n) return true;
    bool any = false;
    for (int k = tb + lane; k < te; k += 32) any |= a.leaf_part[k] >= a.t_begin && a.leaf_part[k] < a.t_end;
    return __any_sync(0xffffffffu, any);
}

// Totals a warp has met, added to the counters once at its end.
struct WalkTotals {
    unsigned long long far = 0, far_pairs = 0, near_pairs = 0;
    __device__ __forceinline__ void flush(const TreeListArgs& a, int lane) const {
        if (lane != 0 || far + near_pairs == 0) return;
        atomicAdd(&a.counters->far, far);
        atomicAdd(&a.counters->far_pairs, far_pairs);
        atomicAdd(&a.counters->near_pairs, near_pairs);
    }
};

// The leaf's list sizes, once its far chunks are closed (lane 0); those of slow_walk_kernel's leaves
// carry a minus sign, as its items do: the chunks walk_kernel had begun for such a leaf are void.
__device__ __forceinline__ void leaf_done(const TreeListArgs& a, int l, int targets, int nf, int nch, bool slow, int nsrc,
                                          WalkTotals& tot) {
    a.far_nch[l] = slow ? -nch : nch;
    a.far_slot[l] = nch > 1 ? (int64_t)atomicAdd(&a.counters->slots, (unsigned long long)nch * targets) : 0;
    a.near_src[l] = nsrc;
    tot.far += nf;
    tot.far_pairs += (unsigned long long)nf * targets;
    tot.near_pairs += (unsigned long long)nsrc * targets;
}

// A place for the n near leaves of leaf l (lane 0); past the pool: an empty list.
__device__ __forceinline__ int near_place(const TreeListArgs& a, int l, int n) {
    const unsigned long long b = atomicAdd(&a.counters->near, (unsigned long long)n);
    const bool ok = (int64_t)b + n <= a.near_cap;
    a.near_beg[l] = ok ? (int32_t)b : 0;
    a.near_end[l] = ok ? (int32_t)b + n : 0;
    return ok ? (int)b : -1;
}

// Every leaf with mass > 0, one warp each (leaves taken from a ticket): the walk of
// build_leaf_interactions (fmm_solver.cpp:254-277) from the root, with a shared-memory stack the
// warp pops 32 nodes at a time (each lane classifies one node; expanded nodes push their children
// with mass > 0; the massless ones would be skipped).  Far nodes are written where the walk meets
// them (the far list holds the reference's nodes in the walk's own, deterministic order; only the
// summation order of the far field depends on it).  Near leaves are collected as ordinals, then
// sorted into the reference's depth-first order (leaf ordinals are depth-first numbers), which
// the near field's exact form relies on; a list longer than the buffer goes to linked segments and
// long_near_kernel.  A leaf whose stack would overflow is left to slow_walk_kernel.
// Bound by the latency of a pop (its node records, the test, the pushes) and, for small trees, by
// the few leaves with thousands of nodes to visit.  N = 65,536 leaf 64 86 us, N = 2^20 leaf 16
// 2.2 ms, against 197 us and 5.0 ms for a count and a fill walk with 56-byte records, near lists
// sorted in shared memory and each leaf's totals added by atomics.
__global__ void __launch_bounds__(kWalkThreads, 8) walk_kernel(const TreeListArgs a) {
    constexpr int W = kWalkThreads / 32;
    __shared__ __align__(16) int s_buf[W][kWalkSlots];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_leaves = leaf_count(a);
    const unsigned lt = (1u << lane) - 1u;
    int* const stk = s_buf[wid];
    const SeparationTest separated(a.theta, n_leaves > 0 ? a.hw[0] : 0.0);
    // consecutive leaves share most of their nodes: a warp takes four at a time when there are many
    const int batch = n_leaves > 8 * W * (int)gridDim.x ? 4 : 1;
    WalkTotals tot;
    for (;;) {
        int l0 = 0;
        if (lane == 0) l0 = atomicAdd(&a.counters->ticket, batch);
        l0 = __shfl_sync(0xffffffffu, l0, 0);
        if (l0 >= n_leaves) break;
        for (int l = l0; l < min(l0 + batch, n_leaves); ++l) {
            const int t = a.leaf_node[l];
            const WalkNode T = load_walk_node(a.wn, t);
            const int tb = a.leaf_off[l], te = a.leaf_off[l + 1];
            FarChunks far;
            far.leaf = l;
            far.wanted = leaf_in_range(a, tb, te, lane);
            int nn = 0, nb = 0, head = -1, top = 1;  // near leaves met, of them in the buffer, segments
            int nsrc = 0;  // bodies of the near leaves this lane met
            bool slow = false;
            // the nb near leaves of the buffer into a new segment
            auto flush_near = [&] {
                unsigned long long c = 0;
                if (lane == 0) c = atomicAdd(&a.counters->segs, 1ull);
                const int64_t seg = (int64_t)__shfl_sync(0xffffffffu, c, 0);
                if (seg < a.seg_cap) {
                    for (int i = lane; i < nb; i += 32) a.seg_near[seg * kNearSeg + i] = stk[kWalkSlots - 1 - i];
                    if (lane == 0) {
                        a.seg_next[seg] = head;
                        a.seg_count[seg] = nb;
                    }
                    head = (int)seg;
                }
                __syncwarp();
                nb = 0;
            };
            __syncwarp();
            if (lane == 0) stk[0] = 0;
            __syncwarp();
            while (top > 0) {
                const int take = min(32, top), base = top - take;
                const bool in = lane < take;
                const int s = in ? stk[base + lane] : t;
                const WalkNode S = load_walk_node(a.wn, s);
                const bool is_far = in && s != t && separated(T, S);
                const bool is_near = in && !is_far && S.child < 0;
                const int m = in && !is_far && !is_near ? S.mask : 0;
                const unsigned mf = __ballot_sync(0xffffffffu, is_far);
                const unsigned mn = __ballot_sync(0xffffffffu, is_near);
                far.append(a, mf, lane, s);
                // children to push: prefix sums of the lanes' counts (0..8) from four ballots
                const int mine = __popc(m);
                const unsigned b0 = __ballot_sync(0xffffffffu, mine & 1), b1 = __ballot_sync(0xffffffffu, mine & 2);
                const unsigned b2 = __ballot_sync(0xffffffffu, mine & 4), b3 = __ballot_sync(0xffffffffu, mine & 8);
                const int add = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2) + 8 * __popc(b3);
                const int at = base + __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt) + 8 * __popc(b3 & lt);
                if (base + add > a.walk_stack) {
                    slow = true;
                    break;
                }
                top = base + add;
                const int kn = __popc(mn);
                if (kn > 0 && (nb + kn > kWalkNear || top + nb + kn > kWalkSlots)) flush_near();
                else if (top + nb > kWalkSlots) flush_near();
                if (is_near) {
                    stk[kWalkSlots - 1 - nb - __popc(mn & lt)] = S.leaf;
                    nsrc += S.count;
                }
                nb += kn;
                nn += kn;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (m >> c & 1) stk[at + __popc(m >> (c + 1))] = S.child + c;
                __syncwarp();
            }
            far.close(a, lane);
            if (slow) {
                if (lane == 0) a.slow_leaf[atomicAdd(&a.counters->n_slow, 1)] = l;
                continue;
            }
            const int src = __reduce_add_sync(0xffffffffu, nsrc);
            if (lane == 0) leaf_done(a, l, te - tb, far.count, far.nch, false, src, tot);
            if (nn != nb) {
                if (nb > 0) flush_near();
                if (lane == 0) {
                    const int k = atomicAdd(&a.counters->n_long, 1);
                    a.long_leaf[k] = l;
                    a.long_head[k] = head;
                    a.long_near[k] = nn;
                }
                continue;
            }
            int nbase = 0;
            if (lane == 0) nbase = near_place(a, l, nn);
            nbase = __shfl_sync(0xffffffffu, nbase, 0);
            if (nbase < 0) continue;
            uint32_t* src_buf = reinterpret_cast<uint32_t*>(stk) + kWalkSlots - nn;  // stack is empty
            int32_t* dst = a.near_leaf + nbase;
            uint32_t* tmp = reinterpret_cast<uint32_t*>(stk);
            if (nn <= 32) warp_sort<1>(src_buf, tmp, nn, lane, dst);
            else if (nn <= 64) warp_sort<2>(src_buf, tmp, nn, lane, dst);
            else if (nn <= 128) warp_sort<4>(src_buf, tmp, nn, lane, dst);
            else if (nn <= 256) warp_sort<8>(src_buf, tmp, nn, lane, dst);
            else warp_sort<16>(src_buf, tmp, nn, lane, dst);
        }
    }
    tot.flush(a, lane);
}

// The leaves whose stack overflowed, one warp each, in two passes: the walk as above
// until the stack would overflow, then every lane walks its pending children and its share of the
// stack depth first with a private stack -- once to count, so that the lists' sizes and the lanes'
// places (lanes in order) are known and the order is deterministic, and once to write.
template <bool WRITE>
__device__ void slow_walk(const TreeListArgs& a, const int t, const WalkNode& T, const SeparationTest& separated,
                          int* stk, const int lane, int64_t fbase, int64_t nbase, int& nf, int& nn, int& nsrc) {
    const unsigned lt = (1u << lane) - 1u;
    nf = nn = nsrc = 0;
    int top = 1, pmask = 0, pchild = 0;
    // 1 far, 2 near, 3 expand
    auto classify = [&](int s, const WalkNode& S) { return s != t && separated(T, S) ? 1 : S.child < 0 ? 2 : 3; };
    __syncwarp();
    if (lane == 0) stk[0] = 0;
    __syncwarp();
    while (top > 0) {
        const int take = min(32, top), base = top - take;
        int s = 0, cls = 0;
        WalkNode S = T;
        if (lane < take) {
            s = stk[base + lane];
            S = load_walk_node(a.wn, s);
            cls = classify(s, S);
        }
        const unsigned mf = __ballot_sync(0xffffffffu, cls == 1);
        const unsigned mn = __ballot_sync(0xffffffffu, cls == 2);
        if (WRITE && cls == 1 && fbase >= 0) a.far_node[fbase + nf + __popc(mf & lt)] = s;
        if (cls == 2) {
            if (WRITE) a.seg_near[nbase + nn + __popc(mn & lt)] = S.leaf;
            nsrc += S.count;
        }
        nf += __popc(mf);
        nn += __popc(mn);
        const int m = cls == 3 ? S.mask : 0, mine = __popc(m);
        int at = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += u;
        }
        const int add = __shfl_sync(0xffffffffu, at, 31);
        top = base;
        if (base + add > a.walk_stack) {
            pmask = m;
            pchild = S.child;
            break;
        }
        at += base - mine;
        for (int c = 7; c >= 0; --c)
            if (m >> c & 1) stk[at++] = S.child + c;
        top += add;
        __syncwarp();
    }
    int st[kStack];
    auto lane_walk = [&](bool write, int64_t fpos, int64_t npos, int& lf, int& ln, int& lsrc) {
        lf = ln = lsrc = 0;
        for (int i = lane - 32; i < top; i += 32) {
            int sp = 0;
            if (i < 0) {
                for (int c = 7; c >= 0; --c)
                    if (pmask >> c & 1) st[sp++] = pchild + c;
            } else {
                st[sp++] = stk[i];
            }
            while (sp > 0) {
                const int s = st[--sp];
                const WalkNode S = load_walk_node(a.wn, s);
                const int cls = classify(s, S);
                if (cls == 1) {
                    if (write && fbase >= 0) a.far_node[fpos + lf] = s;
                    ++lf;
                } else if (cls == 2) {
                    if (write) a.seg_near[npos + ln] = S.leaf;
                    ++ln;
                    lsrc += S.count;
                } else {
                    for (int c = 7; c >= 0; --c)
                        if (S.mask >> c & 1) st[sp++] = S.child + c;
                }
            }
        }
    };
    int lf, ln, lsrc;
    lane_walk(false, 0, 0, lf, ln, lsrc);
    nsrc += lsrc;
    int ef = lf, en = ln;  // inclusive prefix sums over the lanes
    for (int o = 1; o < 32; o <<= 1) {
        const int uf = __shfl_up_sync(0xffffffffu, ef, o), un = __shfl_up_sync(0xffffffffu, en, o);
        if (lane >= o) {
            ef += uf;
            en += un;
        }
    }
    if (WRITE) lane_walk(true, fbase + nf + ef - lf, nbase + nn + en - ln, lf, ln, lsrc);
    nf += __shfl_sync(0xffffffffu, ef, 31);
    nn += __shfl_sync(0xffffffffu, en, 31);
}

__global__ void __launch_bounds__(kWalkThreads) slow_walk_kernel(const TreeListArgs a) {
    constexpr int W = kWalkThreads / 32;
    __shared__ int s_stk[W][kWalkStack];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_slow = a.counters->n_slow;
    const SeparationTest separated(a.theta, n_slow > 0 ? a.hw[0] : 0.0);
    WalkTotals tot;
    for (int q = blockIdx.x * W + wid; q < n_slow; q += gridDim.x * W) {
        const int l = a.slow_leaf[q], t = a.leaf_node[l];
        const WalkNode T = load_walk_node(a.wn, t);
        const int tb = a.leaf_off[l], te = a.leaf_off[l + 1];
        int nf, nn, nsrc;
        slow_walk<false>(a, t, T, separated, s_stk[wid], lane, 0, 0, nf, nn, nsrc);
        const int src = __reduce_add_sync(0xffffffffu, nsrc);
        const int nch = leaf_in_range(a, tb, te, lane) ? (nf + kM2PChunk - 1) / kM2PChunk : 0;
        const int ns = (nn + kNearSeg - 1) / kNearSeg;
        unsigned long long c0 = 0, s0 = 0;
        if (lane == 0) {
            c0 = atomicAdd(&a.counters->chunks, (unsigned long long)nch);
            s0 = atomicAdd(&a.counters->segs, (unsigned long long)ns);
            leaf_done(a, l, te - tb, nf, nch, true, src, tot);
        }
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        s0 = __shfl_sync(0xffffffffu, s0, 0);
        if ((int64_t)c0 + nch > a.far_cap || (int64_t)s0 + ns > a.seg_cap) {
            // the totals tell; the reserved chunks that do exist are void
            for (int64_t c = (int64_t)c0 + lane; c < min((int64_t)c0 + nch, a.far_cap); c += 32)
                ((M2PItem*)a.items)[c].leaf = -1;
            continue;
        }
        // a leaf without a target in range keeps no far list (place -1)
        slow_walk<true>(a, t, T, separated, s_stk[wid], lane, nch > 0 ? (int64_t)c0 * kM2PChunk : (int64_t)-1,
                        (int64_t)s0 * kNearSeg, nf, nn, nsrc);
        for (int c = lane; c < nch; c += 32) {
            M2PItem it;
            it.leaf = l;
            it.chunk = c;
            it.nchunks = -1;
            it.count = min(kM2PChunk, nf - c * kM2PChunk);
            it.fb = ((int64_t)c0 + c) * kM2PChunk;
            it.scratch = 0;
            ((M2PItem*)a.items)[c0 + c] = it;
        }
        for (int k = lane; k < ns; k += 32) {
            a.seg_next[s0 + k] = k > 0 ? (int)(s0 + k - 1) : -1;
            a.seg_count[s0 + k] = min(kNearSeg, nn - k * kNearSeg);
        }
        if (lane == 0) {
            const int k = atomicAdd(&a.counters->n_long, 1);
            a.long_leaf[k] = l;
            a.long_head[k] = (int)(s0 + ns - 1);
            a.long_near[k] = nn;
        }
    }
    tot.flush(a, lane);
}

// Near lists that went to segments, one block each: the ordinals set bits in shared memory, and the
// set bits in order are the sorted list (kLongBits leaves per round).  Replaces sorting networks
// in shared memory and ranks by binary search: N = 65,536 leaf 64 (9 lists of 500 to 1200) 11 us, N = 2^20
// leaf 16 (1100 lists) 69 us, against 42 and 310 us.
constexpr int kLongThreads = 512;
constexpr int kLongWords = 8192;
__global__ void __launch_bounds__(kLongThreads) long_near_kernel(const TreeListArgs a) {
    __shared__ unsigned s_bits[kLongWords];
    __shared__ int s_warp[kLongThreads / 32];
    __shared__ int s_base;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int n_long = a.counters->n_long, n_leaves = leaf_count(a);
    if ((int64_t)a.counters->segs > a.seg_cap) return;  // a list is incomplete: the totals tell
    for (int q = blockIdx.x; q < n_long; q += gridDim.x) {
        if (tid == 0) s_base = near_place(a, a.long_leaf[q], a.long_near[q]);
        __syncthreads();
        if (s_base >= 0) {
            int out = s_base;
            for (int r0 = 0; r0 < n_leaves; r0 += 32 * kLongWords) {
                const int words = (min(32 * kLongWords, n_leaves - r0) + 31) / 32;
                const int per = (words + kLongThreads - 1) / kLongThreads;  // consecutive words of a thread
                for (int w = tid; w < words; w += kLongThreads) s_bits[w] = 0;
                __syncthreads();
                for (int seg = a.long_head[q]; seg >= 0; seg = a.seg_next[seg]) {
                    if (tid < a.seg_count[seg]) {
                        const int o = a.seg_near[(int64_t)seg * kNearSeg + tid] - r0;
                        if (o >= 0 && o < 32 * kLongWords) atomicOr(&s_bits[o >> 5], 1u << (o & 31));
                    }
                }
                __syncthreads();
                const int wb = min(tid * per, words), we = min(wb + per, words);
                int mine = 0;
                for (int w = wb; w < we; ++w) mine += __popc(s_bits[w]);
                int incl = mine;
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                if (lane == 31) s_warp[wid] = incl;
                __syncthreads();
                int pos = out + incl - mine, total = 0;
                for (int w = 0; w < kLongThreads / 32; ++w) {
                    if (w < wid) pos += s_warp[w];
                    total += s_warp[w];
                }
                for (int w = wb; w < we; ++w)
                    for (unsigned b = s_bits[w]; b != 0; b &= b - 1) a.near_leaf[pos++] = r0 + 32 * w + __ffs(b) - 1;
                out += total;
                __syncthreads();
            }
        }
        __syncthreads();
    }
}
static_assert(kLongThreads == kNearSeg, "one thread per entry of a segment");

// Far-field items, largest first (cost = targets x nodes): fewer long items at the tail.
// Sort keys: the cost of the real items (n_real of them, from the device count when given) on
// a log scale with four steps per octave (1..127, 7 bits: one radix pass), 0 for the rest of
// the capacity, so that the real items come first, largest first.  The order only balances
// the blocks' work: a leaf's partial sums are added in chunk order whatever it is.
__device__ __forceinline__ bool item_valid(const TreeListArgs& a, const M2PItem& it) {
    return it.leaf >= 0 && (a.far_nch[it.leaf] < 0) == (it.nchunks < 0);
}
__global__ void __launch_bounds__(256) item_cost_kernel(const TreeListArgs a, int n, const unsigned long long* n_real,
                                                        const int* overflow, uint32_t* cost, int32_t* idx) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= n) return;
    const int real = (overflow && *overflow) ? 0 : n_real ? (int)min(*n_real, (unsigned long long)n) : n;
    uint32_t c = 0;
    if (k < real) {
        const M2PItem it = ((const M2PItem*)a.items)[k];
        if (item_valid(a, it)) {
            const uint32_t v = far_item_cost(a.leaf_off[it.leaf + 1] - a.leaf_off[it.leaf], it.count);
            const int msb = 31 - __clz(v);
            c = v < 4u ? v : (uint32_t)(msb * 4 + ((v >> (msb - 2)) & 3));
        }
    }
    cost[k] = c;
    idx[k] = k;
}

// Marks an overflow when a list or item pool reserved by capacity is too small for this
// evaluation's totals, or the topology build could not complete on the device.
__global__ void pool_check_kernel(const TreeListArgs a, const int32_t* tree_hdr) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const ListCounters& t = *a.counters;
    if (a.need) {
        atomicMax(&a.need[0], (unsigned long long)(tree_hdr[0] > 0 ? tree_hdr[0] : 0));
        atomicMax(&a.need[1], t.chunks);
        atomicMax(&a.need[2], t.near);
        atomicMax(&a.need[3], t.slots);
        // levels of the tree; a tree cut short by too few sorted key levels asks for all
        atomicMax(&a.need[4], (unsigned long long)(tree_hdr[2] & 4 ? kKeyLevels : max(tree_hdr[1], 0)));
        atomicMax(&a.need[5], t.segs);
    }
    if (t.chunks > (unsigned long long)a.far_cap || t.near > (unsigned long long)a.near_cap ||
        t.segs > (unsigned long long)a.seg_cap || t.slots > (unsigned long long)a.slot_cap || tree_hdr[2] != 0) {
        *a.overflow = 1;
        if (a.overflow_sticky) atomicOr(a.overflow_sticky, tree_hdr[2] & 1 ? 3 : 1);  // bit 1: too deep
    }
}

__global__ void __launch_bounds__(256) item_gather_kernel(const TreeListArgs a, const int32_t* idx, int n,
                                                          const uint32_t* cost, M2PItem* out) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= n) return;
    M2PItem it;
    it.leaf = -1;
    if (cost ? cost[k] > 0 : item_valid(a, ((const M2PItem*)a.items)[k])) {  // real and valid
        it = ((const M2PItem*)a.items)[cost ? idx[k] : k];
        it.nchunks = abs(a.far_nch[it.leaf]);
        it.scratch = a.far_slot[it.leaf];
    }
    out[k] = it;
}

// One warp per leaf.  With the lists in order on the device the host copies no more than they hold:
// build_leaf_lists with N = 2^20 leaf 16 takes 89 ms, against 219 with the whole pool copied to the host
// and put in order there (N = 65,536 leaf 64 1.05 ms, 1.76).
__global__ void __launch_bounds__(256) near_gather_kernel(int n_leaves, const int32_t* near_beg, const int32_t* near_leaf,
                                                          const int32_t* off, int32_t* out) {
    const int l = (int)((blockIdx.x * 256u + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (l >= n_leaves) return;
    const int32_t* const from = near_leaf + near_beg[l];
    const int o = off[l], cnt = off[l + 1] - o;
    for (int k = lane; k < cnt; k += 32) out[o + k] = from[k];
}

size_t scan_bytes(int count) {
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (const int32_t*)nullptr, (int32_t*)nullptr, count);
    return b;
}

}  // namespace

// Temporary storage of launch_tree_build: ticket and depth starts, each block's first ranks, the
// list of splitting nodes (at most kKeyLevels (n / (cap + 1) + 1): the depth-L prefixes that
// split hold more than cap bodies each and are disjoint), then the radix sort's own storage.
namespace {
int split_capacity(int32_t n, int64_t cap) {
    const int64_t c = (int64_t)kKeyLevels * ((int64_t)n / (std::max<int64_t>(cap, 0) + 1) + 1);
    return (int)std::min<int64_t>(c, 0x7fffffff);
}
}  // namespace

namespace {
size_t aligned(size_t b) { return (b + 255) & ~(size_t)255; }
int topo_blocks(int32_t n) { return (n + kTopoBodies - 1) / kTopoBodies; }
constexpr size_t kTopoHead = 256;  // ticket and kKeyLevels + 1 starts
static_assert((kKeyLevels + 2) * sizeof(int) <= kTopoHead, "head of the build's scratch");
}  // namespace

size_t tree_build_temp_bytes(int32_t n, int64_t cap) {
    size_t b = 0;
    cub::DoubleBuffer<uint64_t> k(nullptr, nullptr);
    cub::DoubleBuffer<int32_t> v(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, b, k, v, n, 0, 3 * kKeyLevels);
    return kTopoHead + aligned((size_t)kKeyLevels * topo_blocks(n) * sizeof(int)) +
           aligned((size_t)split_capacity(n, cap) * sizeof(int2)) + aligned(b);
}

cudaError_t launch_tree_build(const TreeBuildArgs& t, void* temp, size_t temp_bytes, int sms, cudaStream_t st) {
    Topology p;
    p.blocks = topo_blocks(t.n);
    p.split_cap = split_capacity(t.n, t.cap);
    p.ticket = (int*)temp;
    p.start = p.ticket + 1;
    const size_t firsts = aligned((size_t)kKeyLevels * p.blocks * sizeof(int));
    p.first = (int*)((char*)temp + kTopoHead);
    p.split = (int2*)((char*)temp + kTopoHead + firsts);
    const size_t used = kTopoHead + firsts + aligned((size_t)p.split_cap * sizeof(int2));
    void* work = (char*)temp + used;
    size_t work_bytes = temp_bytes - used;
    const int gn = (t.n + kBboxThreads - 1) / kBboxThreads;
    const int bbox_blocks = std::min(gn, kBboxBlocks);
    bbox_partial_kernel<<<bbox_blocks, kBboxThreads, 0, st>>>(t);
    keys_kernel<<<std::min(gn, sms * 8), kBboxThreads, 0, st>>>(t, bbox_blocks, p.ticket);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cub::DoubleBuffer<uint64_t> k(t.keys, t.keys_alt);
    cub::DoubleBuffer<int32_t> v(t.idx, t.perm);
    const int sorted = t.key_levels > 0 ? std::min(t.key_levels, kKeyLevels) : kKeyLevels;
    if ((e = cub::DeviceRadixSort::SortPairs(work, work_bytes, k, v, t.n, 3 * (kKeyLevels - sorted), 3 * kKeyLevels,
                                             st)) != cudaSuccess)
        return e;
    if (v.Current() != t.perm) gather_perm_kernel<<<(t.n + 255) / 256, 256, 0, st>>>(v.Current(), t.perm, t.n);
    split_count_kernel<<<p.blocks, kTopoThreads, 0, st>>>(t, k.Current(), p);
    split_emit_kernel<<<p.blocks, kTopoThreads, 0, st>>>(t, k.Current(), p);
    tree_children_kernel<<<sms * 8, 256, 0, st>>>(t, k.Current(), p);
    return cudaGetLastError();
}

cudaError_t launch_tree_leaf_order(const TreeBuildArgs& t, int32_t n_nodes, void* temp, size_t temp_bytes,
                                   cudaStream_t st) {
    (void)temp;
    (void)temp_bytes;
    leaf_sort_kernel<<<(n_nodes + 7) / 8, 256, 0, st>>>(t, n_nodes);
    return cudaGetLastError();
}

size_t tree_list_temp_bytes(int32_t n, int32_t n_nodes) {
    (void)n_nodes;
    size_t b = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, b, (const int64_t*)nullptr, (int64_t*)nullptr, n + 1);
    return std::max(b, scan_bytes(n + 1));
}

// The walk prefers a 70% shared-memory carveout (8 blocks of 19 KiB; the rest is L1): a setting of
// the current device's copy of the kernel.
static cudaError_t walk_carveout() {
    static std::atomic<unsigned long long> set_on{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (set_on.load() & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(walk_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 70);
    if (e == cudaSuccess) set_on.fetch_or(bit);
    return e;
}

cudaError_t launch_tree_lists(const TreeListArgs& a, void* temp, size_t temp_bytes, int sms, cudaStream_t st) {
    cudaError_t e;
    if ((e = cudaMemsetAsync(a.mark, 0, (size_t)(a.n + 1) * sizeof(int64_t), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.counters, 0, sizeof(ListCounters), st)) != cudaSuccess) return e;
    leaf_mark_kernel<<<(unsigned)((8 * (int64_t)a.n_nodes + 255) / 256), 256, 0, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    size_t tb = temp_bytes;
    if ((e = cub::DeviceScan::ExclusiveSum(temp, tb, a.mark, a.place, a.n + 1, st)) != cudaSuccess) return e;
    leaf_emit_kernel<<<(std::max(a.n_nodes, a.n) + 255) / 256, 256, 0, st>>>(a);
    if ((e = walk_carveout()) != cudaSuccess) return e;
    constexpr int W = kWalkThreads / 32;
    walk_kernel<<<std::min((a.n_nodes + W - 1) / W, sms * 8), kWalkThreads, 0, st>>>(a);
    slow_walk_kernel<<<sms, kWalkThreads, 0, st>>>(a);
    long_near_kernel<<<sms * 4, kLongThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_near_gather(int32_t n_leaves, const int32_t* near_beg, const int32_t* near_leaf, const int32_t* off,
                               int32_t* out, cudaStream_t st) {
    if (n_leaves <= 0) return cudaSuccess;
    near_gather_kernel<<<(n_leaves + 7) / 8, 256, 0, st>>>(n_leaves, near_beg, near_leaf, off, out);
    return cudaGetLastError();
}

cudaError_t launch_tree_massive(const TreeListArgs& a, void* temp, size_t temp_bytes, cudaStream_t st) {
    // the flags go to mark (free until the list pass clears it), the counts to mprefix
    massive_flags_kernel<<<(a.n + 256) / 256, 256, 0, st>>>(a, (int32_t*)a.mark);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    size_t tb = temp_bytes;
    return cub::DeviceScan::ExclusiveSum(temp, tb, (const int32_t*)a.mark, a.mprefix, a.n + 1, st);
}

cudaError_t launch_pool_check(const TreeListArgs& a, const int32_t* tree_hdr, cudaStream_t st) {
    pool_check_kernel<<<1, 32, 0, st>>>(a, tree_hdr);
    return cudaGetLastError();
}

size_t item_order_temp_bytes(int32_t n_items) {
    size_t b = 0;
    cub::DoubleBuffer<uint32_t> k(nullptr, nullptr);
    cub::DoubleBuffer<int32_t> v(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairsDescending(nullptr, b, k, v, n_items);
    return b;
}

cudaError_t launch_item_order(const TreeListArgs& a, int32_t n_items, const unsigned long long* n_real,
                              const int* overflow, uint32_t* cost, uint32_t* cost_alt, int32_t* idx, int32_t* idx_alt,
                              void* temp, size_t temp_bytes, M2PItem* out, int sms, cudaStream_t st) {
    if (n_items == 0) return cudaSuccess;
    const int g = (n_items + 255) / 256;
    // Items that are all resident at once (M2P runs at least four blocks per SM) need no order: at
    // N = 1000 the costs and the sort take two launches, 10 of 176 us of device time.
    if (!n_real && n_items <= sms * 4) {
        item_gather_kernel<<<g, 256, 0, st>>>(a, nullptr, n_items, nullptr, out);
        return cudaGetLastError();
    }
    item_cost_kernel<<<g, 256, 0, st>>>(a, n_items, n_real, overflow, cost, idx);
    cub::DoubleBuffer<uint32_t> k(cost, cost_alt);
    cub::DoubleBuffer<int32_t> v(idx, idx_alt);
    cudaError_t e = cub::DeviceRadixSort::SortPairsDescending(temp, temp_bytes, k, v, n_items, 0, 7, st);
    if (e != cudaSuccess) return e;
    item_gather_kernel<<<g, 256, 0, st>>>(a, v.Current(), n_items, k.Current(), out);
    return cudaGetLastError();
}

}  // namespace gx
