// A mesh's bottom-level tree rebuilt on the device from new vertex positions: the binned surface-area-
// heuristic build of src/bvh.cpp:46-174 (16 bins, leaves of at most 4 triangles, depth at most 60) and the
// packing of src/mesh_build.cpp:91-157, giving the host build's tree node for node, its triangles in the
// same leaf order and the same bits.
//
// The host builds depth first from a stack; here the nodes of one depth are split together, one CTA per
// node, level after level, and the host's node numbering is restored at the end:
//   - a node's box, centroid box and bin boxes are min/max reductions. The host's sequential std::min keeps
//     the first of equal values, which matters only for -0 and +0; every reduction here carries the range
//     position of its value and keeps the smallest position among equal values, so the bits are the host's;
//   - std::partition (libstdc++'s bidirectional form) swaps the k-th element from the left that fails the
//     test with the k-th element from the right that passes it, until the two meet: the same swaps are made
//     here from two prefix counts, in parallel;
//   - the host gives a node's two children the indices 2k + 1 and 2k + 2 when it splits the k-th internal
//     node in depth-first, left-first order. An internal node X is preceded in that order by every internal
//     node that starts (in the leaf order) before X does, and by the internal nodes that start where X starts
//     and lie above it (a chain of left children at consecutive depths), so its rank is a prefix count over
//     the start positions plus its depth below the chain's top, with no walk over the tree.
// Node and tree sizes: a tree over T triangles has at most 2T - 1 nodes, numbered in scratch arrays of
// 2T - 1 in level order. The whole build is one cooperative launch: the CTAs (a CTA per large node, a warp per
// small one) split one depth, meet at a grid-wide barrier, and go on to the next depth, whose nodes the splits
// appended after the depth's last node; then the numbering and the packing, between further barriers.
#include <climits>
#include <cstdint>

#include <cooperative_groups.h>

#include "kernels.h"

namespace ngb {
namespace {

constexpr int BINS = 16;
constexpr int MAX_LEAF = 4;
constexpr int MAX_DEPTH = 60;
constexpr int BUILD_THREADS = 512;  // per CTA
constexpr int LARGE_NODE = 256;     // nodes above this are split by a CTA, the others by a warp
constexpr unsigned FULL = 0xffffffffu;

// A float as an int ordered like it, -0 and +0 as one value.
__device__ __forceinline__ int order_of(float v) { return to_ordered(v == 0.0f ? 0.0f : v); }

// The host's box arithmetic (bvh::grow with std::min / std::max, bvh::surface_area).
struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ float area(const Box &b) {
    const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    if (dx < 0.0f || dy < 0.0f || dz < 0.0f) return 0.0f;
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}

// Bins per length, finite also for extents below 16 / FLT_MAX (as the host build's).
__device__ __forceinline__ float bin_scale(float extent) { return fminf(static_cast<float>(BINS) / extent, 3.402823466e38f); }

__device__ __forceinline__ int bin_of(float c, float lo, float scale) {
    const int b = static_cast<int>((c - lo) * scale);
    return b < 0 ? 0 : b < BINS - 1 ? b : BINS - 1;  // (never below 0 for finite vertices)
}

// Triangle boxes (the vertices' std::fmin / std::fmax in vertex order, src/mesh_build.cpp, as the host build
// computes them: of two equal values, -0 and +0, the later one) and centroids (0.5 (lo + hi),
// src/bvh.cpp:55-56); the order starts as the identity and the root spans every triangle.
__device__ void prepare_item(const MeshBuildArgs &a, const MeshBuildScratch &t, int i) {
    t.starts[i] = 0;
    t.top[i] = INT_MAX;
    const float inf = __int_as_float(0x7f800000);
    Box b{{inf, inf, inf}, {-inf, -inf, -inf}};
    for (int k = 0; k < 3; ++k) {
        const float *v = a.vertices + 3 * static_cast<size_t>(__ldg(a.indices + 3 * static_cast<size_t>(i) + k));
        for (int c = 0; c < 3; ++c) {
            const float x = __ldg(v + c);
            b.lo[c] = b.lo[c] < x ? b.lo[c] : x;
            b.hi[c] = b.hi[c] > x ? b.hi[c] : x;
        }
    }
    for (int c = 0; c < 3; ++c) {
        t.box[6 * static_cast<size_t>(i) + c] = b.lo[c];
        t.box[6 * static_cast<size_t>(i) + 3 + c] = b.hi[c];
        t.centre[3 * static_cast<size_t>(i) + c] = 0.5f * (b.lo[c] + b.hi[c]);
    }
    t.order[i] = static_cast<uint32_t>(i);
}

template <int WARPS>
struct SplitSmem {
    int bound[12];               // node box lo/hi (6), centroid box lo/hi (6), as ordered ints
    int bin_bound[3][BINS][6];   // per axis and bin: its box lo/hi, as ordered ints
    int bin_count[3][BINS];
    int zero_at[6];              // node box bounds that are zero: the first range position that holds them
    int warp_sum[WARPS];
    int best_axis, best_bin;
    float best_cost;
    int item_at[64];             // a warp's swap: the lanes of the k-th failing and the k-th passing item
};

// A barrier over the threads that split one node: the CTA, or one warp.
template <int WARPS>
__device__ __forceinline__ void group_sync() {
    if constexpr (WARPS == 1) __syncwarp();
    else __syncthreads();
}

// Exclusive prefix sum of v over the group's threads (gtid: the thread's place in the group; in thread order,
// or from the last thread down when reverse), and the group's total.
template <int WARPS>
__device__ __forceinline__ int cta_scan(SplitSmem<WARPS> &sm, int v, bool reverse, int &total, int gtid) {
    const int lane = gtid & 31, warp = gtid >> 5;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = reverse ? __shfl_down_sync(FULL, incl, o) : __shfl_up_sync(FULL, incl, o);
        if (reverse ? lane + o < 32 : lane >= o) incl += u;
    }
    if (reverse ? lane == 0 : lane == 31) sm.warp_sum[warp] = incl;
    group_sync<WARPS>();
    int before = 0;
    total = 0;
    for (int w = 0; w < WARPS; ++w) {
        before += (reverse ? w > warp : w < warp) ? sm.warp_sum[w] : 0;
        total += sm.warp_sum[w];
    }
    group_sync<WARPS>();
    return before + incl - v;
}

// The cheapest split plane over a node's bins, the axes in order, the first of equally cheap ones (src/bvh.cpp:108-125),
// by one warp: a half warp per axis with a lane per bin, prefix and suffix boxes by shuffles (min and max in any order
// give the host's boxes but for the sign of a zero, which no area shows).
template <int WARPS>
__device__ __forceinline__ void sweep_bins(SplitSmem<WARPS> &sm, const float *cb, int lane) {
    constexpr unsigned NONE = 0xffffffffu;
    unsigned best = NONE;
    int best_axis = -1, best_bin = 0;
    for (int round = 0; round < 2; ++round) {
        const int axis = round == 0 ? lane >> 4 : 2, b = lane & 15;
        int lo[3], hi[3], n = sm.bin_count[axis][b];
        for (int c = 0; c < 3; ++c) {
            lo[c] = sm.bin_bound[axis][b][c];
            hi[c] = sm.bin_bound[axis][b][3 + c];
        }
        int slo[3] = {lo[0], lo[1], lo[2]}, shi[3] = {hi[0], hi[1], hi[2]}, sn = n;
        for (int off = 1; off < BINS; off <<= 1) {
            const bool up = b >= off, down = b + off < BINS;
            for (int c = 0; c < 3; ++c) {
                const int l = __shfl_up_sync(FULL, lo[c], off, BINS), h = __shfl_up_sync(FULL, hi[c], off, BINS);
                if (up) {
                    lo[c] = min(lo[c], l);
                    hi[c] = max(hi[c], h);
                }
                const int sl = __shfl_down_sync(FULL, slo[c], off, BINS), sh = __shfl_down_sync(FULL, shi[c], off, BINS);
                if (down) {
                    slo[c] = min(slo[c], sl);
                    shi[c] = max(shi[c], sh);
                }
            }
            const int k = __shfl_up_sync(FULL, n, off, BINS), q = __shfl_down_sync(FULL, sn, off, BINS);
            if (up) n += k;
            if (down) sn += q;
        }
        Box left, right;
        for (int c = 0; c < 3; ++c) {
            left.lo[c] = from_ordered(lo[c]);
            left.hi[c] = from_ordered(hi[c]);
            right.lo[c] = from_ordered(slo[c]);
            right.hi[c] = from_ordered(shi[c]);
        }
        const float right_area = __shfl_down_sync(FULL, area(right), 1, BINS);
        const int right_count = __shfl_down_sync(FULL, sn, 1, BINS);
        unsigned key = NONE;
        if (b < BINS - 1 && (round == 0 || lane < BINS) && cb[3 + axis] - cb[axis] > 0.0f && n != 0 && right_count != 0) {
            const float cost = static_cast<float>(n) * area(left) + static_cast<float>(right_count) * right_area;
            if (cost < __int_as_float(0x7f800000)) key = __float_as_uint(cost);  // never negative: ordered as an integer
        }
        const unsigned least = __reduce_min_sync(FULL, key);
        if (least < best) {
            const int at = __ffs(__ballot_sync(FULL, key == least)) - 1;
            best = least;
            best_axis = round == 0 ? at >> 4 : 2;
            best_bin = at & 15;
        }
    }
    if (lane == 0) {
        sm.best_axis = best_axis;
        sm.best_bin = best_bin;
        sm.best_cost = best == NONE ? __int_as_float(0x7f800000) : __uint_as_float(best);
    }
}

// Splits node x at this depth with a group of THREADS threads (tid: the thread's place in the group): a CTA for large
// nodes, one warp for small ones. Its children, if any, take the next two places after next_first (the next depth's
// first node) counted by next.nodes, and are listed for the next depth by size.
// What bounds a depth is this chain of dependent steps, not work: reductions are one instruction per bound over a warp
// (redux on ordered ints, where (value, position) pairs took ten shuffles each), bins are 32-bit shared atomics, and the
// sweep over the bins is a scan by lanes (one thread swept the 3 x 16 bins both ways before): a depth of small nodes
// 17 -> 6 us, a rebuild 0.66 -> 0.25 ms for 5,120 triangles and 1.45 -> 0.56 ms for 20,480 (update_mesh, B200).
template <int THREADS>
__device__ void split_node(const MeshBuildArgs &a, const MeshBuildScratch &t, int x, int depth, SplitSmem<THREADS / 32> &sm,
    int tid, int next_first, int *next) {
    constexpr int WARPS = THREADS / 32;
    const int lane = tid & 31;
    const int begin = t.begin[x], end = t.end[x], count = end - begin;
    if (tid == 0) t.depth[x] = depth;
    for (int k = tid; k < 12; k += THREADS) sm.bound[k] = (k % 6) < 3 ? INT_MAX : INT_MIN;
    // An empty bin is the empty box, +inf to -inf.
    const int pos_inf = to_ordered(__int_as_float(0x7f800000)), neg_inf = to_ordered(-__int_as_float(0x7f800000));
    for (int k = tid; k < 3 * BINS * 6; k += THREADS) (&sm.bin_bound[0][0][0])[k] = (k % 6) < 3 ? pos_inf : neg_inf;
    for (int k = tid; k < 3 * BINS; k += THREADS) (&sm.bin_count[0][0])[k] = 0;
    if (tid < 6) sm.zero_at[tid] = INT_MAX;
    group_sync<WARPS>();

    // The node's box and centroid box.
    {
        int b[12];
        for (int k = 0; k < 12; ++k) b[k] = (k % 6) < 3 ? INT_MAX : INT_MIN;
        for (int i = begin + tid; i < end; i += THREADS) {
            const size_t p = t.order[i];
            for (int c = 0; c < 3; ++c) {
                b[c] = min(b[c], order_of(t.box[6 * p + c]));
                b[3 + c] = max(b[3 + c], order_of(t.box[6 * p + 3 + c]));
                const int m = order_of(t.centre[3 * p + c]);
                b[6 + c] = min(b[6 + c], m);
                b[9 + c] = max(b[9 + c], m);
            }
        }
        for (int k = 0; k < 12; ++k) {
            const int v = (k % 6) < 3 ? __reduce_min_sync(FULL, b[k]) : __reduce_max_sync(FULL, b[k]);
            if (lane == 0) {
                if (WARPS == 1) sm.bound[k] = v;
                else if ((k % 6) < 3) atomicMin(&sm.bound[k], v);
                else atomicMax(&sm.bound[k], v);
            }
        }
    }
    group_sync<WARPS>();
    Box box;
    float cb[6];
    bool zero = false;
    for (int k = 0; k < 3; ++k) {
        box.lo[k] = from_ordered(sm.bound[k]);
        box.hi[k] = from_ordered(sm.bound[3 + k]);
        cb[k] = from_ordered(sm.bound[6 + k]);
        cb[3 + k] = from_ordered(sm.bound[9 + k]);
        zero = zero || box.lo[k] == 0.0f || box.hi[k] == 0.0f;
    }
    // A box bound that is a zero has the sign of the first one in range order (the host's std::min and std::max keep
    // the first of equal values).
    if (zero) {
        for (int i = begin + tid; i < end; i += THREADS) {
            const size_t p = t.order[i];
            for (int c = 0; c < 6; ++c)
                if (t.box[6 * p + c] == 0.0f && (c < 3 ? box.lo[c] : box.hi[c - 3]) == 0.0f) atomicMin(&sm.zero_at[c], i);
        }
        group_sync<WARPS>();
        for (int c = 0; c < 6; ++c) {
            float &v = c < 3 ? box.lo[c] : box.hi[c - 3];
            if (v == 0.0f && sm.zero_at[c] != INT_MAX) v = t.box[6 * static_cast<size_t>(t.order[sm.zero_at[c]]) + c];
        }
    }

    // Bins on every axis whose centroids spread (src/bvh.cpp:94-107).
    int best_axis = -1, best_bin = 0;
    float best_cost = __int_as_float(0x7f800000);
    if (count > 1) {
        float scale[3];
        for (int axis = 0; axis < 3; ++axis) scale[axis] = bin_scale(cb[3 + axis] - cb[axis]);
        for (int i = begin + tid; i < end; i += THREADS) {
            const size_t p = t.order[i];
            int b[6];
            for (int c = 0; c < 6; ++c) b[c] = order_of(t.box[6 * p + c]);
            for (int axis = 0; axis < 3; ++axis) {
                if (!(cb[3 + axis] - cb[axis] > 0.0f)) continue;
                const int bin = bin_of(t.centre[3 * p + axis], cb[axis], scale[axis]);
                atomicAdd(&sm.bin_count[axis][bin], 1);
                int *slot = sm.bin_bound[axis][bin];
                // A bound only moves one way, so a value that does not beat it now never will: most are dropped by a
                // plain read instead of a contended atomic.
                for (int c = 0; c < 3; ++c) {
                    if (b[c] < *reinterpret_cast<volatile int *>(slot + c)) atomicMin(slot + c, b[c]);
                    if (b[3 + c] > *reinterpret_cast<volatile int *>(slot + 3 + c)) atomicMax(slot + 3 + c, b[3 + c]);
                }
            }
        }
        group_sync<WARPS>();
        if (tid < 32) sweep_bins<WARPS>(sm, cb, lane);
        group_sync<WARPS>();
        best_axis = sm.best_axis;
        best_bin = sm.best_bin;
        best_cost = sm.best_cost;
    }
    // The leaf test (src/bvh.cpp:126-146).
    const float leaf_cost = static_cast<float>(count) * area(box);
    const float split_cost = 1.0f * area(box) + best_cost;
    const bool leaf = count == 1 || depth >= MAX_DEPTH || (count <= MAX_LEAF && (best_axis < 0 || leaf_cost <= split_cost));
    if (tid == 0)
        for (int c = 0; c < 6; ++c) t.node_box[6 * static_cast<size_t>(x) + c] = c < 3 ? box.lo[c] : box.hi[c - 3];
    if (leaf) {
        if (tid == 0) t.left[x] = -1;
        group_sync<WARPS>();
        return;
    }

    // std::partition over the range by (bin <= best_bin): the k-th failing element from the left swaps with the k-th
    // passing element from the right, for every k before the two runs meet.
    int mid = begin + count / 2;
    if (best_axis >= 0) {
        const float lo = cb[best_axis];
        const float scale = bin_scale(cb[3 + best_axis] - lo);
        auto passes_item = [&](uint32_t p) {
            return bin_of(t.centre[3 * static_cast<size_t>(p) + best_axis], lo, scale) <= best_bin;
        };
        if (WARPS == 1 && count <= 32) {
            // A lane per item: the ranks from ballots, the partners' lanes through shared memory.
            const bool in = lane < count;
            const uint32_t item = in ? t.order[begin + lane] : 0u;
            const bool pass = in && passes_item(item);
            const unsigned mask = __ballot_sync(FULL, pass);
            const int passing = __popc(mask);
            const unsigned left = passing == 32 ? FULL : (1u << passing) - 1u;
            const unsigned fails = ~mask & left, moves = mask & ~left;  // equally many
            const bool failing = fails >> lane & 1u, moving = moves >> lane & 1u;
            const int k = failing ? __popc(fails & ((1u << lane) - 1u)) : __popc(moves & ~((2u << lane) - 1u));
            if (failing) sm.item_at[k] = lane;
            if (moving) sm.item_at[32 + k] = lane;
            __syncwarp();
            const int partner = failing ? sm.item_at[32 + k] : moving ? sm.item_at[k] : lane;
            const uint32_t now = __shfl_sync(FULL, item, partner);
            if (failing || moving) t.order[begin + lane] = now;
            mid = begin + passing;
        } else {
            auto passes = [&](int i) { return passes_item(t.order[i]); };
            // Each thread takes a contiguous run of the range: it counts, the group scans the counts, and it writes its
            // run's positions in order.
            const int run = (count + THREADS - 1) / THREADS;
            const int r0 = begin + tid * run < end ? begin + tid * run : end;
            const int r1 = r0 + run < end ? r0 + run : end;
            int mine = 0;
            for (int i = r0; i < r1; ++i) mine += passes(i) ? 1 : 0;
            int passing;
            cta_scan(sm, mine, false, passing, tid);
            const int meet = begin + passing;
            // Failing elements left of meet, ranked from the left; passing ones right of it, from the right.
            const int l1 = r1 < meet ? r1 : meet, q0 = r0 > meet ? r0 : meet;
            int fails = 0, passes_right = 0;
            for (int i = r0; i < l1; ++i) fails += passes(i) ? 0 : 1;
            for (int j = q0; j < r1; ++j) passes_right += passes(j) ? 1 : 0;
            int swaps, found;
            const int lbase = cta_scan(sm, fails, false, swaps, tid);
            const int rbase = cta_scan(sm, passes_right, true, found, tid);
            for (int i = r0, k = lbase; i < l1; ++i)
                if (!passes(i)) t.lpos[begin + k++] = i;
            for (int j = r1 - 1, k = rbase; j >= q0; --j)
                if (passes(j)) t.rpos[begin + k++] = j;
            group_sync<WARPS>();
            for (int k = tid; k < swaps; k += THREADS) {
                const int l = t.lpos[begin + k], r = t.rpos[begin + k];
                const uint32_t pl = t.order[l];
                t.order[l] = t.order[r];
                t.order[r] = pl;
            }
            mid = meet;
        }
        if (mid == begin || mid == end) mid = begin + count / 2;
    }
    if (tid == 0) {
        const int c = next_first + atomicAdd(next, 2);
        t.left[x] = c;
        t.begin[c] = begin;
        t.end[c] = mid;
        t.begin[c + 1] = mid;
        t.end[c + 1] = end;
        for (int k = 0; k < 2; ++k) {
            const bool large = (k == 0 ? mid - begin : end - mid) > LARGE_NODE;
            int *list = large ? t.large : t.small;
            list[atomicAdd(next + (large ? 1 : 2), 1)] = c + k;
        }
    }
    group_sync<WARPS>();
}

// The packed tree (src/mesh_build.cpp:91-157): bvh::Node records with global indices, and the child-pair
// records of the internal nodes.
__device__ void write_node(const MeshBuildArgs &a, const MeshBuildScratch &t, int x) {
    const int i = t.index[x];
    const float *b = t.node_box + 6 * static_cast<size_t>(x);
    const int l = t.left[x];
    float4 *node = a.blas + 2 * (static_cast<size_t>(a.node_base) + i);
    float4 *pair = a.pairs + 4 * (static_cast<size_t>(a.node_base) + i);
    if (l < 0) {
        node[0] = make_float4(b[0], b[1], b[2], __int_as_float(a.tri_base + t.begin[x]));
        node[1] = make_float4(b[3], b[4], b[5], __int_as_float(t.end[x] - t.begin[x]));
        const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        pair[0] = pair[1] = pair[2] = pair[3] = z;
        return;
    }
    node[0] = make_float4(b[0], b[1], b[2], __int_as_float(a.node_base + t.index[l]));
    node[1] = make_float4(b[3], b[4], b[5], __int_as_float(0));
    const float *lb = t.node_box + 6 * static_cast<size_t>(l), *rb = t.node_box + 6 * static_cast<size_t>(l + 1);
    int ref[4];
    for (int c = 0; c < 2; ++c) {
        const int y = l + c;
        const bool y_leaf = t.left[y] < 0;
        ref[2 * c] = y_leaf ? a.tri_base + t.begin[y] : a.node_base + t.index[y];
        ref[2 * c + 1] = y_leaf ? t.end[y] - t.begin[y] : 0;
    }
    pair[0] = make_float4(lb[0], lb[1], lb[2], lb[3]);
    pair[1] = make_float4(lb[4], lb[5], rb[0], rb[1]);
    pair[2] = make_float4(rb[2], rb[3], rb[4], rb[5]);
    pair[3] = make_float4(__int_as_float(ref[0]), __int_as_float(ref[1]), __int_as_float(ref[2]), __int_as_float(ref[3]));
}

// Triangles in leaf order (v0, e1 = v1 - v0, e2 = v2 - v0), their mesh indices both ways, and their vertex
// normals (ATTR_NORMALS, src/mesh_build.h:28) where the scene keeps them.
__device__ void write_triangle(const MeshBuildArgs &a, const MeshBuildScratch &t, int p) {
    const uint32_t tri = t.order[p];
    const size_t packed = static_cast<size_t>(a.tri_base) + p;
    float3 v[3];
    for (int k = 0; k < 3; ++k) {
        const float *q = a.vertices + 3 * static_cast<size_t>(__ldg(a.indices + 3 * static_cast<size_t>(tri) + k));
        v[k] = make_float3(__ldg(q), __ldg(q + 1), __ldg(q + 2));
    }
    a.tris[3 * packed] = make_float4(v[0].x, v[0].y, v[0].z, 0.0f);
    a.tris[3 * packed + 1] = make_float4(v[1].x - v[0].x, v[1].y - v[0].y, v[1].z - v[0].z, 0.0f);
    a.tris[3 * packed + 2] = make_float4(v[2].x - v[0].x, v[2].y - v[0].y, v[2].z - v[0].z, 0.0f);
    a.tri_index[packed] = static_cast<int>(tri);
    a.tri_of_local[static_cast<size_t>(a.tri_base) + tri] = static_cast<int>(packed);
    if (!a.attrs) return;
    float rec[16] = {};
    if (a.normals)
        for (int k = 0; k < 3; ++k) {
            const float *q = a.normals + 3 * static_cast<size_t>(__ldg(a.indices + 3 * static_cast<size_t>(tri) + k));
            rec[4 * k] = __ldg(q);
            rec[4 * k + 1] = __ldg(q + 1);
            rec[4 * k + 2] = __ldg(q + 2);
        }
    rec[15] = __int_as_float(a.normals ? 1 : 0);
    for (int k = 0; k < 4; ++k) a.attrs[4 * packed + k] = make_float4(rec[4 * k], rec[4 * k + 1], rec[4 * k + 2], rec[4 * k + 3]);
}

// The slots of this mesh: their root reference, their box in mesh space, and no convexity claim (the new
// shape is not checked).
__device__ void write_slot(const MeshBuildArgs &a, const MeshBuildScratch &t, const int *slot_mesh, int mesh,
    int2 *slot_root, float *slot_bounds, float4 *slot_hull, int s) {
    if (slot_mesh[s] != mesh) return;
    const bool leaf = t.left[0] < 0;
    slot_root[s] = leaf ? make_int2(a.tri_base, a.triangles) : make_int2(a.node_base, 0);
    for (int c = 0; c < 6; ++c) slot_bounds[6 * static_cast<size_t>(s) + c] = t.node_box[c];
    slot_hull[s].w = -1.0f;
}

// The whole build, one cooperative launch; grid-wide barriers between its phases. A depth's counts (level_count, three per
// depth) are its nodes, and the places that its large and small nodes end at in their lists (t.large, t.small: every
// depth's after the ones before).
__global__ void __launch_bounds__(BUILD_THREADS, 1) build_mesh_kernel(const MeshBuildArgs a, const MeshBuildScratch t,
    const int *slot_mesh, int slots, int mesh, int2 *slot_root, float *slot_bounds, float4 *slot_hull) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    constexpr int WARPS = BUILD_THREADS / 32;
    __shared__ union {
        SplitSmem<WARPS> cta;
        SplitSmem<1> warp[WARPS];
    } smem;
    __shared__ int prefix_warp[WARPS];
    const long long rank = grid.thread_rank(), size = grid.size();
    const int T = a.triangles;
    const long long cap = 2LL * T - 1;

    // The mesh's whole node run cleared, the triangles' boxes, the root spanning every triangle.
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (long long k = rank; k < 2 * cap; k += size) a.blas[2LL * a.node_base + k] = zero;
    for (long long k = rank; k < 4 * cap; k += size) a.pairs[4LL * a.node_base + k] = zero;
    for (long long i = rank; i < T; i += size) prepare_item(a, t, static_cast<int>(i));
    for (long long d = rank; d < 3 * (MESH_LEVELS + 1); d += size) t.level_count[d] = 0;
    if (rank == 0) {
        t.begin[0] = 0;
        t.end[0] = T;
        t.index[0] = 0;
    }
    grid.sync();

    // Depth after depth: the splits of depth d append depth d + 1's nodes after depth d's last, and list them by size.
    // A depth's lists start where the one before ended: list positions are counted from there.
    int first = 0, last = 1, large0 = 0, large1 = T > LARGE_NODE ? 1 : 0, small0 = 0, small1 = 1 - large1;
    for (int depth = 0; depth < MESH_LEVELS && first < last; ++depth) {
        int *next = t.level_count + 3 * (depth + 1);
        MeshBuildScratch u = t;
        u.large = t.large + large1;
        u.small = t.small + small1;
        for (int k = large0 + blockIdx.x; k < large1; k += gridDim.x)
            split_node<BUILD_THREADS>(a, u, depth == 0 ? 0 : t.large[k], depth, smem.cta, threadIdx.x, last, next);
        __syncthreads();
        const int w = threadIdx.x >> 5;
        // Small nodes over the CTAs first, then over a CTA's warps.
        for (int k = small0 + blockIdx.x + gridDim.x * w; k < small1; k += gridDim.x * WARPS)
            split_node<32>(a, u, depth == 0 ? 0 : t.small[k], depth, smem.warp[w], threadIdx.x & 31, last, next);
        grid.sync();
        first = last;
        last += __ldcg(next);
        large0 = large1;
        large1 += __ldcg(next + 1);
        small0 = small1;
        small1 += __ldcg(next + 2);
    }
    const int nodes = last;

    // Per start position: the internal nodes starting there and the least depth among them; their prefix sum
    // (one CTA); then the host's node indices: the k-th internal node in depth-first order has children 2k + 1
    // and 2k + 2.
    for (long long x = rank; x < nodes; x += size)
        if (t.left[x] >= 0) {
            atomicAdd(t.starts + t.begin[x], 1);
            atomicMin(t.top + t.begin[x], t.depth[x]);
        }
    grid.sync();
    if (blockIdx.x == 0) {
        constexpr int RUN = 8;  // consecutive positions per thread
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        int carry = 0;
        for (int base = 0; base < T; base += BUILD_THREADS * RUN) {
            const int i0 = base + threadIdx.x * RUN;
            int v[RUN], sum = 0;
            for (int k = 0; k < RUN; ++k) {
                v[k] = i0 + k < T ? __ldcg(t.starts + i0 + k) : 0;
                sum += v[k];
            }
            int incl = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) prefix_warp[warp] = incl;
            __syncthreads();
            int at = carry + incl - sum;
            for (int k = 0; k < WARPS; ++k) {
                if (k < warp) at += prefix_warp[k];
                carry += prefix_warp[k];
            }
            for (int k = 0; k < RUN; ++k) {
                if (i0 + k < T) t.prefix[i0 + k] = at;
                at += v[k];
            }
            __syncthreads();
        }
    }
    grid.sync();
    for (long long x = rank; x < nodes; x += size) {
        const int l = t.left[x];
        if (l < 0) continue;
        const int b = t.begin[x];
        const int k = t.prefix[b] + t.depth[x] - __ldcg(t.top + b);
        t.index[l] = 2 * k + 1;
        t.index[l + 1] = 2 * k + 2;
    }
    if (rank == 0) *t.counter = nodes;
    grid.sync();

    // The packed tree, its triangles, and the slots of this mesh.
    for (long long x = rank; x < nodes; x += size) write_node(a, t, static_cast<int>(x));
    for (long long p = rank; p < T; p += size) write_triangle(a, t, static_cast<int>(p));
    for (long long k = rank; k < slots; k += size)
        write_slot(a, t, slot_mesh, mesh, slot_root, slot_bounds, slot_hull, static_cast<int>(k));
}

}  // namespace

cudaError_t launch_mesh_build(const MeshBuildArgs &a, const MeshBuildScratch &t, const int *slot_mesh, int slots,
    int mesh, int2 *slot_root, float *slot_bounds, float4 *slot_hull, cudaStream_t stream) {
    int device = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, build_mesh_kernel, BUILD_THREADS, 0);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    // Every CTA resident at once (the barriers need it); no more CTAs than about one per 8 triangles.
    long long blocks = static_cast<long long>(sms) * per_sm;
    const long long want = (static_cast<long long>(a.triangles) + 7) / 8;
    if (blocks > want) blocks = want;
    if (blocks < 1) blocks = 1;
    void *args[] = {const_cast<MeshBuildArgs *>(&a), const_cast<MeshBuildScratch *>(&t), &slot_mesh, &slots, &mesh,
        &slot_root, &slot_bounds, &slot_hull};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void *>(build_mesh_kernel), dim3(static_cast<unsigned>(blocks)),
        dim3(BUILD_THREADS), args, 0, stream);
}

}  // namespace ngb
