// wide_tree.cuh -- trees of boxes over Morton-sorted leaves, without links.
//
// Level 0 holds the leaves' boxes, level 1 the boxes of 8 leaves, every further level those
// of 32 nodes; the children of node i of a level above 1 are nodes 32 i .. 32 i + 31 of the
// level below.  A warp tests 32 boxes per step (32 children, or the leaves of four level-1
// nodes), all of them neighbours in memory and known without following a link, so a query
// of millions of leaves has five dependent steps where a binary tree has about twenty; the
// boxes come from one pass over the leaves and one small launch per level, where a linked
// hierarchy takes three kernels and an atomic climb.
#pragma once
#include "traverse.cuh"

namespace gvc {

struct Box6 {
    float lx, ly, lz, hx, hy, hz;
};

__device__ __forceinline__ Box6 empty_box() {
    return Box6{INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
}

__device__ __forceinline__ void grow(Box6& b, const Box6& o) {
    b.lx = fminf(b.lx, o.lx);
    b.ly = fminf(b.ly, o.ly);
    b.lz = fminf(b.lz, o.lz);
    b.hx = fmaxf(b.hx, o.hx);
    b.hy = fmaxf(b.hy, o.hy);
    b.hz = fmaxf(b.hz, o.hz);
}

__device__ __forceinline__ Box6 shfl_xor_box(const Box6& b, int off) {
    return Box6{__shfl_xor_sync(0xffffffffu, b.lx, off), __shfl_xor_sync(0xffffffffu, b.ly, off),
                __shfl_xor_sync(0xffffffffu, b.lz, off), __shfl_xor_sync(0xffffffffu, b.hx, off),
                __shfl_xor_sync(0xffffffffu, b.hy, off), __shfl_xor_sync(0xffffffffu, b.hz, off)};
}

__device__ __forceinline__ void store_box(float4* dst, int64_t i, const Box6& b) {
    dst[2 * i] = make_float4(b.lx, b.ly, b.lz, 0.f);
    dst[2 * i + 1] = make_float4(b.hx, b.hy, b.hz, 0.f);
}

// Box of 32 lanes' points, on every lane (`in` false or NaN coordinates: not counted).
__device__ __forceinline__ Box6 warp_point_box(bool in, float x, float y, float z) {
    Box6 b = empty_box();
    if (in) grow(b, Box6{x, y, z, x, y, z});
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) grow(b, shfl_xor_box(b, off));
    return b;
}

constexpr int kWideLeaves = 8;  // leaves of a level-1 node
constexpr int kWideLevels = 7;
struct WideTree {
    const float4* box[kWideLevels];  // per level: (lo, hi) of each node
    int n[kWideLevels];
    int top;
};

// Shared memory of one walking warp.
struct WideStack {
    int2 node[kWideLevels];  // per level: (children left to visit, first child)
    int list[64];            // queued level-1 nodes: at most 3 before a step adds up to 32
};

// Tests the children [first, first + 32) of a level above 0 against a box: lane i tests
// first + i.
__device__ __forceinline__ uint32_t wide_hits(const WideTree& tree, int level, int first, float3 lo, float3 hi) {
    const int i = first + (threadIdx.x & 31);
    bool h = false;
    if (i < tree.n[level]) {
        const float4* p = tree.box[level] + 2 * (int64_t)i;
        h = box_overlap(__ldg(p), __ldg(p + 1), lo, hi);
    }
    return __ballot_sync(0xffffffffu, h);
}

// Walks the tree with the box [lo, hi] and hands the level-1 nodes it meets to
// visit(first, mask): nodes first + i for the bits i of the mask.  Warp-collective; visit
// returns false to stop.  The order of the nodes depends on the tree and the box alone.
template <bool COUNT, class Visit>
__device__ __forceinline__ void wide_walk_nodes(const WideTree& tree, float3 lo, float3 hi, WideStack& st,
                                                int& n_tested, Visit visit) {
    const int lane = threadIdx.x & 31;
    for (int f = 0; f < tree.n[tree.top]; f += 32) {
        int level = tree.top, first = f;
        uint32_t m = wide_hits(tree, level, f, lo, hi);
        if (COUNT) n_tested += 32;
        while (true) {
            if (level == 1) {
                if (!visit(first, m)) return;
                m = 0;
            }
            if (m == 0) {
                if (level == tree.top) break;
                level++;
                const int2 s = st.node[level];
                m = (uint32_t)s.x;
                first = s.y;
                continue;
            }
            const int node = first + __ffs(m) - 1;
            m &= m - 1;
            __syncwarp();
            if (lane == 0) st.node[level] = make_int2((int)m, first);
            __syncwarp();
            level--;
            first = 32 * node;
            m = wide_hits(tree, level, first, lo, hi);
            if (COUNT) n_tested += 32;
        }
    }
}

// The same for the leaves of those nodes: visit(leaf, valid), 32 per call, eight lanes for each
// of four nodes.  `mine` selects level-1 nodes by their number modulo 32.
template <bool COUNT, class Visit>
__device__ __forceinline__ void wide_walk(const WideTree& tree, float3 lo, float3 hi, uint32_t mine, WideStack& st,
                                          int& n_tested, Visit visit) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = lane_lt_mask();
    int queued = 0;
    bool stopped = false;
    wide_walk_nodes<COUNT>(tree, lo, hi, st, n_tested, [&](int first, uint32_t m) -> bool {
        m &= mine;
        if ((m >> lane) & 1u) st.list[queued + __popc(m & lt)] = first + lane;
        queued += __popc(m);
        __syncwarp();
        while (queued >= 4) {
            queued -= 4;
            if (COUNT) n_tested += 32;
            const int leaf = st.list[queued + (lane >> 3)] * kWideLeaves + (lane & 7);
            if (!visit(leaf, leaf < tree.n[0])) {
                stopped = true;
                return false;
            }
        }
        __syncwarp();
        return true;
    });
    if (queued > 0 && !stopped) {
        if (COUNT) n_tested += 32;
        const int leaf = (lane >> 3) < queued ? st.list[lane >> 3] * kWideLeaves + (lane & 7) : tree.n[0];
        visit(leaf, leaf < tree.n[0]);
    }
}

// Host side: levels, sizes and addresses of a tree over n leaves (boxes: the leaves' boxes
// and then the levels above, 2 float4 per node).
struct WideTreeSize {
    int64_t n[kWideLevels];
    int top;
    int64_t boxes;
};

inline WideTreeSize wide_tree_size(int64_t n_leaves) {
    WideTreeSize z{};
    z.n[0] = n_leaves;
    int64_t n = (n_leaves + kWideLeaves - 1) / kWideLeaves;
    z.n[1] = n;
    z.top = 1;
    while (n > 64 && z.top + 1 < kWideLevels) {  // at most two steps over the top level
        n = (n + 31) / 32;
        z.n[++z.top] = n;
    }
    for (int l = 0; l <= z.top; l++) z.boxes += z.n[l];
    return z;
}

inline WideTree wide_tree_at(const WideTreeSize& z, const float4* boxes) {
    WideTree t{};
    t.top = z.top;
    for (int l = 0; l <= z.top; l++) {
        t.box[l] = boxes;
        t.n[l] = (int)z.n[l];
        boxes += 2 * z.n[l];
    }
    return t;
}

// Levels 2 and up from level 1 (wide_tree.cu).
cudaError_t launch_wide_levels(const WideTreeSize& z, float4* boxes, cudaStream_t st);

}  // namespace gvc
