// lbvh.cuh -- LBVH builder interface of the Gaussians, points and cells.
#pragma once
#include "gvc_internal.cuh"

namespace gvc {

// Radix sort tile: 8 warps x 16 iterations x 32 lanes = 4096 keys per block.
constexpr int kRsWarps = 8;
constexpr int kRsIters = 16;
constexpr int kRsTile = kRsWarps * kRsIters * 32;

// Bytes each Lbvh buffer must hold for an LBVH build over n boxes (lbvh_build_boxes);
// the builder sizes its buffers with exactly these, and callers that provide the buffers
// themselves (the allocation-free sampler) check their views against them.
struct LbvhBytes {
    static constexpr int64_t internal(int64_t n) { return n > 1 ? n - 1 : 1; }
    static constexpr size_t keys(int64_t n) { return sizeof(uint32_t) * (size_t)n; }  // keys, keys_alt, perm, perm_alt
    static constexpr size_t hist(int64_t n) {
        return sizeof(uint32_t) * (256 * (size_t)((n + kRsTile - 1) / kRsTile) + 256);
    }
    static constexpr size_t onesweep(int64_t n) {  // digit counts [4][256], tickets, a look-back word per tile and digit
        return sizeof(uint32_t) * (4 * 256 + 64 + 4 * 256 * (size_t)((n + kRsTile - 1) / kRsTile));
    }
    static constexpr size_t bounds() { return sizeof(uint32_t) * 8; }
    static constexpr size_t sorted_boxes(int64_t n) { return 2 * 16 * (size_t)n; }
    static constexpr size_t flags(int64_t n) { return sizeof(uint32_t) * (size_t)internal(n); }
    static constexpr size_t nodes(int64_t n) { return sizeof(BvhNode) * (size_t)n; }
};

// Stable LSD sort of n indices by a key of several 32-bit words (words[0] least
// significant); bits[w] = significant bits of word w (ceil(bits / 8) radix passes).
// Result in L.perm (sorted position -> input index); L.keys / keys_alt are scratch.
cudaError_t radix_sort_words(Lbvh& L, int64_t n, const uint32_t* const* words, const int* bits, int nwords,
                             cudaStream_t st);

// 30-bit Morton keys of box centroids over the centroid bounds, then a stable radix sort:
// L.keys (sorted) and L.perm (sorted position -> input index).
cudaError_t morton_sort_boxes(Lbvh& L, int64_t n, const float4* boxes, cudaStream_t st);
// Same for points [n][3].
cudaError_t morton_sort_points(Lbvh& L, int64_t n, const float* pts, cudaStream_t st);

// Test hook: morton_sort_points (over more than one tile) with the first tile of every pass
// withheld and an order that held no index, so that each look-back runs out.
cudaError_t morton_sort_points_withheld(Lbvh& L, int64_t n, const float* pts, cudaStream_t st);

// Common prefix of the keys at i and j of the sorted order, equal keys told apart by position.
__device__ __forceinline__ int lbvh_delta(const uint32_t* __restrict__ keys, int i, int j) {
    const uint32_t a = keys[i], b = keys[j];
    return a == b ? 32 + __clz((uint32_t)(i ^ j)) : __clz(a ^ b);
}
// Whether the subtree over the leaves [l, r], not all n, is its parent's left child.
__device__ __forceinline__ bool lbvh_is_left(const uint32_t* __restrict__ keys, int n, int l, int r) {
    if (l == 0) return true;
    if (r == n - 1) return false;
    return lbvh_delta(keys, r, r + 1) > lbvh_delta(keys, l - 1, l);
}

// The tree (L.nodes) over keys and leaf boxes already in sorted order.
cudaError_t lbvh_hierarchy(Lbvh& L, int64_t n, const uint32_t* sorted_keys, const float4* sorted_leaf_boxes,
                           cudaStream_t st);

// The same over points (x, y, z, any).
cudaError_t lbvh_hierarchy_points(Lbvh& L, int64_t n, const uint32_t* sorted_keys, const float4* sorted_points,
                                  cudaStream_t st);

// Full build from boxes in input order: keys, sort, gather, hierarchy.
cudaError_t lbvh_build_boxes(Lbvh& L, int64_t n, const float4* boxes, cudaStream_t st);

}  // namespace gvc
