// wide_tree.cu -- the upper levels of the link-free box trees (wide_tree.cuh).
#include "wide_tree.cuh"

namespace gvc {

// One warp per node: the box of its up to 32 children.
__global__ void __launch_bounds__(256) k_wide_up(int n_child, const float4* __restrict__ child, int n_node,
                                                 float4* __restrict__ node) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= n_node) return;
    Box6 b = empty_box();
    const int64_t c = 32 * (int64_t)i + lane;
    if (c < n_child) {
        const float4 lo = child[2 * c], hi = child[2 * c + 1];
        b = Box6{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) grow(b, shfl_xor_box(b, off));
    if (lane == 0) store_box(node, i, b);
}

cudaError_t launch_wide_levels(const WideTreeSize& z, float4* boxes, cudaStream_t st) {
    float4* child = boxes + 2 * z.n[0];
    for (int l = 2; l <= z.top; l++) {
        float4* node = child + 2 * z.n[l - 1];
        k_wide_up<<<(unsigned)((z.n[l] + 7) / 8), 256, 0, st>>>((int)z.n[l - 1], child, (int)z.n[l], node);
        note_launch();
        child = node;
    }
    return cudaGetLastError();
}

}  // namespace gvc
