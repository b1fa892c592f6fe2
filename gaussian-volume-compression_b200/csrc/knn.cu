// knn.cu -- mean squared distance to the three nearest other points.
//
// This is the initial-scale rule of the training code: scene/gaussian_model.py:175-179
// (create_from_pcd) and :729-733 (densify_in_empty) call simple-knn's distCUDA2, a
// third-party extension that is not part of the reference tree.  Its published
// behaviour, restated: for every point, the three smallest squared Euclidean distances
// to any other index (duplicates count with distance 0), kept in ascending order and
// averaged as (b0 + b1 + b2) / 3 in float32; neighbours that do not exist (n < 4)
// count as FLT_MAX.
//
// B200 design: the points are the leaves of the library's LBVH over their Morton order (64-byte
// nodes holding both child boxes).  One thread per Morton-sorted query: the 3rd-best distance
// among its +-3 Morton neighbours bounds the search, then a near-child-first traversal prunes
// every child whose box distance exceeds min(bound, current 3rd best).  Distances are
// rounded after every operation (no FMA contraction), which makes a box's distance
// never exceed the distance of any point inside it, so the pruning is exact and the
// result is bit-identical to the CPU restatement.
//
// Bound by the latency of the dependent loads and the divergence of the walks, 2M clustered
// points 675 us of the call's 1030.  Evaluating children of up to 4, 8 or 16 points whole, side by side in the
// sorted order, in place of descending them took 1.12, 1.2 and 1.45 times as long; a warp per 32 points
// walking a wide tree with one box 1.7 times (that box meets a hundred nodes, a ball five).
#include <float.h>

#include "lbvh.cuh"
#include "render.cuh"

namespace gvc {

namespace {

constexpr int kKnnStack = 64;  // the tree's depth is bounded by the 62 key + index bits

__global__ void __launch_bounds__(256) k_knn_points(int64_t n, const float* __restrict__ pts,
                                                    int32_t* __restrict__ perm, float4* __restrict__ sorted) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t o = order_at(perm, i, n);
    sorted[i] = make_float4(pts[3 * o], pts[3 * o + 1], pts[3 * o + 2], __int_as_float((int)o));
}

// Squared distance from q to the box [lo, hi]; for a degenerate box (a point) this is
// the point's squared distance ((dx*dx + dy*dy) + dz*dz, every operation rounded).
__device__ __forceinline__ float box_dist2(float4 q, float4 lo, float4 hi) {
    const float gx = fmaxf(fmaxf(__fsub_rn(lo.x, q.x), __fsub_rn(q.x, hi.x)), 0.f);
    const float gy = fmaxf(fmaxf(__fsub_rn(lo.y, q.y), __fsub_rn(q.y, hi.y)), 0.f);
    const float gz = fmaxf(fmaxf(__fsub_rn(lo.z, q.z), __fsub_rn(q.z, hi.z)), 0.f);
    return __fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)), __fmul_rn(gz, gz));
}

// the three smallest distances, ascending
struct Best3 {
    float b0, b1, b2;
    // `use` false, or a distance that is no number or not below the third: no change
    __device__ __forceinline__ void keep(float d, bool use) {
        d = use && d < b2 ? d : FLT_MAX;
        b2 = fminf(b2, fmaxf(d, b1));
        b1 = fminf(b1, fmaxf(d, b0));
        b0 = fminf(b0, d);
    }
};

__global__ void __launch_bounds__(128) k_knn3(int n, const float4* __restrict__ sorted,
                                              const BvhNode* __restrict__ nodes, float* __restrict__ out,
                                              int* status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 q = __ldg(sorted + i);
    Best3 best{FLT_MAX, FLT_MAX, FLT_MAX};
    // bound from the Morton neighbours i-3 .. i+3
#pragma unroll
    for (int k = -3; k <= 3; k++) {
        if (k == 0) continue;
        const float4 p = __ldg(sorted + min(max(i + k, 0), n - 1));
        best.keep(box_dist2(q, p, p), i + k >= 0 && i + k < n);
    }
    const float reject = best.b2;
    best = Best3{FLT_MAX, FLT_MAX, FLT_MAX};

    uint2 stack[kKnnStack];  // (node, bits of its distance)
    int sp = 0;
    int node = 0;
    while (true) {
        const float4* np = reinterpret_cast<const float4*>(nodes + node);
        const float4 a = __ldg(np), b = __ldg(np + 1), c = __ldg(np + 2), d = __ldg(np + 3);
        const uint32_t cl = __float_as_uint(a.w), cr = __float_as_uint(d.w);
        const float dl = box_dist2(q, a, b), dr = box_dist2(q, c, d);
        // leaves: the box distance is the point distance
        if (cl & kLeafBit) best.keep(dl, (int)(cl & ~kLeafBit) != i);
        if (cr & kLeafBit) best.keep(dr, (int)(cr & ~kLeafBit) != i);
        const float bound = fminf(reject, best.b2);
        const bool gl = !(cl & kLeafBit) && dl <= bound;
        const bool gr = !(cr & kLeafBit) && dr <= bound;
        if (gl && gr) {
            const bool left_first = dl <= dr;
            if (sp < kKnnStack) {
                stack[sp++] = left_first ? make_uint2(cr, __float_as_uint(dr)) : make_uint2(cl, __float_as_uint(dl));
            } else {
                atomicOr(status, kStatusStackOverflow);
            }
            node = (int)(left_first ? cl : cr);
            continue;
        }
        if (gl || gr) {
            node = (int)(gl ? cl : cr);
            continue;
        }
        // pop the next subtree that can still hold a closer point
        bool found = false;
        while (sp > 0) {
            const uint2 e = stack[--sp];
            if (__uint_as_float(e.y) <= fminf(reject, best.b2)) {
                node = (int)e.x;
                found = true;
                break;
            }
        }
        if (!found) break;
    }
    out[__float_as_int(q.w)] = __fdiv_rn(__fadd_rn(__fadd_rn(best.b0, best.b1), best.b2), 3.0f);
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

cudaError_t launch_knn_points(int64_t n, const float* pts, int32_t* perm, float4* sorted, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_knn_points<<<nblk(n, 256), 256, 0, st>>>(n, pts, perm, sorted); gvc::note_launch();
    return cudaGetLastError();
}

cudaError_t launch_knn3(int64_t n, const float4* sorted, const BvhNode* nodes, float* out, int* status,
                        cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    k_knn3<<<nblk(n, 128), 128, 0, st>>>((int)n, sorted, nodes, out, status); gvc::note_launch();
    return cudaGetLastError();
}

}  // namespace gvc
