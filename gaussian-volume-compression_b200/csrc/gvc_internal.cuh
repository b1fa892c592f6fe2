// gvc_internal.cuh -- shared device helpers, constants and the context layout.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>

#include "gvc.h"

namespace gvc {

// diff-gaussian-rasterization/cuda_rasterizer/config.h:9
constexpr float kWeightCutoff = 1e-2f;
// Sample slots are padded to a multiple of it.
constexpr int kTile = 32;
// Per-warp traversal stack (entries of int32) in shared memory.
constexpr int kStackCap = 512;
// Gaussians whose covariance condition estimate exceeds this get an FP64 inverse.
constexpr float kCondFp64 = 1.0e2f;

// Counts kernel launches issued by this library (reported by gvc_launch_count()).
void note_launch(int n = 1);

// Device status bits (OR-ed into ctx->d_status).
constexpr int kStatusStackOverflow = 1;
constexpr int kStatusTimeout = 2;  // a bounded wait gave up (mbarrier, radix-sort look-back)

// Entry i of a sorted order of n elements, for the kernel that reads the order first.  Where a
// look-back of the sort gave up (kStatusTimeout), slots of the order may never have been written:
// what is no index becomes 0, in the order itself too, for the kernels that read it later.
__device__ __forceinline__ int32_t order_at(int32_t* __restrict__ order, int64_t i, int64_t n) {
    const int32_t o = order[i];
    if ((uint32_t)o < (uint32_t)n) return o;
    order[i] = 0;
    return 0;
}

// Gaussian evaluation record, one per Gaussian in Morton order: 80 bytes.
//   r0 = (mu.x, mu.y, mu.z, w)
//   r1 = (c0, c1, c2, c3)  -- conic xx, xy, xz, yy as written to the conics output
//   r2 = (c4, c5, v, cover) -- conic yz, zz, value; cover = 1 where the window covers the AABB
//   r3 = (lo.x, lo.y, lo.z, 0), r4 = (hi.x, hi.y, hi.z, 0): the AABB
struct __align__(16) GaussRec {
    float4 r0, r1, r2, r3, r4;
};

// LBVH internal node with both children's boxes: 64 bytes.
//   a = (L.lo.xyz, left child),  b = (L.hi.xyz, first leaf),
//   c = (R.lo.xyz, last leaf),   d = (R.hi.xyz, right child)
// Child: internal node k > 0, or leaf i as (i | 0x80000000).  Node k > 0 holds the leaves from
// its first to k - 1 on its left and from k to its last on its right; node 0 is the root's copy.
struct __align__(16) BvhNode {
    float4 a, b, c, d;
};

constexpr uint32_t kLeafBit = 0x80000000u;

// Growable device buffer owned by the context; for a while a view of memory that the caller lends,
// with what the context owns kept aside.
struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    bool lent = false;
    void* own_ptr = nullptr;  // while lent
    size_t own_bytes = 0;
    cudaError_t ensure(size_t need) {
        if (need <= bytes && ptr) return cudaSuccess;
        if (lent) {
            give_back();
            if (need <= bytes && ptr) return cudaSuccess;
        }
        if (ptr) {
            cudaError_t e = cudaFree(ptr);
            if (e != cudaSuccess) return e;
            ptr = nullptr;
            bytes = 0;
        }
        size_t n = need < 256 ? 256 : need;
        n = (n + 255) & ~size_t(255);
        cudaError_t e = cudaMalloc(&ptr, n);
        if (e == cudaSuccess) bytes = n;
        return e;
    }
    template <class T>
    T* as() const { return reinterpret_cast<T*>(ptr); }
    void release() {
        give_back();
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
    // takes a view in place of memory of its own
    void lend(void* p, size_t n) {
        give_back();
        own_ptr = ptr;
        own_bytes = bytes;
        ptr = p;
        bytes = n;
        lent = true;
    }
    void give_back() {
        if (!lent) return;
        ptr = own_ptr;
        bytes = own_bytes;
        lent = false;
        own_ptr = nullptr;
        own_bytes = 0;
    }
};

// Radix-sort workspace and LBVH storage for one set of boxes.
struct Lbvh {
    int64_t n = 0;
    DevBuf keys, keys_alt, perm, perm_alt;  // sorted keys / permutation (sorted pos -> input idx)
    DevBuf sorted_boxes;                    // leaf boxes in sorted order, 2 x float4
    DevBuf flags;                           // children that have reached a node
    DevBuf nodes;                           // [n] BvhNode
    DevBuf hist, bounds;                    // sort histograms, centroid bounds
    DevBuf onesweep;                        // one-kernel-per-pass sort: digit counts, tickets, look-back words
    int* status = nullptr;                  // device status word; null keeps the three-kernel sort passes
};

}  // namespace gvc

struct gvc_ctx {
    int device = 0;
    std::string err;
    // options
    int cov_grad_mode = 0;
    int bwd_mode = 0;
    int eval_path = 0;
    int cand_log = 1;       // GVC_OPT_CAND_LOG
    int count_pairs = 0;
    int time_kernels = 0;   // record CUDA events around the evaluation kernels
    double fwd_kernel_ms = 0.0, bwd_kernel_ms = 0.0;
    int64_t fwd_kernel_calls = 0, bwd_kernel_calls = 0;
    cudaEvent_t ev_pool[64];  // pairs of (start, stop) events pending read-out
    int ev_kind[32];          // 0 = forward, 1 = backward
    int ev_pending = 0;
    bool ev_init = false;
    // sample state (gvc_build_bvh)
    const float* samples = nullptr;
    int64_t S = 0;
    int64_t n_tiles = 0;
    bool samples_ready = false;
    // candidate log of the last forward (for the tensor-core backward)
    gvc::DevBuf clog, cmask, cend;
    bool clog_ready = false;
    bool clog_masks = false;  // its masks are written
    gvc::DevBuf moved;        // whether a backward's Gaussians have other boxes than the log's
    // (out, W) per sorted slot as the last FP32 forward wrote them, and the
    // output arrays it wrote them to (the backward uses the copy for those arrays only)
    gvc::DevBuf fwd_sorted;
    const float* fwd_out_cells = nullptr;
    const float* fwd_out_weights = nullptr;
    bool fwd_sorted_ready = false;
    // the Gaussian arrays of the last forward: its AABBs (gtmp) and records (grec) are
    // reused by a backward handed the same arrays
    const float* fwd_means = nullptr;
    const float* fwd_scales = nullptr;
    const float* fwd_rots = nullptr;
    const float* fwd_values = nullptr;
    const float* fwd_weights = nullptr;
    const float* fwd_conics = nullptr;
    float fwd_scale_mod = 0.f;
    bool fwd_recs_ready = false;
    gvc::DevBuf s_sorted;   // [n_tiles*32] float4 (x, y, z, bits of caller index or -1)
    gvc::DevBuf blk_desc;   // [ceil(S/128)] uint2 block-group descriptors
    gvc::DevBuf blk_boxes;  // [ceil(S/128) * 8] block-group boxes, 2 x float4
    gvc::DevBuf blk_desc_c;   // the same with the coarser split of the tensor-core kernels' forward
    gvc::DevBuf blk_boxes_c;
    bool blk_c_ready = false;
    gvc::DevBuf s_grad;     // [n_tiles*32] float4 (x, y, z, gx) backward sample records
    gvc::DevBuf s_gyz;      // [n_tiles*32] float gyz (see k_sample_grads)
    gvc::DevBuf s_ok;       // [n_tiles*32] uint8 1 iff W > 0.01 (pair statistics only)
    gvc::Lbvh s_sort;       // sample sort (keys/perm only)
    gvc::DevBuf b_rows;     // gradient rows in chunks of 16 (Gaussian-owned backward, bwd_gauss.cu)
    gvc::DevBuf b_boxes;    // wide tree over the chunks
    // Gaussian state (forward)
    int64_t P = 0;
    bool gauss_ready = false;
    gvc::Lbvh gsort;        // Gaussian order (Morton order of the AABBs' centres), and with the
                            // tensor-core kernels the LBVH over it
    bool glinks_ready = false;  // its LBVH is built
    gvc::DevBuf gtree;      // leaf boxes in that order, and the wide tree's levels over them
    gvc::DevBuf grec;       // [P] GaussRec in Morton order
    gvc::DevBuf gtmp;       // preprocess scratch: AABBs in caller order
    // mesh samplers: the cells' Morton order, the wide tree and the tetrahedra's records in it
    gvc::Lbvh cells;
    gvc::DevBuf cell_tree, cell_recs;
    // three-nearest-neighbour distances (points in Morton order and the LBVH over them)
    gvc::Lbvh knn;
    gvc::DevBuf knn_points;
    // training sample batches: unsorted points, Morton / batch key words
    gvc::Lbvh ts_sort;
    gvc::DevBuf ts_points, ts_words;
    // status and statistics
    int* d_status = nullptr;          // device status word
    unsigned long long* d_stats = nullptr;  // [16] device counters
    int* h_status = nullptr;          // pinned mirror
};
