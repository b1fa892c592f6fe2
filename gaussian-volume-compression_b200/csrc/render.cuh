// render.cuh -- launch interfaces of the forward / backward evaluation kernels and
// of the preprocessing kernels (prep.cu).
#pragma once
#include "wide_tree.cuh"

namespace gvc {

// Candidate log of the forwards, read by the tensor-core backward instead of walking the
// LBVH again: the Gaussians whose boxes overlap a block's coarse groups in order in the
// block's kCandLogPerBlock slots, coarse group g's ending at cend[blk * 8 + g], and with each
// a byte whose bit b says that it meets the block's group b (box overlap and window test;
// fwd_blocks.cu writes them, after the other forwards launch_log_masks does); a block
// with more candidates than slots gets -1 for every group, and the backward walks.
constexpr int kCandLogPerBlock = 4096;

struct CandLog {
    int32_t* ids = nullptr;  // this block's slots, or null (no log)
    uint8_t* masks = nullptr;
    int pos = 0;             // candidates appended (warp-uniform)
    bool over = false;
    int gend = 0;  // on lane g: end of group g

    // appends lanes 0 .. n - 1
    __device__ __forceinline__ void append(int n, int id, uint32_t mask) {
        const int lane = threadIdx.x & 31;
        if (pos + n > kCandLogPerBlock) {
            over = true;
        } else if (lane < n) {
            ids[pos + lane] = id;
            if (masks) masks[pos + lane] = (uint8_t)mask;
        }
        pos += n;
    }
    __device__ __forceinline__ void end_group(int g) {
        if ((threadIdx.x & 31) == g) gend = pos;
    }
    __device__ __forceinline__ void finish(int32_t* cend_blk, int ng) {
        if (ids && (int)(threadIdx.x & 31) < ng) cend_blk[threadIdx.x & 31] = over ? -1 : gend;
    }
};

struct FwdArgs {
    int64_t P;
    const float4* s_sorted;
    int64_t S;
    const uint2* bdesc;    // [n_blocks] block-group descriptors
    const float4* bboxes;  // [n_blocks * 8] block-group boxes (lo, hi)
    WideTree tree;         // over the Gaussians in Morton order (level 0: their AABBs)
    const BvhNode* nodes;  // the LBVH over the same order: walked instead when given
    const GaussRec* recs;  // the same order
    float* out_cells;
    float* out_weights;
    float2* out_sorted;    // (out, W) per sorted slot, read by the backward's rows (FP32 only); or null
    int32_t* clog;         // candidate log, or null
    uint8_t* cmask;        // its masks (FP32 forward)
    int32_t* cend;
    const uint2* fdesc;    // the block's finer groups (the bits of cmask)
    const float4* fboxes;
    int* status;
    unsigned long long* stats;
    bool count;
};
// fwd_blocks.cu: FP32, one warp per block of 128 samples (or per part of it)
cudaError_t launch_forward_blocks(const FwdArgs& a, cudaStream_t st);
// Rows per warp of it by the LBVH, or 0 where launch_forward_cta's three warps per block are
// faster.  us at 32 rows / three warps / 128 rows: 200k Gaussians x 60k samples
// 797 / 895 / 1423, x 262k 901 / 632 / 833, x 524k 1122 / 729 / 698, x 4M 3971 / 2427 / 1741;
// 300k clustered x 524k 779 / 528 / 605; 1M clustered x 130k 2377 / 2413 / 4006,
// x 1M 3121 / 1869 / 2152, x 4M 6063 / 3689 / 3206; 20k x 60k 102 / 122 / 173.
inline int forward_linked_rows(int64_t S, int64_t P) {
    return S < 100000 ? 32 : S >= 500000 && S >= 2 * P ? 128 : 0;
}
// cta.cu: by the LBVH
cudaError_t launch_forward_cta(const FwdArgs& a, cudaStream_t st);
// fwd_points.cu: FP32, one warp per sample (no candidate log)
cudaError_t launch_forward_points(const FwdArgs& a, cudaStream_t st);
// fwd_tc.cu: the exponent on tcgen05, one CTA per block
cudaError_t launch_forward_tc(const FwdArgs& a, cudaStream_t st);

// Groups of the 128-sample blocks (cta.cu): a run of rows splits where both halves' boxes have
// at most `ratio` of the whole's half-perimeter.  kBlockSplit for the FP32 forward and the
// tensor-core backward; with the tensor-core kernels the forward's groups are coarser.
// FP32 forward and tensor-core backward at 0.45 / 0.55 / 0.65 / 0.75, ms: 2M x 16M
// 11.3 / 11.1 / 11.1 / 12.4 and 17.3 / 15.8 / 14.6 / 14.1; 1M x 4M clustered forward
// 2.84 / 2.54 / 2.51 / 2.64; 256^3 grid x 500k forward 5.42 / 5.42 / 5.42 / 6.91.
constexpr float kBlockSplit = 0.65f;
constexpr float kBlockSplitCoarse = 0.45f;
// Block groups with `ratio`; with bdesc2 also a second set with `ratio2` from the same
// loaded rows (one launch).
cudaError_t launch_sample_blocks(int64_t S, const float4* s_sorted, const uint32_t* skeys, uint2* bdesc,
                                 float4* bboxes, float ratio, cudaStream_t st, uint2* bdesc2 = nullptr,
                                 float4* bboxes2 = nullptr, float ratio2 = 0.f);

struct BwdArgs {
    int64_t P;
    const float4* boxes;       // caller order, lo/hi
    const float* conics;
    // Gaussian-owned sums
    const int32_t* gorder;     // processing order (sorted pos -> caller idx) or null
    const float* means;
    const float* values;
    const float* weights;
    // tensor-core sums
    const int32_t* gperm;      // Morton order -> caller idx
    int64_t S;
    const uint2* bdesc;        // block groups
    const float4* bboxes;
    const float4* s_grad;      // (x, y, z, gx) per sorted slot
    const float* s_gyz;        // gyz per sorted slot
    const uint8_t* s_ok;       // W > 0.01 per sorted slot (pair statistics)
    const BvhNode* nodes;      // LBVH over the Gaussians in Morton order
    const int32_t* clog;       // the forward's candidate log (null: walk)
    const uint8_t* cmask;      // its masks
    const int32_t* cend;
    const uint2* cdesc;        // the coarse groups of the log
    const GaussRec* recs;      // Morton order
    float* gacc;               // [P][16] caller order
    int* status;
    unsigned long long* stats;
    bool count;
};

cudaError_t launch_tc_gemm_test(const void* A, const void* B, int N, float* D, int* status, cudaStream_t st);
// One block waiting on an mbarrier nothing arrives on: the bounded wait runs out and
// records kStatusTimeout (tests the host-side report of device timeouts).
cudaError_t launch_wait_timeout_test(int* status, cudaStream_t st);

// bwd_gauss.cu: gradient rows in chunks of 16 under a wide tree (leaves: chunks), and the
// Gaussian-owned sums that walk it
constexpr int kChunkRows = 16;
constexpr int kChunkFloats = 5 * kChunkRows;  // x, y, z, gx, gyz
constexpr int kRowsPerNode = kWideLeaves * kChunkRows;
struct RowTreeSize {
    WideTreeSize tree;
    size_t rows_bytes;  // gradient rows
};
RowTreeSize row_tree_size(int64_t S);
// out_sorted: the forward's (out, W) per sorted slot when the caller's out_cells /
// out_weights are that forward's outputs (else null: they are gathered).
cudaError_t launch_backward_rows(int64_t S, const RowTreeSize& z, const float4* s_sorted, const float2* out_sorted,
                                 const float* out_cells, const float* out_weights, const float* gout, const float* gw,
                                 float* rows, float4* boxes, cudaStream_t st);
cudaError_t launch_backward_gauss(const BwdArgs& a, const WideTree& tree, const float* rows, cudaStream_t st);

// bwd_tc.cu: reduction over samples on tcgen05, one CTA per 128 samples
cudaError_t launch_backward_tc(const BwdArgs& a, cudaStream_t st);
// `moved` (device, or null) nonzero: the log is of other boxes than `recs`', and every block's is
// struck out instead.
cudaError_t launch_log_masks(const BwdArgs& a, uint8_t* cmask, int32_t* cend, const int* moved, cudaStream_t st);
cudaError_t launch_finalize(int64_t P, const float* gacc, const float* scales, const float* rots, const float* conics,
                            float sm, int ref_compat, float* dmeans, float* dscales, float* drots, float* dvalues,
                            float* dweights, cudaStream_t st);

// prep.cu (compiled without FMA contraction so that its arithmetic matches the oracle)
cudaError_t launch_preprocess(int64_t P, const float* means, const float* scales, const float* rots,
                              const float* weights, float sm, float* conics_out, float4* boxes_out, cudaStream_t st);
// Records in Morton order, and their wide tree at `tree_boxes` (levels false: its two lowest
// levels only).  `moved` (device, or null): set if a leaf differs from what tree_boxes held.
cudaError_t launch_gather_recs(int64_t P, int32_t* perm, const float* means, const float* values,
                               const float* weights, const float* conics, const float4* boxes, GaussRec* recs,
                               float4* tree_boxes, bool levels, int* moved, cudaStream_t st);
// Sorted sample slots: (x, y, z, bits of the caller's index or -1).
cudaError_t launch_sample_slots(int64_t S, int64_t n_slots, const float* samples, int32_t* perm,
                                float4* s_sorted, cudaStream_t st);
// out_sorted: the forward's (out, W) per sorted slot when the caller's out_cells /
// out_weights are that forward's outputs (else null: they are gathered).
cudaError_t launch_sample_grads(int64_t n_slots, const float4* s_sorted, const float2* out_sorted,
                                const float* out_cells, const float* out_weights, const float* gout, const float* gw,
                                float4* s_grad, float* s_gyz, uint8_t* s_ok, cudaStream_t st);
cudaError_t launch_fill_zero_outputs(int64_t S, float* out_cells, float* out_weights, cudaStream_t st);

// mesh.cu
cudaError_t launch_sample_uniform(const int64_t dims[3], const float origin[3], const float spacing[3],
                                  const void* values, int dtype, int64_t N, const float* samples, void* out,
                                  cudaStream_t st);
// Cells as int64 arrays: types_out / conn_out (truncated to 32 bits) and the six words of
// gvc_check_cells' result.
cudaError_t launch_check_cells(int64_t C, const int64_t* types, const int64_t* offsets, int64_t n_conn,
                               const int64_t* conn, int64_t npts, uint8_t* types_out, int32_t* conn_out,
                               int64_t* result, cudaStream_t st);
cudaError_t launch_tet_boxes(int64_t C, const float* pts, const int32_t* conn4, float4* boxes, cudaStream_t st);
cudaError_t launch_cell_boxes(int64_t C, const float* pts, const uint8_t* types, const int64_t* offsets,
                              const int32_t* conn, float4* boxes, cudaStream_t st);
// Tree over the cells in Morton order and, of tetrahedra (conn4 given), their records (8 float4
// per cell).
cudaError_t launch_cell_tree(int64_t C, int32_t* perm, const float4* boxes, const float* pts,
                             const int32_t* conn4, float4* recs, float4* tree_boxes, cudaStream_t st);
struct LocateArgs {
    int64_t N, C;
    const float* samples;
    int32_t* sperm;            // Morton order of the samples, or null: they are sorted
    const float4* tree_boxes;
    const int32_t* cperm;
    const double* values;
    const float4* recs;        // tetrahedra, or null and:
    const float* pts;
    const uint8_t* types;
    const int64_t* offsets;
    const int32_t* conn;
    double* out;
    float* out32;              // instead of out
    int64_t* cell_ids;         // or null
};
cudaError_t launch_locate(const LocateArgs& a, cudaStream_t st);
cudaError_t launch_sample_tets(int64_t N, const float* samples, const int32_t* sperm, const float* pts,
                               const int32_t* conn4, const double* values, const BvhNode* cnodes,
                               const int32_t* cperm, int64_t C, double* out, int64_t* cell_ids, int* status,
                               cudaStream_t st);

// trainsamp.cu
cudaError_t launch_tet_points(int64_t N, int64_t S, uint64_t seed, const float* pts, const int32_t* conn4, int64_t C,
                              float* out, uint32_t* w_lo, uint32_t* w_hi, uint32_t* w_batch, cudaStream_t st);
cudaError_t launch_gather_points(int64_t N, const float* src, int32_t* perm, float* dst, cudaStream_t st);

// knn.cu: the points in Morton order with their index in .w, and the LBVH over them
cudaError_t launch_knn_points(int64_t n, const float* pts, int32_t* perm, float4* sorted, cudaStream_t st);
cudaError_t launch_knn3(int64_t n, const float4* sorted, const BvhNode* nodes, float* out, int* status,
                        cudaStream_t st);

}  // namespace gvc
