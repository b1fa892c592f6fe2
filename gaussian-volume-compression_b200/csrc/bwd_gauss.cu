// bwd_gauss.cu -- deterministic backward of the mixture field: every Gaussian owns its sums
// (replaces BACKWARD::renderCUDA, diff-gaussian-rasterization/cuda_rasterizer/
// backward.cu:127-337, and its sample-side counterpart :339-559, whose atomics it needs not).
//
// Rows.  k_backward_rows turns the Morton-sorted samples into gradient rows, stored by
// chunks of 16: 16 x, 16 y, 16 z, 16 gx, 16 gyz (320 bytes), so that a lane reads two
// neighbouring rows of each field as one float2.  The same kernel reduces the boxes of the
// chunks and of runs of 8 chunks, the lower levels of a wide tree (wide_tree.cuh).  A row
// without a gradient (W below the cutoff, an upstream gradient of zero, or a sample that is no point)
// adds nothing to any sum and is left out of the boxes; its coordinates are stored as zeros, since
// a zero times a NaN or an infinity would not be one.
//
// Sums.  A warp walks that tree with its Gaussian's AABB, 32 children per step:
// neighbouring children lie in neighbouring memory, and five levels cover 16M samples,
// where a binary tree took about seventeen dependent steps.  Chunks that overlap the box
// and may hold a point of the power window (cull.cuh) are queued and evaluated four at a
// time, two rows per lane; the eleven moments (pair.cuh) stay in registers.  One reduction
// over the warp per Gaussian; no atomics; bitwise reproducible.  Where there are few
// Gaussians each has four warps; where there are many, four that follow one another in
// Morton order share one warp and one walk.
//
// What bounds it: the rows evaluated and the instructions per row and per tested box.
// Chunks of 16 rows with the window test evaluate 2.8 rows per contributing pair (300k
// Gaussians x 2.1M samples), where lane groups of up to 32 rows behind a binary tree took
// 3.8 and a ring of gathered row numbers; 8 rows per chunk would save 22 % of the rows and
// double the tests.  That case 4.23 -> 2.38 ms (69 % of the issue slots, 32 warps per SM);
// 1M clustered Gaussians x 4M samples 7.75 -> 4.06 ms; 4096 x 64^3 0.174 -> 0.053 ms.
#include "cull.cuh"
#include "pair.cuh"
#include "render.cuh"
#include "wide_tree.cuh"

namespace gvc {

namespace {

constexpr int kRowThreads = 256;   // k_backward_rows: four rows per thread, one level-1 node per warp
constexpr int kGaussMinWarps = 32;  // resident warps per SM asked of the register allocator
constexpr int kFlushChunks = 4;    // chunks per evaluation
constexpr int kChunkCap = 64;      // queued chunks: below kFlushChunks + 32
constexpr int kUnionCap = 512;     // chunks listed for the Gaussians of one warp
constexpr int kShare = 4;          // Gaussians of one warp where they share a walk

// One warp per level-1 node: 128 sorted rows, four per lane.  Per row (x, y, z) and, where
// W > 0.01, gx = dL/dout / W and gyz = -dL/dout * out / W + dL/dW (backward.cu:252-298 folds
// the same factors per pair); zeros otherwise.  (out, W) come from the forward's sorted copy
// when out_sorted is given, else they are gathered like dL/dout and dL/dW.
__global__ void __launch_bounds__(kRowThreads) k_backward_rows(
    int64_t S, int n_nodes, const float4* __restrict__ s_sorted, const float2* __restrict__ out_sorted,
    const float* __restrict__ out_cells, const float* __restrict__ out_weights, const float* __restrict__ gout,
    const float* __restrict__ gw, float* __restrict__ rows, float4* __restrict__ chunk_boxes,
    float4* __restrict__ level1) {
    const int lane = threadIdx.x & 31;
    const int node = blockIdx.x * (kRowThreads / 32) + (threadIdx.x >> 5);
    if (node >= n_nodes) return;  // warp-uniform
    const int64_t r0 = (int64_t)node * kRowsPerNode + 4 * lane;
    float x[4], y[4], z[4], gx[4], gyz[4];
    Box6 b = empty_box();
    float4 sp[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
        sp[k] = r0 + k < S ? s_sorted[r0 + k] : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int o = __float_as_int(sp[k].w);
        x[k] = sp[k].x;
        y[k] = sp[k].y;
        z[k] = sp[k].z;
        gx[k] = gyz[k] = 0.f;
        if (o >= 0 && x[k] == x[k]) {
            const float2 ow = out_sorted ? out_sorted[r0 + k] : make_float2(out_cells[o], out_weights[o]);
            if (ow.y > kWeightCutoff) {
                const float g = gout[o];
                gx[k] = __fdiv_rn(g, ow.y);
                gyz[k] = __fadd_rn(__fdiv_rn(-__fmul_rn(g, ow.x), ow.y), gw[o]);
            }
        }
        if (!(gx[k] == 0.f && gyz[k] == 0.f)) grow(b, Box6{x[k], y[k], z[k], x[k], y[k], z[k]});
        else x[k] = y[k] = z[k] = 0.f;
    }
    float4* dst = reinterpret_cast<float4*>(rows + (r0 / kChunkRows) * kChunkFloats) + (lane & 3);
    dst[0] = make_float4(x[0], x[1], x[2], x[3]);
    dst[4] = make_float4(y[0], y[1], y[2], y[3]);
    dst[8] = make_float4(z[0], z[1], z[2], z[3]);
    dst[12] = make_float4(gx[0], gx[1], gx[2], gx[3]);
    dst[16] = make_float4(gyz[0], gyz[1], gyz[2], gyz[3]);
    grow(b, shfl_xor_box(b, 1));
    grow(b, shfl_xor_box(b, 2));
    if ((lane & 3) == 0) store_box(chunk_boxes, r0 / kChunkRows, b);
    grow(b, shfl_xor_box(b, 4));
    grow(b, shfl_xor_box(b, 8));
    grow(b, shfl_xor_box(b, 16));
    if (lane == 0) store_box(level1, node, b);
}

// One Gaussian's sums over the chunks handed to it (every value but the moments is
// warp-uniform).
template <bool COUNT>
struct GaussSums {
    const WideTree& tree;
    const float* __restrict__ rows;
    int* queue;  // shared [kChunkCap]
    int n_queue;
    float t;        // cull_allowance
    float3 lo, hi;  // AABB
    float mx, my, mz, v, q0, q1, q2, q3, q4, q5;
    float m[11];
    int n_pairs, n_chunks;

    // 32 chunks, one per lane: those that may hold a contributing row are queued, and
    // evaluated kFlushChunks at a time
    __device__ __forceinline__ void test(int c, bool valid) {
        bool h = false;
        if (valid) {
            const float4* p = tree.box[0] + 2 * (int64_t)c;
            const float4 clo = __ldg(p), chi = __ldg(p + 1);
            h = box_overlap(clo, chi, lo, hi) &&
                !outside_window(CullGauss{mx, my, mz, q0, q1, q2, q3, q4, q5, t}, clo, chi);
        }
        const uint32_t k = __ballot_sync(0xffffffffu, h);
        if (h) queue[n_queue + __popc(k & lane_lt_mask())] = c;
        n_queue += __popc(k);
        __syncwarp();
        while (n_queue >= kFlushChunks) {
            n_queue -= kFlushChunks;
            eval(queue + n_queue, kFlushChunks);
        }
        __syncwarp();
    }

    __device__ __forceinline__ void row(float x, float y, float z, float gxr, float gyz) {
        const bool in = lo.x <= x && x <= hi.x && lo.y <= y && y <= hi.y && lo.z <= z && z <= hi.z;
        const float dx = x - mx, dy = y - my, dz = z - mz;
        // the forward's power, operation by operation (pair.cuh)
        const float p2 = dx * fmaf(q0, dx, fmaf(q1, dy, q2 * dz)) + dy * fmaf(q3, dy, q4 * dz) + dz * (q5 * dz);
        const bool c = in && p2 >= kLog2Floor && p2 <= 0.f;
        float e = ex2_approx(p2);
        e = c ? e : 0.f;
        const float s = fmaf(v, gxr, gyz) * e;
        const float gx = s * dx, gy = s * dy, gz = s * dz;
        m[0] = fmaf(gxr, e, m[0]);
        m[1] += s;
        m[2] += gx;
        m[3] += gy;
        m[4] += gz;
        m[5] = fmaf(gx, dx, m[5]);
        m[6] = fmaf(gx, dy, m[6]);
        m[7] = fmaf(gx, dz, m[7]);
        m[8] = fmaf(gy, dy, m[8]);
        m[9] = fmaf(gy, dz, m[9]);
        m[10] = fmaf(gz, dz, m[10]);
        if (COUNT) n_pairs += c && !(gxr == 0.f && gyz == 0.f);
    }

    // up to kFlushChunks queued chunks: eight lanes per chunk, two rows per lane
    __device__ __forceinline__ void eval(const int* ids, int n) {
        const int lane = threadIdx.x & 31;
        float2 X, Y, Z, GX, GYZ;
        X = Y = Z = GX = GYZ = make_float2(0.f, 0.f);
        if ((lane >> 3) < n) {
            const float2* p = reinterpret_cast<const float2*>(rows + (int64_t)ids[lane >> 3] * kChunkFloats) + (lane & 7);
            X = __ldg(p);
            Y = __ldg(p + 8);
            Z = __ldg(p + 16);
            GX = __ldg(p + 24);
            GYZ = __ldg(p + 32);
        }
        row(X.x, Y.x, Z.x, GX.x, GYZ.x);
        row(X.y, Y.y, Z.y, GX.y, GYZ.y);
        if (COUNT) n_chunks += n;
    }
};

// GPW > 1: a warp owns GPW Gaussians that follow one another in Morton order.  One walk with
// the union of their boxes lists the chunks near all of them (boxes only); then each
// Gaussian tests the list.  If the list does not hold the chunks, each walks by itself.
// WPG > 1: a Gaussian is owned by WPG warps: warp `part` takes the level-1 nodes whose
// number is part modulo WPG, and the warps' sums are added in that order.
template <int WPG, int GPW, bool COUNT>
__global__ void __launch_bounds__(WPG * 32, kGaussMinWarps / WPG) k_backward_gauss(
    int P, const int32_t* __restrict__ gorder, const float* __restrict__ means, const float* __restrict__ values,
    const float* __restrict__ weights, const float* __restrict__ conics, const float4* __restrict__ boxes,
    const __grid_constant__ WideTree tree, const float* __restrict__ rows, float* __restrict__ gacc,
    unsigned long long* stats) {
    static_assert(WPG == 1 || GPW == 1, "one of the two");
    __shared__ int s_queue[WPG][kChunkCap];
    __shared__ WideStack s_walk[WPG];
    __shared__ int s_list[WPG][GPW > 1 ? kUnionCap : 1];
    __shared__ float s_part[WPG][16];
    const int warp = WPG > 1 ? threadIdx.x >> 5 : 0, lane = threadIdx.x & 31;
    const int part = WPG > 1 ? warp : 0;
    const int g0 = blockIdx.x * GPW;
    int n_tested = 0, n_pairs = 0, n_chunks = 0;
    int n_list = 0;  // chunks listed, kUnionCap + 1: they did not fit
    if (GPW > 1) {
        float4 blo = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
        float4 bhi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
        if (lane < GPW && g0 + lane < P) {
            const int64_t o = gorder ? gorder[g0 + lane] : g0 + lane;
            blo = __ldg(boxes + 2 * o);
            bhi = __ldg(boxes + 2 * o + 1);
        }
        Box6 u{blo.x, blo.y, blo.z, bhi.x, bhi.y, bhi.z};
#pragma unroll
        for (int off = GPW / 2; off > 0; off >>= 1) grow(u, shfl_xor_box(u, off));
        const float3 lo = make_float3(__shfl_sync(0xffffffffu, u.lx, 0), __shfl_sync(0xffffffffu, u.ly, 0),
                                      __shfl_sync(0xffffffffu, u.lz, 0));
        const float3 hi = make_float3(__shfl_sync(0xffffffffu, u.hx, 0), __shfl_sync(0xffffffffu, u.hy, 0),
                                      __shfl_sync(0xffffffffu, u.hz, 0));
        int* list = s_list[warp];
        wide_walk<COUNT>(tree, lo, hi, 0xffffffffu, s_walk[warp], n_tested,
                           [&](int c, bool valid) -> bool {
                               bool h = false;
                               if (valid) {
                                   const float4* p = tree.box[0] + 2 * (int64_t)c;
                                   h = box_overlap(__ldg(p), __ldg(p + 1), lo, hi);
                               }
                               const uint32_t k = __ballot_sync(0xffffffffu, h);
                               if (n_list + __popc(k) > kUnionCap) {
                                   n_list = kUnionCap + 1;
                                   return false;
                               }
                               if (h) list[n_list + __popc(k & lane_lt_mask())] = c;
                               n_list += __popc(k);
                               return true;
                           });
        __syncwarp();
    }
    uint32_t mine = 0xffffffffu;  // level-1 nodes of this warp (by number modulo 32)
    if (WPG > 1) {
        mine = 0u;
#pragma unroll
        for (int k = 0; k < 32 / WPG; k++) mine |= 1u << (k * WPG);
        mine <<= part;
    }
#pragma unroll 1
    for (int j = 0; j < GPW; j++) {
        const int gi = g0 + j;
        if (GPW > 1 && gi >= P) break;
        const bool live = gi < P;  // warp-uniform
        const int64_t o = live ? (gorder ? gorder[gi] : gi) : 0;
        const float* cp = conics + 6 * o;
        const float4 blo = __ldg(boxes + 2 * o), bhi = __ldg(boxes + 2 * o + 1);
        const GaussB g = gauss_b(__ldg(means + 3 * o), __ldg(means + 3 * o + 1), __ldg(means + 3 * o + 2),
                                 __ldg(values + o), __ldg(cp), __ldg(cp + 1), __ldg(cp + 2), __ldg(cp + 3),
                                 __ldg(cp + 4), __ldg(cp + 5), blo, bhi);
        GaussSums<COUNT> sums{tree, rows, s_queue[warp], 0, cull_allowance(g.q0, g.q1, g.q2, g.q3, g.q4, g.q5, true),
                              make_float3(blo.x, blo.y, blo.z), make_float3(bhi.x, bhi.y, bhi.z),
                              g.mx, g.my, g.mz, g.v, g.q0, g.q1, g.q2, g.q3, g.q4, g.q5};
#pragma unroll
        for (int k = 0; k < 11; k++) sums.m[k] = 0.f;
        sums.n_pairs = sums.n_chunks = 0;
        if (GPW > 1 && n_list <= kUnionCap) {
            for (int i = 0; i < n_list; i += 32) {
                const bool v = i + lane < n_list;
                sums.test(v ? s_list[warp][i + lane] : 0, v);
            }
        } else if (live) {
            wide_walk<COUNT>(tree, sums.lo, sums.hi, mine, s_walk[warp], n_tested,
                               [&](int c, bool valid) -> bool {
                                   sums.test(c, valid);
                                   return true;
                               });
        }
        if (sums.n_queue > 0) sums.eval(sums.queue, sums.n_queue);
        if (COUNT) {
            n_pairs += sums.n_pairs;
            n_chunks += sums.n_chunks;
        }
        float v16[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v16[k] = k < 11 ? sums.m[k] : 0.f;
        float tot = warp_transpose_reduce16(v16);
        if (WPG > 1) {
            if (!(lane & 1)) s_part[warp][lane >> 1] = tot;
            __syncthreads();
            if (part == 0) {
                tot = 0.f;
#pragma unroll
                for (int w = 0; w < WPG; w++) tot += s_part[w][lane >> 1];
            }
        }
        if (live && part == 0) {
            const float term = moments_to_terms(tot, __ldg(weights + o), __ldg(cp), __ldg(cp + 1), __ldg(cp + 2),
                                                __ldg(cp + 3), __ldg(cp + 4), __ldg(cp + 5));
            if (!(lane & 1)) gacc[16 * o + (lane >> 1)] = term;
        }
        __syncwarp();
    }
    if (COUNT) {
        unsigned long long a = (unsigned long long)n_pairs;
        for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
        if (lane == 0) {
            atomicAdd(&stats[2], a);
            atomicAdd(&stats[7], (unsigned long long)n_chunks);
            atomicAdd(&stats[8], (unsigned long long)n_tested);
            atomicAdd(&stats[10], (unsigned long long)n_chunks * kChunkRows);
        }
    }
}

inline unsigned nblk(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

// Fewer Gaussians than the chip holds warps (148 x 32): four warps for each.  Measured with
// 1M samples, four warps / one warp: 2000 Gaussians 41 / 51 us, 5000 81 / 85, 10000 153 / 129.
constexpr int kFewGaussians = 148 * 32;
// From this many on, one warp for four Gaussians that share a walk.  One each / four, us:
// 60k samples: 40k Gaussians 92 / 91, 80k 164 / 143, 160k 299 / 245; 1M samples: 80k
// 606 / 664, 160k 1025 / 989; 1M clustered Gaussians x 4M: 5260 / 4060.
constexpr int kManyGaussians = 100000;

}  // namespace

RowTreeSize row_tree_size(int64_t S) {
    RowTreeSize z;
    const int64_t nodes = (S + kRowsPerNode - 1) / kRowsPerNode;
    z.tree = wide_tree_size(nodes * kWideLeaves);
    z.rows_bytes = sizeof(float) * kChunkFloats * kWideLeaves * (size_t)nodes;
    return z;
}

cudaError_t launch_backward_rows(int64_t S, const RowTreeSize& z, const float4* s_sorted, const float2* out_sorted,
                                 const float* out_cells, const float* out_weights, const float* gout, const float* gw,
                                 float* rows, float4* boxes, cudaStream_t st) {
    if (S <= 0) return cudaSuccess;
    const int64_t nodes = z.tree.n[1];
    k_backward_rows<<<nblk(nodes, kRowThreads / 32), kRowThreads, 0, st>>>(
        S, (int)nodes, s_sorted, out_sorted, out_cells, out_weights, gout, gw, rows, boxes, boxes + 2 * z.tree.n[0]);
    note_launch();
    return launch_wide_levels(z.tree, boxes, st);
}

template <int WPG, int GPW>
static void launch_gauss(const BwdArgs& a, const WideTree& tree, const float* rows, cudaStream_t st) {
    const unsigned nb = nblk(a.P, GPW);
    if (a.count)
        k_backward_gauss<WPG, GPW, true><<<nb, WPG * 32, 0, st>>>(
            (int)a.P, a.gorder, a.means, a.values, a.weights, a.conics, a.boxes, tree, rows, a.gacc, a.stats);
    else
        k_backward_gauss<WPG, GPW, false><<<nb, WPG * 32, 0, st>>>(
            (int)a.P, a.gorder, a.means, a.values, a.weights, a.conics, a.boxes, tree, rows, a.gacc, a.stats);
}

cudaError_t launch_backward_gauss(const BwdArgs& a, const WideTree& tree, const float* rows, cudaStream_t st) {
    if (a.P <= 0) return cudaSuccess;
    if (a.P < kFewGaussians) launch_gauss<4, 1>(a, tree, rows, st);
    else if (a.P < kManyGaussians) launch_gauss<1, 1>(a, tree, rows, st);
    else launch_gauss<1, kShare>(a, tree, rows, st);
    note_launch();
    return cudaGetLastError();
}

}  // namespace gvc
