// fwd_points.cu -- forward evaluation where the samples are sparse among the Gaussians.
//
// One warp owns one sample: it walks the tree of Gaussians with the point itself, so that
// the exact AABB test is the walk's own leaf test, and every lane evaluates another Gaussian
// that holds the point.  A block of 128 sparse samples spans many Gaussians that reach only
// one or two of its rows each; a point meets none but its own.  Bound by the latency of the
// walk, about 25 dependent steps for a million Gaussians; 4 ns per sample with the chip full
// (1M Gaussians x 14k samples: 0.10 ms, 14.4 ms by blocks).
#include "pair.cuh"
#include "render.cuh"

namespace gvc {

namespace {

struct PointSmem {
    int cand[64];  // at most 31 before a step of the walk adds up to 32
    WideStack walk;
};

template <bool COUNT>
__global__ void __launch_bounds__(32, 32)
    k_forward_points(const float4* __restrict__ s_sorted, const __grid_constant__ WideTree tree,
                     const GaussRec* __restrict__ recs, float* __restrict__ out_cells, float* __restrict__ out_weights,
                     float2* __restrict__ out_sorted, unsigned long long* stats) {
    __shared__ PointSmem sm;
    const int lane = threadIdx.x;
    const int64_t slot = blockIdx.x;
    const float4 p = s_sorted[slot];
    const float3 x = make_float3(p.x, p.y, p.z);
    float W = 0.f, V = 0.f;
    int n_wait = 0, n_tested = 0, n_cand = 0, n_contrib = 0;
    auto batch = [&](const int* ids, int n) {
        if (lane < n) {
            const float4* rp = reinterpret_cast<const float4*>(recs + ids[lane]);
            const float4 r0 = __ldg(rp), r1 = __ldg(rp + 1), r2 = __ldg(rp + 2);
            const GaussB g = gauss_b(r0.x, r0.y, r0.z, r2.z, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r0, r0);
            const float dx = x.x - g.mx, dy = x.y - g.my, dz = x.z - g.mz;
            const float p2 =
                dx * fmaf(g.q0, dx, fmaf(g.q1, dy, g.q2 * dz)) + dy * fmaf(g.q3, dy, g.q4 * dz) + dz * (g.q5 * dz);
            if (p2 >= kLog2Floor && p2 <= 0.f) {
                const float wt = r0.w * ex2_approx(p2);
                W += wt;
                V = fmaf(wt, g.v, V);
                if (COUNT) n_contrib++;
            }
        }
        if (COUNT) n_cand += n;
        __syncwarp();
    };
    wide_walk<COUNT>(tree, x, x, 0xffffffffu, sm.walk, n_tested, [&](int leaf, bool valid) -> bool {
        bool h = false;
        if (valid) {
            const float4* q = tree.box[0] + 2 * (int64_t)leaf;
            h = box_overlap(__ldg(q), __ldg(q + 1), x, x);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, h);
        if (h) sm.cand[n_wait + __popc(m & lane_lt_mask())] = leaf;
        n_wait += __popc(m);
        __syncwarp();
        if (n_wait >= 32) {
            n_wait -= 32;
            batch(sm.cand + n_wait, 32);
        }
        return true;
    });
    if (n_wait > 0) batch(sm.cand, n_wait);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        W += __shfl_xor_sync(0xffffffffu, W, off);
        V += __shfl_xor_sync(0xffffffffu, V, off);
    }
    if (lane == 0) {
        const int orig = __float_as_int(p.w);
        const bool ok = !(W <= kWeightCutoff);
        const float o = ok ? V / W : -1.0f, w = ok ? W : 0.0f;
        out_cells[orig] = o;
        out_weights[orig] = w;
        if (out_sorted) out_sorted[slot] = make_float2(o, w);
    }
    if (COUNT) {
        const int c = __reduce_add_sync(0xffffffffu, n_contrib);
        if (lane == 0) {
            atomicAdd(&stats[0], (unsigned long long)n_cand);
            atomicAdd(&stats[1], (unsigned long long)c);
            atomicAdd(&stats[5], (unsigned long long)n_cand);
            atomicAdd(&stats[6], (unsigned long long)n_tested);
            atomicAdd(&stats[9], (unsigned long long)n_cand);
        }
    }
}

}  // namespace

cudaError_t launch_forward_points(const FwdArgs& a, cudaStream_t st) {
    if (a.S <= 0) return cudaSuccess;
    if (a.count)
        k_forward_points<true><<<(unsigned)a.S, 32, 0, st>>>(a.s_sorted, a.tree, a.recs, a.out_cells, a.out_weights,
                                                             a.out_sorted, a.stats);
    else
        k_forward_points<false><<<(unsigned)a.S, 32, 0, st>>>(a.s_sorted, a.tree, a.recs, a.out_cells, a.out_weights,
                                                              a.out_sorted, a.stats);
    note_launch();
    return cudaGetLastError();
}

}  // namespace gvc
