// fwd_blocks.cu -- forward evaluation of the mixture field in FP32 (replaces
// FORWARD::sampleRenderCUDA / renderCUDA + normalizeCUDA,
// diff-gaussian-rasterization/cuda_rasterizer/forward.cu:116-274).
//
// One warp owns R runs ("chains") of 32 Morton-sorted samples of a 128-sample block, one
// sample of each chain per lane, and does everything for them without a barrier: per block
// group (k_sample_blocks) it walks the tree of Gaussians with the group's box
// (wide_tree.cuh), takes 32 candidates at a time, loads one candidate's record per lane,
// tests its box and power window against each chain's rows of the group (cull.cuh), stages
// the records in shared memory and evaluates every candidate for the chains it can reach: the
// exact AABB test, the power, the window, ex2 and the sums, all in registers.  No atomics;
// the order of a sample's sum depends on the tree and the block alone.
//
// With the tensor-core kernels selected it walks the LBVH instead, by coarser groups: the
// order of the sums is then that of fwd_tc.cu's batches.  The tensor-core backward shifts its
// moments to a Gaussian's mean in FP32, and a last-bit change of W moves the scale gradient of
// a thin Gaussian by up to 1e-3, so its forward keeps to one order whatever walks come.
//
// What bounds it: the issue slots of the evaluated (chain, Gaussian) pairs, about 30
// instructions each, 3.5 evaluated lanes per contributing pair (300k x 2.1M; 64 rows behind a
// box test took 5.9).  A staged record is broadcast from shared memory, and a broadcast
// LDS.128 fills 512 bytes of registers, four cycles of the SM's shared-memory path: one chain
// per warp is bound by that (L1 at 89 %, 2.02 ms for 300k x 2.1M, even with two Gaussians per
// packed f32x2 step), four chains share each load.  Producer and consumer warps with a
// barrier pipeline took 1.94 ms for the same, this 1.38 ms; 2M x 16M 16.9 -> 11.1 ms; a 256^3
// grid x 500k 9.2 -> 5.4 ms; 200k x 1M clustered 0.43 -> 0.33 ms.
#include <cstddef>

#include "cta.cuh"
#include "cull.cuh"
#include "pair.cuh"

namespace gvc {

namespace {

// One warp per CTA: what is uniform over the warp then is uniform over the CTA, and a slow
// block holds back no other (2M x 16M: 10.9 ms, against 12.1 with four warps per CTA).
// Resident CTAs per SM asked of the register allocator: 28, 72 registers.
constexpr int kFwdMinCtas = 28;

struct FwdSmem {
    // per staged candidate: (mu, w), (s0..s3), (lo, s4), (hi, s5) with s = -q (pair.cuh), and
    // (v, bits of the chains it can reach)
    float4 rec[32][4];
    float2 vm[32];
    float4 chain[4][2];  // boxes (lo, hi) of the chains' rows of the current group
    float4 fine[8][2];   // boxes of the block's finer groups (candidate log)
    union {
        struct {
            int cand[64];  // at most 31 before a step of the walk adds up to 32
            WideStack walk;
        };
        struct {
            int lcand[kCandCap];
            int stack[kStackCap];
        };
    };
};

// Smaller where the LBVH is not walked.
constexpr size_t kWideSmem = offsetof(FwdSmem, walk) + sizeof(WideStack);

template <int R, bool COUNT>
struct BlockEval {
    FwdSmem& sm;
    const GaussRec* __restrict__ recs;
    float x[R], y[R], z[R], W[R], V[R];  // x NaN: no row of the current group
    CandLog log;
    int f0, f1;  // the finer groups of the current group
    int n_cand, n_contrib, n_lane;

    // whether a staged candidate contributes to this lane's row of chain k, and its weight
    __device__ __forceinline__ bool weight(float4 a, float4 s, float4 bl, float4 bh, int k, float& wt) {
        const bool inside = bl.x <= x[k] && x[k] <= bh.x && bl.y <= y[k] && y[k] <= bh.y && bl.z <= z[k] &&
                            z[k] <= bh.z;
        const float dx = x[k] - a.x, dy = y[k] - a.y, dz = z[k] - a.z;
        // every rounding spelled out: the compiler's choice of what to fuse would differ from one
        // instantiation to the next, and with it the last bit (see the top)
        float t = __fmul_rn(dx, fmaf(s.x, dx, fmaf(s.y, dy, __fmul_rn(s.z, dz))));
        t = fmaf(dy, fmaf(s.w, dy, __fmul_rn(bl.w, dz)), t);
        t = fmaf(dz, __fmul_rn(bh.w, dz), t);
        // t = -p2 is in the window [0, -kLog2Floor] iff its bits, as an unsigned number, are at
        // most the floor's (a negative t or a NaN has larger ones; t is never -0: the squares
        // enter it as +0)
        const bool c = inside && __float_as_uint(t) <= __float_as_uint(-kLog2Floor);
        wt = __fmul_rn(a.w, ex2_approx(-t));
        if (COUNT) {
            n_cand += inside;
            n_contrib += c;
        }
        return c;
    }
    __device__ __forceinline__ float pair(int j, int k, float& v) {
        float wt;
        v = sm.vm[j].x;
        const bool c = weight(sm.rec[j][0], sm.rec[j][1], sm.rec[j][2], sm.rec[j][3], k, wt);
        return c ? wt : 0.f;
    }

    // up to 32 candidates whose boxes overlap the group's
    __device__ __forceinline__ void operator()(const int* ids, int n) {
        const int lane = threadIdx.x & 31;
        uint32_t reach = 0, meets = 0;
        int id = 0;
        float4 r0, q, lo, hi;
        float v;
        if (lane < n) {
            id = ids[lane];
            const float4* rp = reinterpret_cast<const float4*>(recs + id);
            r0 = __ldg(rp);
            const float4 r1 = __ldg(rp + 1), r2 = __ldg(rp + 2);
            lo = __ldg(rp + 3);
            hi = __ldg(rp + 4);
            v = r2.z;
            const GaussB g = gauss_b(r0.x, r0.y, r0.z, v, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, lo, hi);
            const CullGauss c{g.mx, g.my, g.mz, g.q0, g.q1, g.q2, g.q3, g.q4, g.q5,
                              cull_allowance(g.q0, g.q1, g.q2, g.q3, g.q4, g.q5, false)};
#pragma unroll
            for (int k = 0; k < R; k++) {
                const float4 bl = sm.chain[k][0], bh = sm.chain[k][1];
                if (box_overlap(lo, hi, make_float3(bl.x, bl.y, bl.z), make_float3(bh.x, bh.y, bh.z)) &&
                    (r2.w != 0.f || !outside_window(c, bl, bh)))
                    reach |= 1u << k;
            }
            if (log.ids) {
                for (int b = f0; b < f1; b++) {
                    const float4 bl = sm.fine[b][0], bh = sm.fine[b][1];
                    if (box_overlap(lo, hi, make_float3(bl.x, bl.y, bl.z), make_float3(bh.x, bh.y, bh.z)) &&
                        (r2.w != 0.f || !outside_window(c, bl, bh)))
                        meets |= 1u << b;
                }
            }
            q = make_float4(-g.q0, -g.q1, -g.q2, -g.q3);
            lo.w = -g.q4;
            hi.w = -g.q5;
        }
        if (log.ids) log.append(n, id, meets);
        const uint32_t m = __ballot_sync(0xffffffffu, reach != 0u);
        if (reach) {
            const int p = __popc(m & lane_lt_mask());
            sm.rec[p][0] = r0;
            sm.rec[p][1] = q;
            sm.rec[p][2] = lo;
            sm.rec[p][3] = hi;
            sm.vm[p] = make_float2(v, __uint_as_float(reach));
        }
        const int np = __popc(m);
        if (COUNT) n_lane += 32 * (int)__reduce_add_sync(0xffffffffu, __popc(reach));
        __syncwarp();
        if constexpr (R == 1) {
            // every staged candidate is for the one chain: four at a time, for the latency of
            // a warp that has its scheduler to itself; added in order
            int j = 0;
            for (; j + 4 <= np; j += 4) {
                float wt[4], v4[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    wt[i] = pair(j + i, 0, v4[i]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    W[0] = __fadd_rn(W[0], wt[i]);
                    V[0] = fmaf(wt[i], v4[i], V[0]);
                }
            }
            for (; j < np; j++) {
                float vj;
                const float wt = pair(j, 0, vj);
                W[0] = __fadd_rn(W[0], wt);
                V[0] = fmaf(wt, vj, V[0]);
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < np; j++) {
                const float4 a = sm.rec[j][0], s = sm.rec[j][1], bl = sm.rec[j][2], bh = sm.rec[j][3];
                const float2 vm = sm.vm[j];
                const uint32_t chains = __float_as_uint(vm.y);
#pragma unroll
                for (int k = 0; k < R; k++) {
                    if (!(chains & (1u << k))) continue;  // warp-uniform
                    float wt;
                    if (weight(a, s, bl, bh, k, wt)) {
                        W[k] = __fadd_rn(W[k], wt);
                        V[k] = fmaf(wt, vm.x, V[k]);
                    }
                }
            }
        }
        __syncwarp();
    }
};

template <int R, bool LINKED, bool COUNT>
__global__ void __launch_bounds__(32, kFwdMinCtas)
    k_forward_blocks(const float4* __restrict__ s_sorted, int64_t S, const uint2* __restrict__ bdesc,
                     const float4* __restrict__ bboxes, const __grid_constant__ WideTree tree,
                     const BvhNode* __restrict__ nodes, const GaussRec* __restrict__ recs,
                     float* __restrict__ out_cells, float* __restrict__ out_weights, float2* __restrict__ out_sorted,
                     int32_t* __restrict__ clog, uint8_t* __restrict__ cmask, int32_t* __restrict__ cend,
                     const uint2* __restrict__ fdesc, const float4* __restrict__ fboxes, int* status,
                     unsigned long long* stats) {
    constexpr int kPerBlock = 4 / R;  // warps per block
    __shared__ __align__(16) unsigned char smem_raw[LINKED ? sizeof(FwdSmem) : kWideSmem];
    FwdSmem& sm = *reinterpret_cast<FwdSmem*>(smem_raw);
    const int lane = threadIdx.x;
    const int64_t unit = blockIdx.x;
    const int64_t blk = unit / kPerBlock;
    const int row0 = (int)(unit % kPerBlock) * R * 32;  // first row of this warp in its block
    if (blk * kBlockRows + row0 >= S) return;
    const uint2 bd = bdesc[blk];
    const int ng = group_count(bd);
    BlockEval<R, COUNT> ev{sm, recs};
#pragma unroll
    for (int k = 0; k < R; k++) ev.W[k] = ev.V[k] = 0.f;
    uint2 fd = make_uint2(0u, 0u);
    int nf = 0;
    if (LINKED && clog && row0 == 0) {
        ev.log.ids = clog + blk * kCandLogPerBlock;
        ev.log.masks = cmask + blk * kCandLogPerBlock;
        fd = fdesc[blk];
        nf = group_count(fd);
        if (lane < 2 * nf) sm.fine[lane >> 1][lane & 1] = fboxes[2 * blk * kBlockGroups + lane];
    }
    ev.f0 = ev.f1 = 0;
    int st = 0;
    ev.n_cand = ev.n_contrib = ev.n_lane = 0;
    int n_tested = 0, n_hits = 0;
#pragma unroll 1
    for (int g = 0; g < ng; g++) {
        const int ra = group_start(bd, g), rb = group_start(bd, g + 1);
        // none of this warp's rows (the log is the first warp's)
        if (R < 4 && (rb <= row0 || ra >= row0 + 32 * R) && !(LINKED && ev.log.ids)) continue;
        Box6 u = empty_box();
#pragma unroll
        for (int k = 0; k < R; k++) {
            const int r = row0 + 32 * k + lane;
            const bool in = r >= ra && r < rb && blk * kBlockRows + r < S;
            const float4 p = in ? s_sorted[blk * kBlockRows + r] : make_float4(NAN, NAN, NAN, 0.f);
            ev.x[k] = p.x;
            ev.y[k] = p.y;
            ev.z[k] = p.z;
            const Box6 b = warp_point_box(in, p.x, p.y, p.z);
            if (lane == 0) {
                sm.chain[k][0] = make_float4(b.lx, b.ly, b.lz, 0.f);
                sm.chain[k][1] = make_float4(b.hx, b.hy, b.hz, 0.f);
            }
            grow(u, b);
        }
        if (LINKED && ev.log.ids) {
            ev.f0 = ev.f1;
            while (ev.f1 < nf && group_start(fd, ev.f1) < rb) ev.f1++;
        }
        __syncwarp();
        if constexpr (LINKED) {
            // the whole group's box, whichever of its rows are this warp's: the order of the sums
            const float4 glo = bboxes[2 * (blk * kBlockGroups + g)], ghi = bboxes[2 * (blk * kBlockGroups + g) + 1];
            const float3 lo = make_float3(glo.x, glo.y, glo.z), hi = make_float3(ghi.x, ghi.y, ghi.z);
            TravCount tc;
            st |= warp_traverse(nodes, lo, hi, sm.stack, sm.lcand, ev, tc);
            if (COUNT) {
                n_hits += tc.leaves;
                n_tested += tc.nodes;
            }
        } else {
            const float3 lo = make_float3(u.lx, u.ly, u.lz), hi = make_float3(u.hx, u.hy, u.hz);
            int n_wait = 0;
            wide_walk<COUNT>(tree, lo, hi, 0xffffffffu, sm.walk, n_tested, [&](int leaf, bool valid) -> bool {
                bool h = false;
                if (valid) {
                    const float4* q = tree.box[0] + 2 * (int64_t)leaf;
                    h = box_overlap(__ldg(q), __ldg(q + 1), lo, hi);
                }
                const uint32_t m = __ballot_sync(0xffffffffu, h);
                if (h) sm.cand[n_wait + __popc(m & lane_lt_mask())] = leaf;
                n_wait += __popc(m);
                if (COUNT) n_hits += __popc(m);
                __syncwarp();
                if (n_wait >= 32) {
                    n_wait -= 32;
                    ev(sm.cand + n_wait, 32);
                }
                return true;
            });
            if (n_wait > 0) ev(sm.cand, n_wait);
        }
        ev.log.end_group(g);
    }
    if (LINKED && ev.log.ids) {
        if (st) ev.log.over = true;
        ev.log.finish(cend + blk * kBlockGroups, ng);
    }
    if (LINKED && st && lane == 0) atomicOr(status, st);
#pragma unroll
    for (int k = 0; k < R; k++) {
        const int64_t row = blk * kBlockRows + row0 + 32 * k + lane;
        if (row < S) {
            const int orig = __float_as_int(s_sorted[row].w);
            const bool ok = !(ev.W[k] <= kWeightCutoff);
            const float o = ok ? ev.V[k] / ev.W[k] : -1.0f, w = ok ? ev.W[k] : 0.0f;
            out_cells[orig] = o;
            out_weights[orig] = w;
            // the same pair in sorted order (coalesced), so that the backward's rows need not
            // gather them back
            if (out_sorted) out_sorted[row] = make_float2(o, w);
        }
    }
    if (COUNT) {
        unsigned long long a = (unsigned long long)ev.n_cand, c = (unsigned long long)ev.n_contrib;
        for (int off = 16; off > 0; off >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            c += __shfl_xor_sync(0xffffffffu, c, off);
        }
        if (lane == 0) {
            atomicAdd(&stats[0], a);
            atomicAdd(&stats[1], c);
            atomicAdd(&stats[5], (unsigned long long)n_hits);
            atomicAdd(&stats[6], (unsigned long long)n_tested);
            atomicAdd(&stats[9], (unsigned long long)ev.n_lane);
        }
    }
}

template <int R, bool LINKED, bool COUNT>
void launch_blocks(const FwdArgs& a, cudaStream_t st) {
    const int64_t units = (a.S + 32 * R - 1) / (32 * R);
    k_forward_blocks<R, LINKED, COUNT><<<(unsigned)units, 32, 0, st>>>(
        a.s_sorted, a.S, a.bdesc, a.bboxes, a.tree, a.nodes, a.recs, a.out_cells, a.out_weights, a.out_sorted, a.clog,
        a.cmask, a.cend, a.fdesc, a.fboxes, a.status, a.stats);
    note_launch();
}

}  // namespace

cudaError_t launch_forward_blocks(const FwdArgs& a, cudaStream_t st) {
    if (a.S <= 0) return cudaSuccess;
    if (a.nodes) {
        // 32 rows per warp for latency, the whole block per warp for throughput; the line
        // between them (and to launch_forward_cta) is forward_linked_rows'
        const bool whole = forward_linked_rows(a.S, a.P) == kBlockRows;
        if (whole) a.count ? launch_blocks<4, true, true>(a, st) : launch_blocks<4, true, false>(a, st);
        else a.count ? launch_blocks<1, true, true>(a, st) : launch_blocks<1, true, false>(a, st);
    } else {
        // Half a block per warp where whole blocks would leave the chip's 148 x 28 resident
        // warps partly idle: 20k Gaussians x 262k samples 96 against 114 us, x 1M 151 against 140.
        const bool whole = a.S >= (int64_t)148 * kFwdMinCtas * kBlockRows;
        if (whole) a.count ? launch_blocks<4, false, true>(a, st) : launch_blocks<4, false, false>(a, st);
        else a.count ? launch_blocks<2, false, true>(a, st) : launch_blocks<2, false, false>(a, st);
    }
    return cudaGetLastError();
}

}  // namespace gvc
