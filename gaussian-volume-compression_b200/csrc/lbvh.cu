// lbvh.cu -- on-device LBVH construction: 30-bit Morton keys, stable LSD radix sort
// (8-bit digits, warp-aggregated stable ranking; one kernel per pass with decoupled
// look-back, or per-pass block histograms + scan + scatter where no status word is
// given), and the binary radix tree built and refitted bottom-up.
//
// Replaces cuBQL::cuda::radixBuilder as called from
// diff-gaussian-rasterization/cuda_rasterizer/rasterizer_impl.cu:78-83 (Gaussian AABBs)
// and diff-gaussian-rasterization/ext.cu:50-54 (sample points).  The declared ordering
// (keys, tie-break, tree) is restated on the CPU by the oracle and checked bit for bit.
#include "lbvh.cuh"

namespace gvc {

// ----------------------------------------------------------------------------------
// Ordered float <-> uint mapping for atomic min/max of floats.
// ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
    uint32_t b = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
    return __uint_as_float(b);
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__device__ __forceinline__ uint32_t quant10(float c, float lo, float scale) {
    float t = __fmul_rn(__fsub_rn(c, lo), scale);
    if (!(t >= 0.0f)) return 0u;
    if (t >= 1023.0f) return 1023u;
    return (uint32_t)t;
}

// Grid of 1024^3 cells over the centroids' bounds (ordered integers).
struct MortonGrid {
    float lo[3], scale[3];
    __device__ __forceinline__ void set(const uint32_t (&l)[3], const uint32_t (&h)[3]) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
            lo[a] = scale[a] = 0.f;
            if (l[a] == 0xffffffffu) continue;  // every centroid was NaN
            lo[a] = ord2f(l[a]);
            const float ext = __fsub_rn(ord2f(h[a]), lo[a]);
            scale[a] = ext > 0.0f ? __fdiv_rn(1024.0f, ext) : 0.0f;
        }
    }
    __device__ __forceinline__ uint32_t key(const float (&c)[3]) const {
        return expand10(quant10(c[0], lo[0], scale[0])) | (expand10(quant10(c[1], lo[1], scale[1])) << 1) |
               (expand10(quant10(c[2], lo[2], scale[2])) << 2);
    }
};

// Centroid of box i ((lo + hi) * 0.5f) or the point itself.
struct BoxSrc {
    const float4* boxes;  // [n][2] lo, hi
    __device__ __forceinline__ void centroid(int64_t i, float c[3]) const {
        float4 lo = boxes[2 * i], hi = boxes[2 * i + 1];
        c[0] = __fmul_rn(__fadd_rn(lo.x, hi.x), 0.5f);
        c[1] = __fmul_rn(__fadd_rn(lo.y, hi.y), 0.5f);
        c[2] = __fmul_rn(__fadd_rn(lo.z, hi.z), 0.5f);
    }
};
struct PointSrc {
    const float* pts;  // [n][3]
    // an infinite coordinate counts as none (NaN): in the bounds it would leave every point with
    // key 0, in no order at all
    static __device__ __forceinline__ float finite(float c) { return isfinite(c) ? c : NAN; }
    __device__ __forceinline__ void centroid(int64_t i, float c[3]) const {
        // (p + p) * 0.5f == p exactly for finite p, as for a degenerate box
        float x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
        c[0] = finite(__fmul_rn(__fadd_rn(x, x), 0.5f));
        c[1] = finite(__fmul_rn(__fadd_rn(y, y), 0.5f));
        c[2] = finite(__fmul_rn(__fadd_rn(z, z), 0.5f));
    }
};

// Bounds of the centroids as ordered integers: [axis] the complement of the least, [3 + axis]
// the greatest, so that both are maxima over words that start at zero.
template <class Src>
__global__ void __launch_bounds__(256) k_bounds(Src src, int64_t n, uint32_t* bounds) {
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float c[3];
        src.centroid(i, c);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (c[a] == c[a]) {  // NaN centroids do not move the bounds (fminf semantics)
                uint32_t o = f2ord(c[a]);
                mn[a] = min(mn[a], o);
                mx[a] = max(mx[a], o);
            }
        }
    }
    // One atomic per bound and block: all of them go to six words of one line, and one per
    // warp of 1184 blocks (57k atomics) took 36-47 us at any n.
    __shared__ uint32_t s_mn[8][3], s_mx[8][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const uint32_t lo = __reduce_min_sync(0xffffffffu, mn[a]), hi = __reduce_max_sync(0xffffffffu, mx[a]);
        if (lane == 0) {
            s_mn[warp][a] = lo;
            s_mx[warp][a] = hi;
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int a = threadIdx.x;
        uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            lo = min(lo, s_mn[w][a]);
            hi = max(hi, s_mx[w][a]);
        }
        atomicMax(&bounds[a], ~lo);
        atomicMax(&bounds[3 + a], hi);
    }
}

// Keys, and with HIST the digit counts of all four passes of the sort (ghist[pass * 256 +
// digit], zeroed by the caller), which would otherwise be another launch and pass over the keys.
template <class Src, bool HIST>
__global__ void __launch_bounds__(256) k_keys(Src src, int64_t n, const uint32_t* __restrict__ bounds,
                                              uint32_t* __restrict__ keys, uint32_t* __restrict__ ghist) {
    __shared__ uint32_t cnt[HIST ? 4 * 256 : 1];
    if (HIST) {
        for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) cnt[i] = 0u;
        __syncthreads();
    }
    MortonGrid grid;
    {
        const uint32_t l[3] = {~bounds[0], ~bounds[1], ~bounds[2]}, h[3] = {bounds[3], bounds[4], bounds[5]};
        grid.set(l, h);
    }
    // several keys per thread where there are many: the scales' divisions cost more than a key
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
        float c[3];
        src.centroid(i, c);
        const uint32_t k = grid.key(c);
        keys[i] = k;
        if (HIST) {
            atomicAdd(&cnt[k & 255u], 1u);
            atomicAdd(&cnt[256 + ((k >> 8) & 255u)], 1u);
            atomicAdd(&cnt[512 + ((k >> 16) & 255u)], 1u);
            atomicAdd(&cnt[768 + (k >> 24)], 1u);
        }
    }
    if (HIST) {
        __syncthreads();
        for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
            const uint32_t v = cnt[i];
            if (v) atomicAdd(&ghist[i], v);
        }
    }
}

// ----------------------------------------------------------------------------------
// Stable LSD radix sort of (uint32 key, int32 value) pairs, 8-bit digits.
//   tile = 8 warps x 16 iterations x 32 lanes = 4096 elements per block.
//   per pass: k_rs_hist (per-block digit counts of the current order),
//   k_rs_scan (per-digit exclusive scan over blocks + digit totals),
//   k_rs_scatter (stable ranks: (warp, iteration, lane) = input order).
// ----------------------------------------------------------------------------------

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__global__ void __launch_bounds__(256) k_rs_hist(const uint32_t* __restrict__ keys, int64_t n, int nb, int pass,
                                                 uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[256];
    for (int t = threadIdx.x; t < 256; t += blockDim.x) cnt[t] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = 8 * pass;
    int64_t base = (int64_t)blockIdx.x * kRsTile + (int64_t)warp * (kRsIters * 32);
#pragma unroll 4
    for (int it = 0; it < kRsIters; it++) {
        int64_t idx = base + it * 32 + lane;
        bool valid = idx < n;
        uint32_t key = valid ? keys[idx] : 0u;
        uint32_t d = (key >> shift) & 255u;
        uint32_t tag = valid ? d : (256u + lane);
        uint32_t peers = __match_any_sync(0xffffffffu, tag);
        if (valid && (__ffs(peers) - 1) == lane) atomicAdd(&cnt[d], (uint32_t)__popc(peers));
    }
    __syncthreads();
    for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[(int64_t)d * nb + blockIdx.x] = cnt[d];
}

// grid (256 digits), 1024 threads: in-place exclusive scan of one digit's row.
__global__ void __launch_bounds__(1024) k_rs_scan(uint32_t* __restrict__ hist, int nb, uint32_t* __restrict__ totals) {
    const int d = blockIdx.x;
    uint32_t* row = hist + (int64_t)d * nb;
    const int per = (nb + blockDim.x - 1) / blockDim.x;
    const int b0 = threadIdx.x * per;
    uint32_t local = 0;
    for (int k = 0; k < per; k++) {
        int b = b0 + k;
        if (b < nb) local += row[b];
    }
    __shared__ uint32_t wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = local;
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t v = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0u;
        uint32_t vi = v;
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xffffffffu, vi, off);
            if (lane >= off) vi += t;
        }
        wsum[lane] = vi - v;  // exclusive warp offsets
        if (lane == 31) totals[d] = vi;
    }
    __syncthreads();
    uint32_t run = wsum[warp] + incl - local;
    for (int k = 0; k < per; k++) {
        int b = b0 + k;
        if (b < nb) {
            uint32_t v = row[b];
            row[b] = run;
            run += v;
        }
    }
}

__global__ void __launch_bounds__(256) k_rs_scatter(const uint32_t* __restrict__ keys_in,
                                                    const int32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
                                                    int32_t* __restrict__ vals_out, int64_t n, int nb, int pass,
                                                    const uint32_t* __restrict__ hist,
                                                    const uint32_t* __restrict__ totals) {
    __shared__ uint32_t wcnt[kRsWarps][256];
    __shared__ uint32_t dbase[256];
    __shared__ uint32_t bstart[256];
    __shared__ uint32_t wsum[kRsWarps];
    __shared__ uint32_t skey[kRsTile];
    __shared__ int32_t sval[kRsTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = 8 * pass;
    for (int t = threadIdx.x; t < kRsWarps * 256; t += blockDim.x) (&wcnt[0][0])[t] = 0;
    // digit bases: exclusive scan of the 256 digit totals + this block's row offset
    if (warp == 0) {
        uint32_t run = 0;
        for (int chunk = 0; chunk < 8; chunk++) {
            int d = chunk * 32 + lane;
            uint32_t v = totals[d];
            uint32_t incl = v;
            for (int off = 1; off < 32; off <<= 1) {
                uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += t;
            }
            dbase[d] = run + incl - v + hist[(int64_t)d * nb + blockIdx.x];
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRsTile + (int64_t)warp * (kRsIters * 32);
    uint32_t kreg[kRsIters];
    int32_t vreg[kRsIters];
    uint32_t rreg[kRsIters];  // (local rank << 8) | digit, or 0xffffffff if invalid
#pragma unroll
    for (int it = 0; it < kRsIters; it++) {
        int64_t idx = base + it * 32 + lane;
        bool valid = idx < n;
        uint32_t key = valid ? keys_in[idx] : 0u;
        int32_t val = valid ? (vals_in ? vals_in[idx] : (int32_t)idx) : 0;
        uint32_t d = (key >> shift) & 255u;
        uint32_t tag = valid ? d : (256u + lane);
        uint32_t peers = __match_any_sync(0xffffffffu, tag);
        uint32_t rank = __popc(peers & lanemask_lt());
        uint32_t pre = valid ? wcnt[warp][d] : 0u;
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) wcnt[warp][d] = pre + __popc(peers);
        __syncwarp();
        kreg[it] = key;
        vreg[it] = val;
        rreg[it] = valid ? (((pre + rank) << 8) | d) : 0xffffffffu;
    }
    __syncthreads();
    // exclusive prefix over warps for each digit; run = this block's count of digit d
    uint32_t run = 0;
    {
        const int d = threadIdx.x;  // 256 threads == 256 digits
#pragma unroll
        for (int w = 0; w < kRsWarps; w++) {
            const uint32_t t = wcnt[w][d];
            wcnt[w][d] = run;
            run += t;
        }
    }
    // block-local start of each digit: exclusive scan of the 256 counts
    {
        uint32_t incl = run;
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t wbase = 0;
        for (int w = 0; w < warp; w++) wbase += wsum[w];
        bstart[threadIdx.x] = wbase + incl - run;
    }
    __syncthreads();
    // place every key at its block-local sorted position, then write the block out in that
    // order: consecutive threads write consecutive addresses of each digit's run
#pragma unroll
    for (int it = 0; it < kRsIters; it++) {
        const uint32_t r = rreg[it];
        if (r != 0xffffffffu) {
            const uint32_t d = r & 255u;
            const uint32_t sp = bstart[d] + wcnt[warp][d] + (r >> 8);
            skey[sp] = kreg[it];
            sval[sp] = vreg[it];
        }
    }
    __syncthreads();
    const int64_t rem = n - (int64_t)blockIdx.x * kRsTile;
    const int cnt = rem < kRsTile ? (int)rem : kRsTile;
    for (int sp = threadIdx.x; sp < cnt; sp += blockDim.x) {
        const uint32_t key = skey[sp];
        const uint32_t d = (key >> shift) & 255u;
        const uint32_t pos = dbase[d] + ((uint32_t)sp - bstart[d]);
        keys_out[pos] = key;
        vals_out[pos] = sval[sp];
    }
}

// ----------------------------------------------------------------------------------
// One kernel per pass (the onesweep scheme of Adinets & Merrill 2022): the digit counts
// of all four passes come from one read of the keys (k_os_hist); in each pass the tiles
// take tickets in the order their blocks start, rank their keys as k_rs_scatter does,
// publish their per-digit counts and find the counts of every tile before them by
// decoupled look-back (Merrill & Garland 2016): the words of the preceding tiles are
// read from the nearest backwards, adding aggregates until an inclusive prefix is met.
// A word packs a 2-bit state (not ready / aggregate / inclusive) with a 30-bit count, so
// n < 2^30.  A tile only waits on tiles with smaller tickets, whose blocks are already
// running and wait only on tiles before their own, so the look-back ends; its spin is
// bounded all the same (kStatusTimeout; the order is invalid then, and may hold what its
// buffers held before: order_at).  Same stable order as the
// three-kernel passes: tile t holds keys [t * kRsTile, (t + 1) * kRsTile) of the pass's
// input whatever block takes ticket t.
// ----------------------------------------------------------------------------------
constexpr uint32_t kOsAggregate = 1u << 30;
constexpr uint32_t kOsInclusive = 2u << 30;
constexpr uint32_t kOsCount = (1u << 30) - 1u;
constexpr long long kOsSpinCycles = 200000000LL;  // ~0.1 s at 2 GHz
// look-back words loaded together: 16M keys 122 us per pass with 4, 125 with 8, 130 with 16, 143
// with 32; 4M 38.8 / 39.3 / 41.8 / -
constexpr int kOsWindow = 4;

__device__ __forceinline__ uint32_t ld_relaxed_gpu(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_gpu(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ghist[pass * 256 + digit] += count over keys[0, n) (ghist zeroed by the caller).
__global__ void __launch_bounds__(256) k_os_hist(const uint32_t* __restrict__ keys, int64_t n,
                                                 uint32_t* __restrict__ ghist) {
    __shared__ uint32_t cnt[4 * 256];
    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) cnt[i] = 0u;
    __syncthreads();
    const int64_t nv = n >> 2;  // uint4 loads (the buffer is 256-byte aligned), then the tail
    const uint4* k4 = reinterpret_cast<const uint4*>(keys);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv + 4; i += stride) {
        uint32_t k[4];
        int m = 0;
        if (i < nv) {
            const uint4 q = k4[i];
            k[0] = q.x;
            k[1] = q.y;
            k[2] = q.z;
            k[3] = q.w;
            m = 4;
        } else if (4 * nv + (i - nv) < n) {
            k[0] = keys[4 * nv + (i - nv)];
            m = 1;
        }
        for (int j = 0; j < m; j++) {
            atomicAdd(&cnt[k[j] & 255u], 1u);
            atomicAdd(&cnt[256 + ((k[j] >> 8) & 255u)], 1u);
            atomicAdd(&cnt[512 + ((k[j] >> 16) & 255u)], 1u);
            atomicAdd(&cnt[768 + (k[j] >> 24)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 256; i += blockDim.x) {
        const uint32_t v = cnt[i];
        if (v) atomicAdd(&ghist[i], v);
    }
}

// Rank of this lane's digit (the low 8 bits of d) among the warp's valid ones so far, counted
// in cnt; warp-collective.
__device__ __forceinline__ uint32_t digit_rank(bool valid, uint32_t d, uint32_t* cnt) {
    const int lane = threadIdx.x & 31;
    // the lanes with this lane's digit: eight votes (match.any took 130 cycles of an SM)
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int bit = 0; bit < 8; bit++) {
        const bool one = (d >> bit) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    // the first of them adds to the warp's count; the sum before is the rank of that lane.  Rounds
    // may add to one count from different lanes: the barrier orders their additions (a shuffle
    // orders no memory), and so the ranks, on which the sort's stability rests.
    __syncwarp();
    const int leader = __ffs(peers) - 1;
    uint32_t pre = 0;
    if (valid && lane == leader) pre = atomicAdd(cnt + (d & 255u), (uint32_t)__popc(peers));
    pre = __shfl_sync(0xffffffffu, pre, leader & 31);
    return pre + __popc(peers & lanemask_lt());
}

// What bounds a pass: the instructions of the ranking and the look-back, at few warps per
// scheduler (43 KB of shared memory and 80 registers: three blocks per SM; four at 64 registers are as fast), and with
// a handful of tiles their latency.  Loads all issued before the first key is ranked, votes and
// one shared-memory addition a round in place of match.any, a read and a write, 32-bit bounds,
// and a window of aggregates added whole: per pass 12.7 -> 7.3 us for 4096 keys, 17.2 -> 9.1
// for 200k, 33 -> 25 for 2M, 60 -> 39 for 4M, 190 -> 122 for 16M.
__global__ void __launch_bounds__(256, 3) k_os_scatter(const uint32_t* __restrict__ keys_in,
                                                       const int32_t* __restrict__ vals_in,
                                                       uint32_t* __restrict__ keys_out, int32_t* __restrict__ vals_out,
                                                       int64_t n, int pass, const uint32_t* __restrict__ ghist,
                                                       uint32_t* __restrict__ look, uint32_t* __restrict__ ticket,
                                                       int* __restrict__ status) {
    __shared__ uint32_t wcnt[kRsWarps][256];  // counts, then tile-local starts of (warp, digit)
    __shared__ uint32_t gpos[256];            // a key's position in the output less its tile-local slot
    __shared__ uint32_t wsum[kRsWarps], dsum[kRsWarps];
    __shared__ uint32_t skey[kRsTile];
    __shared__ int32_t sval[kRsTile];
    __shared__ uint32_t s_tile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int shift = 8 * pass;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    const uint32_t dcount = ghist[pass * 256 + threadIdx.x];
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) wcnt[w][threadIdx.x] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t first = tile * kRsTile + warp * (kRsIters * 32) + lane;  // this lane's first key
    // the lane's keys: rounds it with 32 it < rem
    const int rem = n - first < kRsIters * 32 ? (int)(n - first) : kRsIters * 32;
    const uint32_t* kp = keys_in + first;
    uint32_t kreg[kRsIters];
    int32_t vreg[kRsIters];
#pragma unroll
    for (int it = 0; it < kRsIters; it++) kreg[it] = 32 * it < rem ? __ldcs(kp + 32 * it) : 0u;
    if (vals_in) {
        const int32_t* vp = vals_in + first;
#pragma unroll
        for (int it = 0; it < kRsIters; it++) vreg[it] = 32 * it < rem ? __ldcs(vp + 32 * it) : 0;
    } else {
#pragma unroll
        for (int it = 0; it < kRsIters; it++) vreg[it] = (int32_t)first + 32 * it;
    }
    // first position of each digit in the output: exclusive scan of the pass's digit counts
    uint32_t gstart = dcount;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, gstart, off);
        if (lane >= off) gstart += t;
    }
    if (lane == 31) dsum[warp] = gstart;
    gstart -= dcount;
    uint32_t rreg[kRsIters / 2];  // ranks among the warp's keys of the same digit, two per word
#pragma unroll
    for (int it = 0; it < kRsIters; it++) {
        const uint32_t rank = digit_rank(32 * it < rem, kreg[it] >> shift, wcnt[warp]);
        rreg[it / 2] = (it & 1) ? (rreg[it / 2] | (rank << 16)) : (rank & 0xffffu);
    }
    __syncthreads();
    // run = this tile's count of digit d
    const int d = threadIdx.x;  // 256 threads == 256 digits
    uint32_t cw[kRsWarps], run = 0;
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) {
        cw[w] = run;
        run += wcnt[w][d];
    }
    // publish it at once, so that later tiles can pass over it
    uint32_t* mine = look + tile * 256 + d;
    st_relaxed_gpu(mine, (tile == 0 ? kOsInclusive : kOsAggregate) | run);
    // tile-local start of each digit: exclusive scan of the 256 counts
    uint32_t lstart = run;
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, lstart, off);
        if (lane >= off) lstart += t;
    }
    if (lane == 31) wsum[warp] = lstart;
    __syncthreads();
    lstart -= run;
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) {
        if (w < warp) {
            lstart += wsum[w];
            gstart += dsum[w];
        }
    }
#pragma unroll
    for (int w = 0; w < kRsWarps; w++) wcnt[w][d] = lstart + cw[w];
    __syncthreads();
    // the keys go to their tile-local sorted slots before the look-back (their registers
    // are free for the look-back's window)
#pragma unroll
    for (int it = 0; it < kRsIters; it++) {
        if (32 * it < rem) {
            const uint32_t sp = wcnt[warp][(kreg[it] >> shift) & 255u] + ((rreg[it / 2] >> (16 * (it & 1))) & 0xffffu);
            skey[sp] = kreg[it];
            sval[sp] = vreg[it];
        }
    }
    // look back for the count of digit d in all tiles before this one, kOsWindow words
    // loaded together: aggregates are added until an inclusive prefix is met; a tile not
    // ready yet ends this window (the words before it are kept) and is read again
    if (tile > 0) {
        uint32_t excl = 0;
        int k = (int)tile - 1;  // nearest tile not accounted for yet
        const uint32_t* lp = look + d;
        const long long t0 = clock64();
        bool ok = true;
        while (true) {
            uint32_t v[kOsWindow], every = ~0u, any = 0u, add = 0u;
#pragma unroll
            for (int i = 0; i < kOsWindow; i++)
                v[i] = k >= i ? ld_relaxed_gpu(lp + (int64_t)(k - i) * 256) : kOsInclusive;
#pragma unroll
            for (int i = 0; i < kOsWindow; i++) {
                every &= v[i];
                any |= v[i];
                add += v[i];
            }
            if ((every & kOsAggregate) && !(any & kOsInclusive)) {
                // aggregates throughout: their states, 2^30 each, vanish from the sum
                static_assert((uint64_t)kOsWindow * kOsAggregate % (uint64_t(1) << 32) == 0, "states vanish");
                excl += add;
                k -= kOsWindow;
                continue;
            }
            add = 0;
            int taken = 0;
            bool inclusive = false, blocked = false;
#pragma unroll
            for (int i = 0; i < kOsWindow; i++) {
                if (!inclusive && !blocked) {
                    const uint32_t state = v[i] & ~kOsCount;
                    if (state == 0u) {
                        blocked = true;
                    } else {
                        add += v[i] & kOsCount;
                        taken++;
                        inclusive = state == kOsInclusive;
                    }
                }
            }
            excl += add;
            if (inclusive) break;
            k -= taken;
            if (blocked) {
                if (clock64() - t0 > kOsSpinCycles) {
                    ok = false;
                    break;
                }
                __nanosleep(32);
            }
        }
        if (!ok) atomicOr(status, kStatusTimeout);
        st_relaxed_gpu(mine, kOsInclusive | ((excl + run) & kOsCount));
        gstart += excl;
    }
    gpos[d] = gstart - lstart;
    __syncthreads();
    const int cnt = n - tile * kRsTile < kRsTile ? (int)(n - tile * kRsTile) : kRsTile;
#pragma unroll 4
    for (int sp = threadIdx.x; sp < cnt; sp += 256) {
        const uint32_t key = skey[sp];
        const uint32_t pos = gpos[(key >> shift) & 255u] + (uint32_t)sp;
        // false only after a look-back gave up: the keys of a pass that lost some to the slots it
        // left unwritten no longer match the digit counts taken before the first pass
        if (pos < (uint32_t)n) {
            keys_out[pos] = key;
            vals_out[pos] = sval[sp];
        }
    }
}

// Words of the one-kernel-per-pass sort: digit counts [4][256], then 64 for the tickets [4] and,
// from kOsBounds, the centroid bounds; then a look-back word per (tile, digit) and pass.
constexpr int kOsHead = 4 * 256 + 64;
constexpr int kOsBounds = 4 * 256 + 8;

// Passes over L.keys; the words are zeroed and the digit counts filled in, the tickets start at
// `withheld` (test hook: the tiles before it never run, and those after wait for them in vain).
static cudaError_t radix_sort_onesweep(Lbvh& L, int64_t n, int withheld, cudaStream_t st) {
    const int64_t T = (n + kRsTile - 1) / kRsTile;
    cudaError_t e;
    if ((e = L.keys_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    uint32_t* ghist = L.onesweep.as<uint32_t>();
    uint32_t* tickets = ghist + 4 * 256;
    uint32_t* look0 = ghist + kOsHead;
    uint32_t* kin = L.keys.as<uint32_t>();
    uint32_t* kout = L.keys_alt.as<uint32_t>();
    int32_t* vin = nullptr;
    int32_t* vout = L.perm_alt.as<int32_t>();
    for (int pass = 0; pass < 4; pass++) {
        k_os_scatter<<<(unsigned)(T - withheld), 256, 0, st>>>(kin, vin, kout, vout, n, pass, ghist,
                                                  look0 + (size_t)pass * 256 * (size_t)T, tickets + pass,
                                                  L.status); gvc::note_launch();
        // ping-pong as in radix_sort_pairs: the result ends in L.keys / L.perm
        uint32_t* tk = kin;
        kin = kout;
        kout = tk;
        vin = vout;
        vout = (vout == L.perm_alt.as<int32_t>()) ? L.perm.as<int32_t>() : L.perm_alt.as<int32_t>();
    }
    return cudaGetLastError();
}

// The three-kernel passes over L.keys.
static cudaError_t radix_sort_pairs(Lbvh& L, int64_t n, cudaStream_t st) {
    const int nb = (int)((n + kRsTile - 1) / kRsTile);
    cudaError_t e;
    if ((e = L.keys_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.hist.ensure(LbvhBytes::hist(n))) != cudaSuccess) return e;
    uint32_t* hist = L.hist.as<uint32_t>();
    uint32_t* totals = hist + 256 * (size_t)nb;
    uint32_t* kin = L.keys.as<uint32_t>();
    uint32_t* kout = L.keys_alt.as<uint32_t>();
    int32_t* vin = nullptr;
    int32_t* vout = L.perm_alt.as<int32_t>();
    for (int pass = 0; pass < 4; pass++) {
        k_rs_hist<<<nb, 256, 0, st>>>(kin, n, nb, pass, hist); gvc::note_launch();
        k_rs_scan<<<256, 1024, 0, st>>>(hist, nb, totals); gvc::note_launch();
        k_rs_scatter<<<nb, 256, 0, st>>>(kin, vin, kout, vout, n, nb, pass, hist, totals); gvc::note_launch();
        // ping-pong: pass 0 keys->alt, 1 alt->keys, 2 keys->alt, 3 alt->keys
        uint32_t* tk = kin;
        kin = kout;
        kout = tk;
        vin = vout;
        vout = (vout == L.perm_alt.as<int32_t>()) ? L.perm.as<int32_t>() : L.perm_alt.as<int32_t>();
    }
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_gather_u32(int64_t n, const uint32_t* __restrict__ src,
                                                    int32_t* __restrict__ perm, uint32_t* __restrict__ dst) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[order_at(perm, i, n)];
}

cudaError_t radix_sort_words(Lbvh& L, int64_t n, const uint32_t* const* words, const int* bits, int nwords,
                             cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int nb = (int)((n + kRsTile - 1) / kRsTile);
    cudaError_t e;
    if ((e = L.keys.ensure(sizeof(uint32_t) * n)) != cudaSuccess) return e;
    if ((e = L.keys_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.hist.ensure(LbvhBytes::hist(n))) != cudaSuccess) return e;
    uint32_t* hist = L.hist.as<uint32_t>();
    uint32_t* totals = hist + 256 * (size_t)nb;
    uint32_t* kin = L.keys.as<uint32_t>();
    uint32_t* kout = L.keys_alt.as<uint32_t>();
    int32_t* vin = nullptr;  // identity before the first pass
    int32_t* vout = L.perm_alt.as<int32_t>();
    const unsigned gb = (unsigned)((n + 255) / 256);
    // one kernel per pass (as radix_sort_pairs) where a status word takes the look-back's report
    const bool os = L.status && n <= (int64_t)kOsCount;
    const size_t os_head = sizeof(uint32_t) * (4 * 256 + 64);
    const size_t os_look = sizeof(uint32_t) * 256 * (size_t)nb;
    if (os && (e = L.onesweep.ensure(os_head + 4 * os_look)) != cudaSuccess) return e;
    uint32_t* ghist = os ? L.onesweep.as<uint32_t>() : nullptr;
    for (int w = 0; w < nwords; w++) {
        const int passes = (bits[w] + 7) / 8;
        if (passes <= 0) continue;
        // this word's keys in the current order
        if (vin) {
            k_gather_u32<<<gb, 256, 0, st>>>(n, words[w], vin, kin); gvc::note_launch();
        } else if ((e = cudaMemcpyAsync(kin, words[w], sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st)) !=
                   cudaSuccess) {
            return e;
        }
        if (os) {
            if ((e = cudaMemsetAsync(ghist, 0, os_head + (size_t)passes * os_look, st)) != cudaSuccess) return e;
            k_os_hist<<<(unsigned)(nb < 148 * 4 ? nb : 148 * 4), 256, 0, st>>>(kin, n, ghist); gvc::note_launch();
        }
        for (int pass = 0; pass < passes; pass++) {
            if (os) {
                k_os_scatter<<<(unsigned)nb, 256, 0, st>>>(kin, vin, kout, vout, n, pass, ghist,
                                                           ghist + os_head / sizeof(uint32_t) +
                                                               (size_t)pass * 256 * (size_t)nb,
                                                           ghist + 4 * 256 + pass, L.status); gvc::note_launch();
            } else {
                k_rs_hist<<<nb, 256, 0, st>>>(kin, n, nb, pass, hist); gvc::note_launch();
                k_rs_scan<<<256, 1024, 0, st>>>(hist, nb, totals); gvc::note_launch();
                k_rs_scatter<<<nb, 256, 0, st>>>(kin, vin, kout, vout, n, nb, pass, hist, totals); gvc::note_launch();
            }
            uint32_t* tk = kin;
            kin = kout;
            kout = tk;
            int32_t* tv = vin;
            vin = vout;
            vout = tv ? tv : (vin == L.perm_alt.as<int32_t>() ? L.perm.as<int32_t>() : L.perm_alt.as<int32_t>());
        }
    }
    if (!vin) return cudaErrorInvalidValue;  // no word had any bits
    if (vin != L.perm.as<int32_t>() &&
        (e = cudaMemcpyAsync(L.perm.ptr, vin, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
        return e;
    return cudaGetLastError();
}

// ----------------------------------------------------------------------------------
// The binary radix tree over the sorted keys (Karras 2012, "Maximizing parallelism in the
// construction of BVHs, octrees and k-d trees"; equal keys told apart by position), built
// and refitted bottom-up in one kernel (the scheme of Apetrei 2014, "Fast and simple
// agglomerative LBVH construction").  The node that splits its leaves after leaf s is stored
// at s + 1, the root once more at 0, where every walk starts.  A thread per leaf carries a
// subtree upwards: the neighbouring key with the longer common prefix tells whether the
// subtree is its parent's left or right child, and so the parent's split; the thread writes
// its half of the parent (box, link, far end of its leaves) and goes on if the other half is
// there already.
// Topology kernel, refit and packing by themselves took 68 + 159 + 64 us for 2M leaves and
// 15 + 34 + 10 us for 200k, this 178 and 38.
// ----------------------------------------------------------------------------------
struct BoxLeaf {
    const float4* boxes;  // [n][2] lo, hi
    __device__ __forceinline__ void box(int i, float4& lo, float4& hi) const {
        lo = __ldg(boxes + 2 * (int64_t)i);
        hi = __ldg(boxes + 2 * (int64_t)i + 1);
    }
};
struct PointLeaf {
    const float4* pts;
    __device__ __forceinline__ void box(int i, float4& lo, float4& hi) const { lo = hi = __ldg(pts + i); }
};

template <class Leaf>
__global__ void __launch_bounds__(256) k_lbvh_build(int n, const uint32_t* __restrict__ keys, Leaf leaf,
                                                    BvhNode* nodes, uint32_t* flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 lo, hi;
    leaf.box(i, lo, hi);
    uint32_t link = (uint32_t)i | kLeafBit;
    float4* root = reinterpret_cast<float4*>(nodes);
    if (n == 1) {
        // a single leaf: a root whose right child can never overlap anything
        root[0] = make_float4(lo.x, lo.y, lo.z, __uint_as_float(link));
        root[1] = make_float4(hi.x, hi.y, hi.z, 0.f);
        root[2] = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
        root[3] = make_float4(-INFINITY, -INFINITY, -INFINITY, __uint_as_float(link));
        return;
    }
    int l = i, r = i;  // the subtree's leaves
    // common prefixes across its ends (-1 past the tree's); never equal, except alone
    int dl = l > 0 ? lbvh_delta(keys, l - 1, l) : -1, dr = r < n - 1 ? lbvh_delta(keys, r, r + 1) : -1;
    while (true) {
        const bool left = dr > dl;
        const int s = left ? r : l - 1;  // the parent's split
        float4* node = reinterpret_cast<float4*>(nodes + s + 1);
        const float4 h0 = make_float4(lo.x, lo.y, lo.z, left ? __uint_as_float(link) : __int_as_float(r));
        const float4 h1 = make_float4(hi.x, hi.y, hi.z, left ? __int_as_float(l) : __uint_as_float(link));
        __stcg(node + (left ? 0 : 2), h0);
        __stcg(node + (left ? 1 : 3), h1);
        // acquire-release at GPU scope: the first child's half is visible to the second arriver
        uint32_t old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(flags + s) : "memory");
        if (old == 0) return;
        const float4 o0 = __ldcg(node + (left ? 2 : 0)), o1 = __ldcg(node + (left ? 3 : 1));
        if (left) r = __float_as_int(o0.w);
        else l = __float_as_int(o1.w);
        if (l == 0 && r == n - 1) {
            root[left ? 0 : 2] = h0;
            root[left ? 1 : 3] = h1;
            root[left ? 2 : 0] = o0;
            root[left ? 3 : 1] = o1;
            return;
        }
        if (left) dr = r < n - 1 ? lbvh_delta(keys, r, r + 1) : -1;
        else dl = l > 0 ? lbvh_delta(keys, l - 1, l) : -1;
        link = (uint32_t)(s + 1);
        lo = make_float4(fminf(lo.x, o0.x), fminf(lo.y, o0.y), fminf(lo.z, o0.z), 0.f);
        hi = make_float4(fmaxf(hi.x, o1.x), fmaxf(hi.y, o1.y), fmaxf(hi.z, o1.z), 0.f);
    }
}

__global__ void __launch_bounds__(256) k_gather_boxes(int64_t n, int32_t* __restrict__ perm,
                                                      const float4* __restrict__ boxes, float4* __restrict__ out) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int64_t p = order_at(perm, i, n);
    out[2 * i] = boxes[2 * p];
    out[2 * i + 1] = boxes[2 * p + 1];
}

static inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

template <class Leaf>
static cudaError_t build_tree(Lbvh& L, int64_t n, const uint32_t* sorted_keys, Leaf leaf, cudaStream_t st) {
    cudaError_t e;
    if ((e = L.flags.ensure(LbvhBytes::flags(n))) != cudaSuccess) return e;
    if ((e = L.nodes.ensure(LbvhBytes::nodes(n))) != cudaSuccess) return e;
    L.n = n;
    if ((e = cudaMemsetAsync(L.flags.ptr, 0, LbvhBytes::flags(n), st)) != cudaSuccess) return e;
    k_lbvh_build<<<blocks_for(n, 256), 256, 0, st>>>((int)n, sorted_keys, leaf, L.nodes.as<BvhNode>(),
                                                     L.flags.as<uint32_t>()); gvc::note_launch();
    return cudaGetLastError();
}

cudaError_t lbvh_hierarchy(Lbvh& L, int64_t n, const uint32_t* sorted_keys, const float4* sorted_leaf_boxes,
                           cudaStream_t st) {
    return build_tree(L, n, sorted_keys, BoxLeaf{sorted_leaf_boxes}, st);
}

cudaError_t lbvh_hierarchy_points(Lbvh& L, int64_t n, const uint32_t* sorted_keys, const float4* sorted_points,
                                  cudaStream_t st) {
    return build_tree(L, n, sorted_keys, PointLeaf{sorted_points}, st);
}

// ----------------------------------------------------------------------------------
// Bounds, keys and the four passes for up to kSmallSort elements in one CTA, the keys staying
// in registers and shared memory.  Such a sort is all latency: a memset and six kernels against
// this one, a call of the 3-nearest search 115 / 92 us for 1024 points, 127 / 113 for 4096,
// 138 / 127 for 8192, 139 / 141 for 12288, 139 / 157 for 16384.
// ----------------------------------------------------------------------------------
constexpr int kSmallSort = 8192;
constexpr int kSmallWarps = 32;
constexpr int kSmallRounds = kSmallSort / (32 * kSmallWarps);

struct SmallSortSmem {
    uint32_t key[kSmallSort];
    int32_t val[kSmallSort];
    uint32_t cnt[kSmallWarps][256];  // counts, then first positions, of (warp, digit)
    uint32_t wsum[kSmallWarps];
    uint32_t lo[kSmallWarps][3], hi[kSmallWarps][3];
};

template <class Src>
__global__ void __launch_bounds__(32 * kSmallWarps) k_morton_sort_small(Src src, int n, uint32_t* __restrict__ keys,
                                                                        int32_t* __restrict__ perm) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSortSmem& sm = *reinterpret_cast<SmallSortSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float c[3];
        src.centroid(i, c);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            if (c[a] == c[a]) {
                const uint32_t o = f2ord(c[a]);
                mn[a] = min(mn[a], o);
                mx[a] = max(mx[a], o);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, mn[a]), h = __reduce_max_sync(0xffffffffu, mx[a]);
        if (lane == 0) {
            sm.lo[warp][a] = l;
            sm.hi[warp][a] = h;
        }
    }
    __syncthreads();
    MortonGrid grid;
    {
        uint32_t l[3], h[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            l[a] = __reduce_min_sync(0xffffffffu, sm.lo[lane][a]);
            h[a] = __reduce_max_sync(0xffffffffu, sm.hi[lane][a]);
        }
        grid.set(l, h);
    }
    // warp w's elements are [w * rounds * 32, (w + 1) * rounds * 32): (warp, round, lane) is input order
    const int rounds = (n + 32 * kSmallWarps - 1) / (32 * kSmallWarps);
    const int first = warp * rounds * 32 + lane;
    uint32_t kreg[kSmallRounds];
    int32_t vreg[kSmallRounds];
#pragma unroll
    for (int it = 0; it < kSmallRounds; it++) {
        const int e = first + 32 * it;
        if (it < rounds && e < n) {
            float c[3];
            src.centroid(e, c);
            kreg[it] = grid.key(c);
            vreg[it] = e;
        }
    }
    for (int pass = 0; pass < 4; pass++) {
        const int shift = 8 * pass;
        for (int i = threadIdx.x; i < 256 * kSmallWarps; i += blockDim.x) (&sm.cnt[0][0])[i] = 0u;
        __syncthreads();
        uint32_t rreg[kSmallRounds / 2];
#pragma unroll
        for (int it = 0; it < kSmallRounds; it++) {
            if (it < rounds) {  // the same for the whole block
                const bool valid = first + 32 * it < n;
                const uint32_t rank = digit_rank(valid, kreg[it] >> shift, sm.cnt[warp]);
                rreg[it / 2] = (it & 1) ? (rreg[it / 2] | (rank << 16)) : (rank & 0xffffu);
            }
        }
        __syncthreads();
        // four threads per digit, eight warps' counts each: first positions in (digit, warp) order
        const int d = threadIdx.x >> 2, w0 = 8 * (threadIdx.x & 3);
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            c[i] = sm.cnt[w0 + i][d];
            sum += c[i];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        if (lane == 31) sm.wsum[warp] = incl;
        __syncthreads();
        const uint32_t before = lane < warp ? sm.wsum[lane] : 0u;
        uint32_t pos = __reduce_add_sync(0xffffffffu, before) + incl - sum;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            sm.cnt[w0 + i][d] = pos;
            pos += c[i];
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kSmallRounds; it++) {
            if (it < rounds && first + 32 * it < n) {
                const uint32_t rank = (rreg[it / 2] >> (16 * (it & 1))) & 0xffffu;
                const uint32_t p = sm.cnt[warp][(kreg[it] >> shift) & 255u] + rank;
                sm.key[p] = kreg[it];
                sm.val[p] = vreg[it];
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < kSmallRounds; it++) {
            const int e = first + 32 * it;
            if (it < rounds && e < n) {
                kreg[it] = sm.key[e];
                vreg[it] = sm.val[e];
            }
        }
    }
#pragma unroll
    for (int it = 0; it < kSmallRounds; it++) {
        const int e = first + 32 * it;
        if (it < rounds && e < n) {
            keys[e] = kreg[it];
            perm[e] = vreg[it];
        }
    }
}

// Result: L.keys sorted, L.perm (sorted position -> input index).
template <class Src>
static cudaError_t morton_sort(Lbvh& L, int64_t n, Src src, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    cudaError_t e;
    if ((e = L.keys.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if (n <= kSmallSort) {
        if ((e = L.perm.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(k_morton_sort_small<Src>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SmallSortSmem))) != cudaSuccess) return e;
        k_morton_sort_small<Src><<<1, 32 * kSmallWarps, sizeof(SmallSortSmem), st>>>(
            src, (int)n, L.keys.as<uint32_t>(), L.perm.as<int32_t>()); gvc::note_launch();
        return cudaGetLastError();
    }
    // one kernel per pass where a status word can take the look-back's timeout report; the bounds
    // then lie among its words, and one memset clears both
    const bool os = L.status && n <= (int64_t)kOsCount;
    uint32_t* ghist = nullptr;
    uint32_t* bounds = nullptr;
    if (os) {
        if ((e = L.onesweep.ensure(LbvhBytes::onesweep(n))) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(L.onesweep.ptr, 0, LbvhBytes::onesweep(n), st)) != cudaSuccess) return e;
        ghist = L.onesweep.as<uint32_t>();
        bounds = ghist + kOsBounds;
    } else {
        if ((e = L.bounds.ensure(LbvhBytes::bounds())) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(L.bounds.ptr, 0, LbvhBytes::bounds(), st)) != cudaSuccess) return e;
        bounds = L.bounds.as<uint32_t>();
    }
    const unsigned nbk = blocks_for(n, 256);
    k_bounds<Src><<<nbk < 148u * 8u ? nbk : 148u * 8u, 256, 0, st>>>(src, n, bounds); gvc::note_launch();
    if (os) {
        k_keys<Src, true><<<nbk < 148u * 4u ? nbk : 148u * 4u, 256, 0, st>>>(src, n, bounds, L.keys.as<uint32_t>(),
                                                                             ghist);
        gvc::note_launch();
        return radix_sort_onesweep(L, n, 0, st);
    }
    k_keys<Src, false><<<nbk < 148u * 8u ? nbk : 148u * 8u, 256, 0, st>>>(src, n, bounds, L.keys.as<uint32_t>(), nullptr);
    gvc::note_launch();
    return radix_sort_pairs(L, n, st);
}

cudaError_t morton_sort_boxes(Lbvh& L, int64_t n, const float4* boxes, cudaStream_t st) {
    return morton_sort(L, n, BoxSrc{boxes}, st);
}

cudaError_t morton_sort_points(Lbvh& L, int64_t n, const float* pts, cudaStream_t st) {
    return morton_sort(L, n, PointSrc{pts}, st);
}

cudaError_t morton_sort_points_withheld(Lbvh& L, int64_t n, const float* pts, cudaStream_t st) {
    if (n <= kRsTile || n > (int64_t)kOsCount || !L.status) return cudaErrorInvalidValue;
    cudaError_t e;
    if ((e = L.keys.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.perm_alt.ensure(LbvhBytes::keys(n))) != cudaSuccess) return e;
    if ((e = L.onesweep.ensure(LbvhBytes::onesweep(n))) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(L.onesweep.ptr, 0, LbvhBytes::onesweep(n), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(L.perm.ptr, 0x7f, LbvhBytes::keys(n), st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(L.perm_alt.ptr, 0x7f, LbvhBytes::keys(n), st)) != cudaSuccess) return e;
    uint32_t* ghist = L.onesweep.as<uint32_t>();
    const uint32_t first[4] = {1, 1, 1, 1};
    if ((e = cudaMemcpyAsync(ghist + 4 * 256, first, sizeof(first), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
    k_bounds<PointSrc><<<8, 256, 0, st>>>(PointSrc{pts}, n, ghist + kOsBounds); gvc::note_launch();
    k_keys<PointSrc, true><<<8, 256, 0, st>>>(PointSrc{pts}, n, ghist + kOsBounds, L.keys.as<uint32_t>(), ghist);
    gvc::note_launch();
    return radix_sort_onesweep(L, n, 1, st);
}

cudaError_t lbvh_build_boxes(Lbvh& L, int64_t n, const float4* boxes, cudaStream_t st) {
    cudaError_t e;
    if (n <= 0) {
        L.n = 0;
        return cudaSuccess;
    }
    if ((e = morton_sort_boxes(L, n, boxes, st)) != cudaSuccess) return e;
    if ((e = L.sorted_boxes.ensure(LbvhBytes::sorted_boxes(n))) != cudaSuccess) return e;
    k_gather_boxes<<<blocks_for(n, 256), 256, 0, st>>>(n, L.perm.as<int32_t>(), boxes, L.sorted_boxes.as<float4>()); gvc::note_launch();
    return lbvh_hierarchy(L, n, L.keys.as<uint32_t>(), L.sorted_boxes.as<float4>(), st);
}

}  // namespace gvc
