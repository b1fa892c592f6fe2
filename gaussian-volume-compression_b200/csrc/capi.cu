// capi.cu -- extern "C" entry points of libgvc.so (declared in include/gvc.h).
//
// Host orchestration of the path that diff-gaussian-rasterization/ext.cu,
// rasterize_points.cu and cuda_rasterizer/rasterizer_impl.cu implement in the
// reference: stream-ordered, no per-call cudaMalloc once the context's buffers have
// grown to the working sizes, no device synchronisation unless debug is set (the
// reference synchronises every call through cudaMalloc/cudaFree and a D2H copy,
// rasterizer_impl.cu:121-169).
#include <atomic>
#include <cstdio>
#include <cstring>
#include <new>

#include "host_io.cuh"
#include "lbvh.cuh"
#include "render.cuh"

using namespace gvc;

static std::atomic<long long> g_launches{0};
void gvc::note_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

namespace {

struct Scratch {
    DevBuf gacc;       // [P][16] per-Gaussian gradient accumulators
    DevBuf tmp_boxes;  // debug hooks / tet boxes
    Lbvh dbg;          // debug LBVH
    Lbvh msamp;        // Morton order of mesh sample points
    Stage stage;       // pinned chunks for host arrays
};

Scratch* scratch_of(gvc_ctx* c);

int fail(gvc_ctx* c, int code, const char* msg) {
    if (c) c->err = msg;
    return code;
}

// The error is reported here: it must not stay behind as the thread's last one, where the next
// launch's check, this library's or another's, takes it for its own.
int cuda_fail(gvc_ctx* c, cudaError_t e, const char* where) {
    (void)cudaGetLastError();
    if (c) {
        c->err = std::string(where) + ": " + cudaGetErrorString(e);
    }
    return GVC_ERR_CUDA;
}

#define GVC_CUDA(call, where)                                   \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, where); \
    } while (0)

__global__ void k_boxes6_to_f4(int64_t n, const float* __restrict__ b6, float4* __restrict__ out) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[2 * i] = make_float4(b6[6 * i], b6[6 * i + 1], b6[6 * i + 2], 0.f);
    out[2 * i + 1] = make_float4(b6[6 * i + 3], b6[6 * i + 4], b6[6 * i + 5], 0.f);
}

// The tree in Karras' numbering: a node's index is the first or the last of its leaves, as it is
// its parent's right or left child, the root's 0.
__device__ int karras_index(const BvhNode* nodes, const uint32_t* keys, int n, int k) {
    const int l = __float_as_int(nodes[k].b.w), r = __float_as_int(nodes[k].c.w);
    if (l == 0 && r == n - 1) return 0;
    return lbvh_is_left(keys, n, l, r) ? r : l;
}

// For node k = 1 + split: its children, its box, and its escape edge (2 p + 1 for the node p
// whose left child's leaves end where this node's do, all ones on the root's right spine).
__global__ void k_karras_tree(int n, const BvhNode* __restrict__ nodes, const uint32_t* __restrict__ keys,
                              int32_t* __restrict__ left, int32_t* __restrict__ right, float* __restrict__ boxes6,
                              int32_t* __restrict__ escape) {
    const int k = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const BvhNode nd = nodes[k];
    const int at = karras_index(nodes, keys, n, k), l = __float_as_int(nd.b.w), r = __float_as_int(nd.c.w);
    if (left) left[at] = l == k - 1 ? (int32_t)((uint32_t)l | kLeafBit) : k - 1;
    if (right) right[at] = r == k ? (int32_t)((uint32_t)r | kLeafBit) : k;
    if (boxes6) {
        boxes6[6 * at] = fminf(nd.a.x, nd.c.x);
        boxes6[6 * at + 1] = fminf(nd.a.y, nd.c.y);
        boxes6[6 * at + 2] = fminf(nd.a.z, nd.c.z);
        boxes6[6 * at + 3] = fmaxf(nd.b.x, nd.d.x);
        boxes6[6 * at + 4] = fmaxf(nd.b.y, nd.d.y);
        boxes6[6 * at + 5] = fmaxf(nd.b.z, nd.d.z);
    }
    if (escape) escape[at] = r == n - 1 ? -1 : 2 * karras_index(nodes, keys, n, r + 1) + 1;
}

__global__ void k_f4_to_boxes6(int64_t n, const float4* __restrict__ in, float* __restrict__ b6) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 lo = in[2 * i], hi = in[2 * i + 1];
    b6[6 * i] = lo.x;
    b6[6 * i + 1] = lo.y;
    b6[6 * i + 2] = lo.z;
    b6[6 * i + 3] = hi.x;
    b6[6 * i + 4] = hi.y;
    b6[6 * i + 5] = hi.z;
}

inline unsigned nb(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// Largest element count handled with 32-bit indices inside the kernels.
constexpr int64_t kMaxElems = (int64_t(1) << 31) - 4096;

struct DebugTimer {
    bool on;
    cudaStream_t st;
    cudaEvent_t ev[8];
    int n = 0;
    DebugTimer(bool on_, cudaStream_t s) : on(on_), st(s) {
        if (on)
            for (auto& e : ev) cudaEventCreate(&e);
    }
    void mark() {
        if (on && n < 8) cudaEventRecord(ev[n++], st);
    }
    float ms(int a, int b) {
        float t = 0.f;
        if (on && b < n) cudaEventElapsedTime(&t, ev[a], ev[b]);
        return t;
    }
    ~DebugTimer() {
        if (on)
            for (auto& e : ev) cudaEventDestroy(e);
    }
};

// Kernel timing: events recorded around the evaluation kernels on the caller's stream;
// read out (after a synchronisation) by gvc_get_stats or when the pool is full.
void drain_events(gvc_ctx* ctx) {
    for (int i = 0; i < ctx->ev_pending; i++) {
        cudaEventSynchronize(ctx->ev_pool[2 * i + 1]);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev_pool[2 * i], ctx->ev_pool[2 * i + 1]);
        if (ctx->ev_kind[i] == 0) {
            ctx->fwd_kernel_ms += ms;
            ctx->fwd_kernel_calls++;
        } else {
            ctx->bwd_kernel_ms += ms;
            ctx->bwd_kernel_calls++;
        }
    }
    ctx->ev_pending = 0;
}

int timer_begin(gvc_ctx* ctx, cudaStream_t st, int kind) {
    if (!ctx->time_kernels) return -1;
    if (!ctx->ev_init) {
        for (auto& e : ctx->ev_pool) cudaEventCreate(&e);
        ctx->ev_init = true;
    }
    if (ctx->ev_pending == 32) drain_events(ctx);
    int i = ctx->ev_pending++;
    ctx->ev_kind[i] = kind;
    cudaEventRecord(ctx->ev_pool[2 * i], st);
    return i;
}

void timer_end(gvc_ctx* ctx, cudaStream_t st, int i) {
    if (i >= 0) cudaEventRecord(ctx->ev_pool[2 * i + 1], st);
}

int debug_check(gvc_ctx* ctx, cudaStream_t st) {
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "debug synchronize");
    e = cudaMemcpy(ctx->h_status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "status copy");
    const int s = *ctx->h_status;
    if (s == 0) return GVC_OK;
    e = cudaMemset(ctx->d_status, 0, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(ctx, e, "status clear");
    if (s & kStatusStackOverflow)
        return fail(ctx, GVC_ERR_TRAVERSAL, "BVH traversal stack overflow: results are invalid");
    return fail(ctx, GVC_ERR_TIMEOUT,
                "a bounded device-side wait ran out (pipeline barrier or radix-sort look-back): results are invalid");
}

}  // namespace

struct gvc_ctx_full : gvc_ctx {
    Scratch scratch;
};

namespace {
Scratch* scratch_of(gvc_ctx* c) { return &static_cast<gvc_ctx_full*>(c)->scratch; }

// The buffers of training_samples and their sizes (ctx null: sizes only).
template <class F>
void training_buffers(gvc_ctx* ctx, int64_t C, int64_t N, bool gt, F f) {
    auto at = [&](auto pick) -> DevBuf* { return ctx ? pick(static_cast<gvc_ctx_full*>(ctx)) : nullptr; };
    f(at([](gvc_ctx_full* c) { return &c->ts_points; }), sizeof(float) * 3 * N);
    f(at([](gvc_ctx_full* c) { return &c->ts_words; }), sizeof(uint32_t) * 3 * N);
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.keys; }), LbvhBytes::keys(N));
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.keys_alt; }), LbvhBytes::keys(N));
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.perm; }), LbvhBytes::keys(N));
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.perm_alt; }), LbvhBytes::keys(N));
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.hist; }), LbvhBytes::hist(N));
    f(at([](gvc_ctx_full* c) { return &c->ts_sort.onesweep; }), LbvhBytes::onesweep(N));
    if (!gt) return;
    f(at([](gvc_ctx_full* c) { return &c->scratch.tmp_boxes; }), sizeof(float4) * 2 * C);
    f(at([](gvc_ctx_full* c) { return &c->cells.keys; }), LbvhBytes::keys(C));
    f(at([](gvc_ctx_full* c) { return &c->cells.keys_alt; }), LbvhBytes::keys(C));
    f(at([](gvc_ctx_full* c) { return &c->cells.perm; }), LbvhBytes::keys(C));
    f(at([](gvc_ctx_full* c) { return &c->cells.perm_alt; }), LbvhBytes::keys(C));
    f(at([](gvc_ctx_full* c) { return &c->cells.bounds; }), LbvhBytes::bounds());
    f(at([](gvc_ctx_full* c) { return &c->cells.onesweep; }), LbvhBytes::onesweep(C));
    f(at([](gvc_ctx_full* c) { return &c->cell_tree; }), sizeof(float4) * 2 * (size_t)wide_tree_size(C).boxes);
    f(at([](gvc_ctx_full* c) { return &c->cell_recs; }), sizeof(float4) * 8 * C);
}

size_t round256(size_t n) { return (n + 255) & ~size_t(255); }
}  // namespace

extern "C" {

int64_t gvc_launch_count(void) { return (int64_t)g_launches.load(std::memory_order_relaxed); }

int gvc_ctx_create(gvc_ctx** out) {
    if (!out) return GVC_ERR_ARG;
    *out = nullptr;
    gvc_ctx_full* c = new (std::nothrow) gvc_ctx_full();
    if (!c) return GVC_ERR_CAPACITY;
    gvc_ctx* ctx = c;
    GVC_CUDA(cudaGetDevice(&c->device), "cudaGetDevice");
    GVC_CUDA(cudaMalloc(&c->d_status, sizeof(int)), "cudaMalloc status");
    GVC_CUDA(cudaMemset(c->d_status, 0, sizeof(int)), "cudaMemset status");
    GVC_CUDA(cudaMalloc(&c->d_stats, sizeof(unsigned long long) * 16), "cudaMalloc stats");
    GVC_CUDA(cudaMemset(c->d_stats, 0, sizeof(unsigned long long) * 16), "cudaMemset stats");
    GVC_CUDA(cudaMallocHost(&c->h_status, sizeof(int)), "cudaMallocHost");
    Lbvh* sorted[] = {&c->s_sort, &c->gsort, &c->cells, &c->knn, &c->ts_sort, &c->scratch.dbg,
                      &c->scratch.msamp};
    for (Lbvh* L : sorted) L->status = c->d_status;
    *out = c;
    return GVC_OK;
}

void gvc_ctx_destroy(gvc_ctx* ctx) {
    if (!ctx) return;
    gvc_ctx_full* c = static_cast<gvc_ctx_full*>(ctx);
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(c->device);
    Lbvh* lbvhs[] = {&c->s_sort,  &c->gsort,        &c->cells,       &c->knn,
                     &c->ts_sort, &c->scratch.dbg, &c->scratch.msamp};
    for (Lbvh* L : lbvhs) {
        DevBuf* bufs[] = {&L->keys, &L->keys_alt, &L->perm, &L->perm_alt, &L->sorted_boxes,
                          &L->flags, &L->nodes, &L->hist, &L->bounds,
                          &L->onesweep};
        for (DevBuf* b : bufs) b->release();
    }
    DevBuf* bufs[] = {&c->s_sorted, &c->fwd_sorted, &c->blk_desc, &c->blk_boxes, &c->blk_desc_c, &c->blk_boxes_c,
                      &c->b_rows, &c->b_boxes, &c->gtree, &c->s_grad, &c->s_gyz, &c->s_ok, &c->grec, &c->gtmp,
                      &c->knn_points, &c->ts_points, &c->ts_words, &c->cell_tree, &c->cell_recs, &c->clog, &c->cmask,
                      &c->cend, &c->moved, &c->scratch.gacc, &c->scratch.tmp_boxes};
    for (DevBuf* b : bufs) b->release();
    c->scratch.stage.release();
    if (c->d_status) cudaFree(c->d_status);
    if (c->d_stats) cudaFree(c->d_stats);
    if (c->h_status) cudaFreeHost(c->h_status);
    if (c->ev_init)
        for (auto& e : c->ev_pool) cudaEventDestroy(e);
    cudaSetDevice(prev);
    delete c;
}

const char* gvc_last_error(const gvc_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int gvc_set_option(gvc_ctx* ctx, int option, int value) {
    if (!ctx) return GVC_ERR_ARG;
    switch (option) {
        case GVC_OPT_COV_GRAD:
            if (value < 0 || value > 1) return fail(ctx, GVC_ERR_ARG, "cov_grad must be 0 or 1");
            ctx->cov_grad_mode = value;
            return GVC_OK;
        case GVC_OPT_BWD_MODE:
            if (value < 0 || value > 3) return fail(ctx, GVC_ERR_ARG, "bwd_mode must be 0, 1, 2 or 3");
            ctx->bwd_mode = value;
            return GVC_OK;
        case GVC_OPT_EVAL_PATH:
            if (value < 0 || value > 2) return fail(ctx, GVC_ERR_ARG, "eval path must be 0, 1 or 2");
            ctx->eval_path = value;
            return GVC_OK;
        case GVC_OPT_COUNT_PAIRS:
            ctx->count_pairs = value ? 1 : 0;
            return GVC_OK;
        case GVC_OPT_CAND_LOG:
            ctx->cand_log = value ? 1 : 0;
            return GVC_OK;
        case GVC_OPT_TRAVERSAL:
            if (value < 0 || value > 1) return fail(ctx, GVC_ERR_ARG, "traversal must be 0 or 1");
            return GVC_OK;
        case GVC_OPT_TIME_KERNELS:
            drain_events(ctx);
            ctx->time_kernels = value ? 1 : 0;
            ctx->fwd_kernel_ms = ctx->bwd_kernel_ms = 0.0;
            ctx->fwd_kernel_calls = ctx->bwd_kernel_calls = 0;
            return GVC_OK;
        default:
            return fail(ctx, GVC_ERR_ARG, "unknown option");
    }
}

int gvc_get_stats(gvc_ctx* ctx, gvc_stats* out, void* stream) {
    if (!ctx || !out) return GVC_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long h[16];
    GVC_CUDA(cudaStreamSynchronize(st), "cudaStreamSynchronize");
    GVC_CUDA(cudaMemcpy(h, ctx->d_stats, sizeof(h), cudaMemcpyDeviceToHost), "stats copy");
    out->fwd_candidates = (int64_t)h[0];
    out->fwd_contributing = (int64_t)h[1];
    out->bwd_contributing = (int64_t)h[2];
    out->max_stack_fwd = (int32_t)h[3];
    out->max_stack_bwd = (int32_t)h[4];
    out->fwd_leaf_hits = (int64_t)h[5];
    out->fwd_node_visits = (int64_t)h[6];
    out->bwd_leaf_hits = (int64_t)h[7];
    out->bwd_node_visits = (int64_t)h[8];
    out->fwd_lane_evals = (int64_t)h[9];
    out->bwd_rows = (int64_t)h[10];
    drain_events(ctx);
    out->fwd_kernel_ms = ctx->fwd_kernel_ms;
    out->bwd_kernel_ms = ctx->bwd_kernel_ms;
    out->fwd_kernel_calls = ctx->fwd_kernel_calls;
    out->bwd_kernel_calls = ctx->bwd_kernel_calls;
    return GVC_OK;
}

int gvc_sync_status(gvc_ctx* ctx, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    return debug_check(ctx, (cudaStream_t)stream);
}

// Whether S samples are sparse among P Gaussians, S < 600 sqrt(P): below the line a warp per
// sample (fwd_points.cu) beats a warp per block of 128 (fwd_blocks.cu), whose box then spans
// many Gaussians that reach one or two of its rows.  Both, us, on either side of it: 2k
// Gaussians 30k samples 24 / 36, 60k 41 / 28; 20k: 60k 98 / 151, 130k 192 / 131; 200k: 130k
// 560 / 870, 262k 1087 / 725; 1M (clustered): 524k 2207 / 2409, 1M 4108 / 1775; far below it,
// 1M Gaussians and 14k samples, 104 / 14395.
static bool sparse_samples(int64_t S, int64_t P) { return (double)S * (double)S < 360000.0 * (double)P; }

// Whether the tensor-core kernels are selected for a call (the forward then prepares what the
// backward reads).
static bool tensor_core_backward(const gvc_ctx* ctx) {
    return ctx->bwd_mode == 3 || (ctx->bwd_mode == 0 && ctx->eval_path == 1);
}

// Morton order of the Gaussians' AABBs, their records in that order and the tree over them:
// the LBVH for the tensor-core kernels, else the wide tree (new_order false: the order of the
// last forward still holds).  `moved`: as launch_gather_recs.
static int prepare_gaussians(gvc_ctx* ctx, int64_t P, const float* means, const float* values, const float* weights,
                             const float* conics, bool new_order, bool linked, int* moved, cudaStream_t st) {
    const float4* boxes = ctx->gtmp.as<float4>();
    if (new_order) GVC_CUDA(morton_sort_boxes(ctx->gsort, P, boxes, st), "Gaussian order");
    GVC_CUDA(ctx->grec.ensure(sizeof(GaussRec) * P), "alloc records");
    GVC_CUDA(ctx->gtree.ensure(sizeof(float4) * 2 * wide_tree_size(P).boxes), "alloc Gaussian tree");
    GVC_CUDA(launch_gather_recs(P, ctx->gsort.perm.as<int32_t>(), means, values, weights, conics, boxes,
                                ctx->grec.as<GaussRec>(), ctx->gtree.as<float4>(), !linked, moved, st),
             "gather records");
    ctx->glinks_ready = false;
    if (linked) {
        GVC_CUDA(lbvh_hierarchy(ctx->gsort, P, ctx->gsort.keys.as<uint32_t>(), ctx->gtree.as<float4>(), st),
                 "Gaussian LBVH");
        ctx->glinks_ready = true;
    }
    return GVC_OK;
}

// The coarser block groups of the tensor-core kernels' forward.
static int ensure_coarse_groups(gvc_ctx* ctx, cudaStream_t st) {
    if (ctx->blk_c_ready || ctx->S == 0) return GVC_OK;
    const int64_t n_blocks = (ctx->S + 127) / 128;
    GVC_CUDA(ctx->blk_desc_c.ensure(sizeof(uint2) * n_blocks), "alloc blk_desc_c");
    GVC_CUDA(ctx->blk_boxes_c.ensure(sizeof(float4) * 2 * 8 * n_blocks), "alloc blk_boxes_c");
    GVC_CUDA(launch_sample_blocks(ctx->S, ctx->s_sorted.as<float4>(), ctx->s_sort.keys.as<uint32_t>(),
                                  ctx->blk_desc_c.as<uint2>(), ctx->blk_boxes_c.as<float4>(), kBlockSplitCoarse, st),
             "coarse block groups");
    ctx->blk_c_ready = true;
    return GVC_OK;
}

int gvc_build_bvh(gvc_ctx* ctx, const float* samples, int64_t S, int debug, int use_gaussian_bvh, void* stream) {
    (void)use_gaussian_bvh;  // both reference modes use the same sample ordering here
    if (!ctx) return GVC_ERR_ARG;
    if (S < 0 || S > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "number of samples out of range");
    if (S > 0 && !samples) return fail(ctx, GVC_ERR_ARG, "samples is null");
    cudaStream_t st = (cudaStream_t)stream;
    DebugTimer tm(debug != 0, st);
    tm.mark();
    ctx->samples = samples;
    ctx->S = S;
    ctx->n_tiles = (S + kTile - 1) / kTile;
    ctx->samples_ready = false;
    ctx->blk_c_ready = false;
    ctx->clog_ready = false;
    ctx->fwd_sorted_ready = false;
    if (S > 0) {
        GVC_CUDA(morton_sort_points(ctx->s_sort, S, samples, st), "sample sort");
        const int64_t slots = ctx->n_tiles * kTile;
        GVC_CUDA(ctx->s_sorted.ensure(sizeof(float4) * slots), "alloc s_sorted");
        GVC_CUDA(launch_sample_slots(S, slots, samples, ctx->s_sort.perm.as<int32_t>(), ctx->s_sorted.as<float4>(), st),
                 "sorted samples");
        const int64_t n_blocks = (S + 127) / 128;
        GVC_CUDA(ctx->blk_desc.ensure(sizeof(uint2) * n_blocks), "alloc blk_desc");
        GVC_CUDA(ctx->blk_boxes.ensure(sizeof(float4) * 2 * 8 * n_blocks), "alloc blk_boxes");
        // when the options already select the tensor-core kernels, their coarser groups come
        // from the same launch
        const bool coarse = tensor_core_backward(ctx) || ctx->eval_path == 1;
        if (coarse) {
            GVC_CUDA(ctx->blk_desc_c.ensure(sizeof(uint2) * n_blocks), "alloc blk_desc_c");
            GVC_CUDA(ctx->blk_boxes_c.ensure(sizeof(float4) * 2 * 8 * n_blocks), "alloc blk_boxes_c");
        }
        GVC_CUDA(launch_sample_blocks(S, ctx->s_sorted.as<float4>(), ctx->s_sort.keys.as<uint32_t>(),
                                      ctx->blk_desc.as<uint2>(), ctx->blk_boxes.as<float4>(), kBlockSplit, st,
                                      coarse ? ctx->blk_desc_c.as<uint2>() : nullptr,
                                      coarse ? ctx->blk_boxes_c.as<float4>() : nullptr, kBlockSplitCoarse),
                 "sample blocks");
        ctx->blk_c_ready = coarse;
    }
    ctx->samples_ready = true;
    tm.mark();
    if (debug) {
        int rc = debug_check(ctx, st);
        printf("Sample BVH time: %g ms\n", tm.ms(0, 1));
        if (rc) return rc;
    }
    return GVC_OK;
}

int gvc_rasterize_gaussians(gvc_ctx* ctx, int64_t P, const float* means3D, const float* scales,
                            const float* rotations, const float* values, const float* weights, float scale_modifier,
                            const float* bounds, float bg, int use_gaussian_bvh, int debug, float* out_cells,
                            float* out_weights, float* conics, void* stream) {
    (void)bounds;
    (void)bg;
    (void)use_gaussian_bvh;
    if (!ctx) return GVC_ERR_ARG;
    if (!ctx->samples_ready) return fail(ctx, GVC_ERR_STATE, "build_bvh must be called before rasterize_gaussians");
    if (P < 0 || P > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "number of Gaussians out of range");
    const int64_t S = ctx->S;
    if (S > 0 && (!out_cells || !out_weights)) return fail(ctx, GVC_ERR_ARG, "null output");
    cudaStream_t st = (cudaStream_t)stream;
    if (P == 0) {  // rasterize_points.cu:51: outputs stay zero
        GVC_CUDA(launch_fill_zero_outputs(S, out_cells, out_weights, st), "zero outputs");
        ctx->gauss_ready = false;
        ctx->clog_ready = false;
        ctx->fwd_sorted_ready = false;
        ctx->fwd_recs_ready = false;
        return GVC_OK;
    }
    if (!means3D || !scales || !rotations || !values || !weights || !conics)
        return fail(ctx, GVC_ERR_ARG, "null Gaussian parameter pointer");
    // this call rewrites the order, AABBs, records, log and sorted outputs: valid again only once
    // it ends (left by a call that fails, an order of more Gaussians would index past the last
    // forward's)
    ctx->gauss_ready = false;
    ctx->clog_ready = false;
    ctx->fwd_recs_ready = false;
    ctx->fwd_sorted_ready = false;
    DebugTimer tm(debug != 0, st);
    if (ctx->count_pairs) GVC_CUDA(cudaMemsetAsync(ctx->d_stats, 0, sizeof(unsigned long long) * 16, st), "stats");
    tm.mark();
    GVC_CUDA(ctx->gtmp.ensure(sizeof(float4) * 2 * P), "alloc boxes");
    float4* boxes = ctx->gtmp.as<float4>();
    GVC_CUDA(launch_preprocess(P, means3D, scales, rotations, weights, scale_modifier, conics, boxes, st),
             "preprocess");
    tm.mark();
    // with the tensor-core kernels selected, the forward walks the LBVH by the coarser groups
    const bool tc_bwd = tensor_core_backward(ctx);
    const bool linked = tc_bwd || ctx->eval_path == 1;
    int rc = prepare_gaussians(ctx, P, means3D, values, weights, conics, true, linked, nullptr, st);
    if (rc == GVC_OK && linked) rc = ensure_coarse_groups(ctx, st);
    if (rc != GVC_OK) return rc;
    tm.mark();
    FwdArgs fa{};
    fa.P = P;
    fa.s_sorted = ctx->s_sorted.as<float4>();
    fa.S = S;
    fa.bdesc = (linked ? ctx->blk_desc_c : ctx->blk_desc).as<uint2>();
    fa.bboxes = (linked ? ctx->blk_boxes_c : ctx->blk_boxes).as<float4>();
    fa.tree = wide_tree_at(wide_tree_size(P), ctx->gtree.as<float4>());
    fa.nodes = linked ? ctx->gsort.nodes.as<BvhNode>() : nullptr;
    fa.recs = ctx->grec.as<GaussRec>();
    fa.out_cells = out_cells;
    fa.out_weights = out_weights;
    fa.status = ctx->d_status;
    fa.stats = ctx->d_stats;
    fa.count = ctx->count_pairs != 0;
    // the candidates are logged for the tensor-core backward when it is the one selected
    if (tc_bwd && ctx->cand_log && S > 0) {
        // 20 KB per 128 samples: where that does not fit in device memory, the forward runs
        // without the log and the backward walks the tree
        const int64_t n_blocks = (S + 127) / 128;
        if (ctx->clog.ensure(sizeof(int32_t) * kCandLogPerBlock * n_blocks) == cudaSuccess &&
            ctx->cmask.ensure(kCandLogPerBlock * n_blocks) == cudaSuccess &&
            ctx->cend.ensure(sizeof(int32_t) * 8 * n_blocks) == cudaSuccess &&
            ctx->moved.ensure(sizeof(int)) == cudaSuccess) {
            fa.clog = ctx->clog.as<int32_t>();
            fa.cmask = ctx->cmask.as<uint8_t>();
            fa.cend = ctx->cend.as<int32_t>();
            fa.fdesc = ctx->blk_desc.as<uint2>();
            fa.fboxes = ctx->blk_boxes.as<float4>();
        } else {
            (void)cudaGetLastError();  // a failed allocation is not sticky: clear it
            ctx->clog.release();
            ctx->cmask.release();
            ctx->cend.release();
        }
    }
    // (out, W) in sorted order as well, for the backward's rows (FP32 only: after a tensor-core
    // evaluation the backward has always read the caller's arrays, changed or not)
    if (S > 0 && ctx->eval_path == 0) {
        if (ctx->fwd_sorted.ensure(sizeof(float2) * ctx->n_tiles * kTile) == cudaSuccess) {
            fa.out_sorted = ctx->fwd_sorted.as<float2>();
        } else {
            (void)cudaGetLastError();
            ctx->fwd_sorted.release();
        }
    }
    const int tk = timer_begin(ctx, st, 0);
    bool masks = false;
    cudaError_t e;
    if (ctx->eval_path == 1) {
        e = launch_forward_tc(fa, st);
    } else if (!linked) {
        e = sparse_samples(S, P) ? launch_forward_points(fa, st) : launch_forward_blocks(fa, st);
    } else if (forward_linked_rows(S, P) == 0) {
        e = launch_forward_cta(fa, st);
    } else {
        e = launch_forward_blocks(fa, st);
        masks = true;
    }
    GVC_CUDA(e, "forward");
    ctx->clog_ready = fa.clog != nullptr;
    ctx->clog_masks = masks;
    ctx->fwd_sorted_ready = fa.out_sorted != nullptr;
    ctx->fwd_out_cells = out_cells;
    ctx->fwd_out_weights = out_weights;
    timer_end(ctx, st, tk);
    tm.mark();
    ctx->P = P;
    ctx->gauss_ready = true;
    ctx->fwd_means = means3D;
    ctx->fwd_scales = scales;
    ctx->fwd_rots = rotations;
    ctx->fwd_values = values;
    ctx->fwd_weights = weights;
    ctx->fwd_conics = conics;
    ctx->fwd_scale_mod = scale_modifier;
    ctx->fwd_recs_ready = true;
    if (debug) {
        int rc = debug_check(ctx, st);
        printf("Preprocess time: %g ms\nBVH time: %g ms\nRender time: %g ms\n", tm.ms(0, 1), tm.ms(1, 2),
               tm.ms(2, 3));
        if (rc) return rc;
    }
    return GVC_OK;
}

int gvc_rasterize_gaussians_backward(gvc_ctx* ctx, int64_t P, const float* means3D, const float* scales,
                                     const float* rotations, const float* conics, const float* values,
                                     const float* weights, const float* out_cells, const float* out_weights,
                                     float scale_modifier, const float* bounds, float bg, const float* dL_dout_cells,
                                     const float* dL_dout_weights, int use_gaussian_bvh, int debug, float* dmeans,
                                     float* dscales, float* drots, float* dvalues, float* dweights, void* stream) {
    (void)bounds;
    (void)bg;
    if (!ctx) return GVC_ERR_ARG;
    if (!ctx->samples_ready)
        return fail(ctx, GVC_ERR_STATE, "build_bvh must be called before rasterize_gaussians_backward");
    if (P < 0 || P > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "number of Gaussians out of range");
    if (P == 0) return GVC_OK;
    if (!means3D || !scales || !rotations || !conics || !values || !weights || !dmeans || !dscales || !drots ||
        !dvalues || !dweights)
        return fail(ctx, GVC_ERR_ARG, "null pointer");
    const int64_t S = ctx->S;
    if (S > 0 && (!out_cells || !out_weights || !dL_dout_cells || !dL_dout_weights))
        return fail(ctx, GVC_ERR_ARG, "null sample-side pointer");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    DebugTimer tm(debug != 0, st);
    tm.mark();
    // Handed the very arrays of the last forward (and its conics), the forward's AABBs and
    // LBVH-ordered records still hold; otherwise both are rebuilt here (and no longer
    // describe that forward).
    const bool same_gauss = ctx->fwd_recs_ready && ctx->gauss_ready && ctx->P == P && means3D == ctx->fwd_means &&
                            scales == ctx->fwd_scales && rotations == ctx->fwd_rots && values == ctx->fwd_values &&
                            weights == ctx->fwd_weights && conics == ctx->fwd_conics &&
                            scale_modifier == ctx->fwd_scale_mod;
    GVC_CUDA(ctx->gtmp.ensure(sizeof(float4) * 2 * P), "alloc boxes");
    float4* boxes = ctx->gtmp.as<float4>();
    if (!same_gauss) {
        ctx->fwd_recs_ready = false;
        GVC_CUDA(launch_preprocess(P, means3D, scales, rotations, weights, scale_modifier, nullptr, boxes, st),
                 "preprocess");
    }
    (void)use_gaussian_bvh;  // both reference modes sum over the same pairs
    GVC_CUDA(sc->gacc.ensure(sizeof(float) * 16 * P), "alloc gacc");
    float* gacc = sc->gacc.as<float>();
    // mode 3, or the tensor-core path in auto mode: reduction over samples on tcgen05; every
    // other mode: the Gaussian-owned sums
    const bool tc_bwd = tensor_core_backward(ctx);
    const bool have_order = ctx->gauss_ready && ctx->P == P;
    if (ctx->n_tiles == 0) {
        GVC_CUDA(cudaMemsetAsync(gacc, 0, sizeof(float) * 16 * P, st), "zero gacc");
        tm.mark();
    } else {
        // the forward's sorted copy of (out, W) when these are the arrays it wrote
        const bool same_out = ctx->fwd_sorted_ready && have_order && out_cells == ctx->fwd_out_cells &&
                              out_weights == ctx->fwd_out_weights;
        const float2* out_sorted = same_out ? ctx->fwd_sorted.as<float2>() : nullptr;
        BwdArgs ba{};
        ba.P = P;
        ba.conics = conics;
        ba.boxes = boxes;
        ba.gacc = gacc;
        ba.status = ctx->d_status;
        ba.stats = ctx->d_stats;
        ba.count = ctx->count_pairs != 0;
        if (tc_bwd) {
            const int64_t slots = ctx->n_tiles * kTile;
            GVC_CUDA(ctx->s_grad.ensure(sizeof(float4) * slots), "alloc s_grad");
            GVC_CUDA(ctx->s_gyz.ensure(sizeof(float) * slots), "alloc s_gyz");
            GVC_CUDA(ctx->s_ok.ensure(slots), "alloc s_ok");
            GVC_CUDA(launch_sample_grads(slots, ctx->s_sorted.as<float4>(), out_sorted, out_cells, out_weights,
                                         dL_dout_cells, dL_dout_weights, ctx->s_grad.as<float4>(),
                                         ctx->s_gyz.as<float>(), ctx->s_ok.as<uint8_t>(), st),
                     "sample grads");
            tm.mark();
            // the forward's candidate log serves the Gaussians whose boxes it holds: the forward's
            // own arrays, or others with the same boxes (copies), which the device finds out
            const bool use_log = have_order && ctx->clog_ready;
            int* moved = nullptr;
            if (!same_gauss) {
                if (!have_order) ctx->gauss_ready = false;  // the order below is not the forward's
                if (use_log) {
                    moved = ctx->moved.as<int>();
                    GVC_CUDA(cudaMemsetAsync(moved, 0, sizeof(int), st), "clear flag");
                }
                const int rc =
                    prepare_gaussians(ctx, P, means3D, values, weights, conics, !have_order, true, moved, st);
                if (rc != GVC_OK) return rc;
            } else if (!ctx->glinks_ready) {
                GVC_CUDA(lbvh_hierarchy(ctx->gsort, P, ctx->gsort.keys.as<uint32_t>(), ctx->gtree.as<float4>(), st),
                         "Gaussian LBVH");
                ctx->glinks_ready = true;
            }
            GVC_CUDA(cudaMemsetAsync(gacc, 0, sizeof(float) * 16 * P, st), "zero gacc");
            ba.gperm = ctx->gsort.perm.as<int32_t>();
            ba.S = S;
            ba.bdesc = ctx->blk_desc.as<uint2>();
            ba.bboxes = ctx->blk_boxes.as<float4>();
            ba.s_grad = ctx->s_grad.as<float4>();
            ba.s_gyz = ctx->s_gyz.as<float>();
            ba.s_ok = ctx->s_ok.as<uint8_t>();
            ba.nodes = ctx->gsort.nodes.as<BvhNode>();
            ba.recs = ctx->grec.as<GaussRec>();
            // it replaces the backward's own walk of the tree
            if (use_log) {
                ba.clog = ctx->clog.as<int32_t>();
                ba.cmask = ctx->cmask.as<uint8_t>();
                ba.cend = ctx->cend.as<int32_t>();
                ba.cdesc = ctx->blk_desc_c.as<uint2>();
                if (!ctx->clog_masks || !same_gauss)
                    GVC_CUDA(launch_log_masks(ba, ctx->cmask.as<uint8_t>(), ctx->cend.as<int32_t>(), moved, st),
                             "log masks");
                ctx->clog_masks = true;
            }
            const int tk = timer_begin(ctx, st, 1);
            GVC_CUDA(launch_backward_tc(ba, st), "backward (tensor core)");
            timer_end(ctx, st, tk);
        } else {
            const RowTreeSize z = row_tree_size(S);
            GVC_CUDA(ctx->b_rows.ensure(z.rows_bytes), "alloc gradient rows");
            GVC_CUDA(ctx->b_boxes.ensure(sizeof(float4) * 2 * z.tree.boxes), "alloc sample tree");
            GVC_CUDA(launch_backward_rows(S, z, ctx->s_sorted.as<float4>(), out_sorted, out_cells, out_weights,
                                          dL_dout_cells, dL_dout_weights, ctx->b_rows.as<float>(),
                                          ctx->b_boxes.as<float4>(), st),
                     "gradient rows");
            tm.mark();
            ba.gorder = have_order ? ctx->gsort.perm.as<int32_t>() : nullptr;
            ba.means = means3D;
            ba.values = values;
            ba.weights = weights;
            const int tk = timer_begin(ctx, st, 1);
            GVC_CUDA(launch_backward_gauss(ba, wide_tree_at(z.tree, ctx->b_boxes.as<float4>()),
                                           ctx->b_rows.as<float>(), st),
                     "backward (Gaussian-owned)");
            timer_end(ctx, st, tk);
        }
    }
    tm.mark();
    GVC_CUDA(launch_finalize(P, gacc, scales, rotations, conics, scale_modifier, ctx->cov_grad_mode, dmeans, dscales,
                             drots, dvalues, dweights, st),
             "finalize");
    tm.mark();
    if (debug) {
        int rc = debug_check(ctx, st);
        printf("Backward render time: %g ms\nBackward preprocess time: %g ms\n", tm.ms(1, 2), tm.ms(2, 3));
        if (rc) return rc;
    }
    return GVC_OK;
}

int gvc_sample_uniform(gvc_ctx* ctx, const int64_t* dims, const float* origin, const float* spacing,
                       const void* values, int dtype, int64_t N, const float* samples, void* out, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (!dims || !origin || !spacing) return fail(ctx, GVC_ERR_ARG, "dims/origin/spacing must be host arrays");
    if (dtype < GVC_F64 || dtype > GVC_U8)
        return fail(ctx, GVC_ERR_UNSUPPORTED, "Unsupported values dtype. Expected float64, float32, uint16, or uint8.");
    for (int a = 0; a < 3; a++)
        if (dims[a] < 1) return fail(ctx, GVC_ERR_ARG, "dims must be >= 1");
    if (N < 0) return fail(ctx, GVC_ERR_ARG, "negative sample count");
    if (N > 0 && (!values || !samples || !out)) return fail(ctx, GVC_ERR_ARG, "null pointer");
    GVC_CUDA(launch_sample_uniform(dims, origin, spacing, values, dtype, N, samples, out, (cudaStream_t)stream),
             "sample_uniform");
    return GVC_OK;
}

// Orders the C cells of scratch tmp_boxes, builds their tree and locates the samples (conn4: of
// tetrahedra).
static int locate(gvc_ctx* ctx, LocateArgs& la, int64_t C, const float* pts, const int32_t* conn4, cudaStream_t st) {
    la.C = C;
    if (C > 0) {
        const float4* boxes = scratch_of(ctx)->tmp_boxes.as<float4>();
        GVC_CUDA(morton_sort_boxes(ctx->cells, C, boxes, st), "cell order");
        GVC_CUDA(ctx->cell_tree.ensure(sizeof(float4) * 2 * wide_tree_size(C).boxes), "alloc cell tree");
        if (conn4) GVC_CUDA(ctx->cell_recs.ensure(sizeof(float4) * 8 * C), "alloc cell records");
        float4* recs = conn4 ? ctx->cell_recs.as<float4>() : nullptr;
        la.cperm = ctx->cells.perm.as<int32_t>();
        la.tree_boxes = ctx->cell_tree.as<float4>();
        la.recs = recs;
        GVC_CUDA(launch_cell_tree(C, ctx->cells.perm.as<int32_t>(), boxes, pts, conn4, recs, ctx->cell_tree.as<float4>(), st), "cell tree");
    }
    GVC_CUDA(launch_locate(la, st), "locate samples");
    return GVC_OK;
}

int gvc_sample_tets(gvc_ctx* ctx, int64_t npts, const float* pts, int64_t C, const int32_t* conn4,
                    const double* values, int64_t N, const float* samples, double* out, int64_t* cell_ids,
                    void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (npts < 0 || C < 0 || N < 0) return fail(ctx, GVC_ERR_ARG, "negative size");
    if (C > kMaxElems || N > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "mesh or sample count out of range");
    if (N > 0 && (!samples || !out)) return fail(ctx, GVC_ERR_ARG, "null pointer");
    if (C > 0 && (!pts || !conn4 || !values)) return fail(ctx, GVC_ERR_ARG, "null mesh pointer");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    if (N == 0) return GVC_OK;
    if (C > 0) {
        GVC_CUDA(sc->tmp_boxes.ensure(sizeof(float4) * 2 * C), "alloc cell boxes");
        GVC_CUDA(launch_tet_boxes(C, pts, conn4, sc->tmp_boxes.as<float4>(), st), "tet boxes");
    }
    GVC_CUDA(morton_sort_points(sc->msamp, N, samples, st), "sample order");
    LocateArgs la{};
    la.N = N;
    la.samples = samples;
    la.sperm = sc->msamp.perm.as<int32_t>();
    la.values = values;
    la.out = out;
    la.cell_ids = cell_ids;
    return locate(ctx, la, C, pts, conn4, st);
}

int gvc_knn3_mean_dist2(gvc_ctx* ctx, int64_t n, const float* pts, float* out, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (n < 0) return fail(ctx, GVC_ERR_ARG, "negative point count");
    if (n > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "point count out of range");
    if (n == 0) return GVC_OK;
    if (!pts || !out) return fail(ctx, GVC_ERR_ARG, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    GVC_CUDA(morton_sort_points(ctx->knn, n, pts, st), "point order");
    GVC_CUDA(ctx->knn_points.ensure(sizeof(float4) * n), "alloc points");
    float4* sorted = ctx->knn_points.as<float4>();
    GVC_CUDA(launch_knn_points(n, pts, ctx->knn.perm.as<int32_t>(), sorted, st), "sorted points");
    GVC_CUDA(lbvh_hierarchy_points(ctx->knn, n, ctx->knn.keys.as<uint32_t>(), sorted, st), "point LBVH");
    GVC_CUDA(launch_knn3(n, sorted, ctx->knn.nodes.as<BvhNode>(), out, ctx->d_status, st), "knn3");
    return GVC_OK;
}

int64_t gvc_training_workspace(int64_t C, int64_t num_batches, int64_t batch_size, int with_gt) {
    if (C < 0 || num_batches < 0 || batch_size < 0 || C > kMaxElems) return 0;
    if (batch_size > 0 && num_batches > kMaxElems / batch_size) return 0;
    size_t total = 0;
    training_buffers(nullptr, C, num_batches * batch_size, with_gt != 0,
                     [&](DevBuf*, size_t n) { total += round256(n); });
    return (int64_t)total;
}

int gvc_training_samples_in(gvc_ctx* ctx, int64_t npts, const float* pts, int64_t C, const int32_t* conn4,
                            const double* values, int64_t num_batches, int64_t batch_size, uint64_t seed,
                            float* samples_out, float* gt_out, void* workspace, int64_t workspace_bytes,
                            void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (workspace_bytes < 0 || (workspace_bytes > 0 && !workspace) || ((uintptr_t)workspace & 255u))
        return fail(ctx, GVC_ERR_ARG, "workspace must be 256-byte aligned");
    const bool sized = C > 0 && C <= kMaxElems && num_batches > 0 && batch_size > 0 &&
                       num_batches <= kMaxElems / batch_size;
    if (sized) {
        char* p = (char*)workspace;
        size_t left = (size_t)workspace_bytes;
        training_buffers(ctx, C, num_batches * batch_size, gt_out != nullptr, [&](DevBuf* b, size_t n) {
            if (round256(n) > left) return;  // the call allocates what does not fit
            b->lend(p, round256(n));
            p += round256(n);
            left -= round256(n);
        });
    }
    const int rc = gvc_training_samples(ctx, npts, pts, C, conn4, values, num_batches, batch_size, seed, samples_out,
                                        gt_out, stream);
    if (sized) training_buffers(ctx, C, num_batches * batch_size, true, [](DevBuf* b, size_t) { b->give_back(); });
    return rc;
}

int gvc_upload(gvc_ctx* ctx, int n, void* const* dst, const void* const* src, const int64_t* bytes, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (n < 0 || (n > 0 && (!dst || !src || !bytes))) return fail(ctx, GVC_ERR_ARG, "null array list");
    for (int i = 0; i < n; i++)
        if (bytes[i] < 0 || (bytes[i] > 0 && (!dst[i] || !src[i]))) return fail(ctx, GVC_ERR_ARG, "null array");
    GVC_CUDA(scratch_of(ctx)->stage.upload(ctx->device, n, dst, src, bytes, (cudaStream_t)stream), "upload");
    return GVC_OK;
}

int gvc_download(gvc_ctx* ctx, void* dst, const void* src, int64_t bytes, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (bytes < 0 || (bytes > 0 && (!dst || !src))) return fail(ctx, GVC_ERR_ARG, "null array");
    GVC_CUDA(scratch_of(ctx)->stage.download(ctx->device, dst, src, bytes, (cudaStream_t)stream), "download");
    return GVC_OK;
}

int gvc_check_cells(gvc_ctx* ctx, int64_t C, const int64_t* cell_types, const int64_t* cell_offsets, int64_t n_conn,
                    const int64_t* conn, int64_t npts, uint8_t* types_out, int32_t* conn_out, int64_t* result,
                    void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (C < 0 || n_conn < 0 || npts < 0) return fail(ctx, GVC_ERR_ARG, "negative size");
    if (!result || (n_conn > 0 && (!conn || !conn_out)) || (cell_types && (!cell_offsets || !types_out)))
        return fail(ctx, GVC_ERR_ARG, "null pointer");
    GVC_CUDA(launch_check_cells(C, cell_types, cell_offsets, n_conn, conn, npts, types_out, conn_out, result,
                                (cudaStream_t)stream),
             "check cells");
    return GVC_OK;
}

int gvc_training_samples(gvc_ctx* ctx, int64_t npts, const float* pts, int64_t C, const int32_t* conn4,
                         const double* values, int64_t num_batches, int64_t batch_size, uint64_t seed,
                         float* samples_out, float* gt_out, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (npts < 0 || C < 0 || num_batches < 0 || batch_size < 0) return fail(ctx, GVC_ERR_ARG, "negative size");
    if (C == 0 || npts == 0) return fail(ctx, GVC_ERR_ARG, "the mesh has no cells or no points");
    if (num_batches == 0 || batch_size == 0) return GVC_OK;
    if (C > kMaxElems || batch_size > kMaxElems || num_batches > kMaxElems / batch_size)
        return fail(ctx, GVC_ERR_CAPACITY, "num_batches * batch_size out of range");
    if (!pts || !conn4 || !samples_out || (gt_out && !values)) return fail(ctx, GVC_ERR_ARG, "null pointer");
    const int64_t N = num_batches * batch_size;
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    GVC_CUDA(ctx->ts_points.ensure(sizeof(float) * 3 * N), "alloc sample points");
    GVC_CUDA(ctx->ts_words.ensure(sizeof(uint32_t) * 3 * N), "alloc sort keys");
    uint32_t* w = ctx->ts_words.as<uint32_t>();
    GVC_CUDA(launch_tet_points(N, batch_size, seed, pts, conn4, C, ctx->ts_points.as<float>(), w, w + N, w + 2 * N,
                               st),
             "tet points");
    // batch index most significant, then the 63-bit Morton code (high word, low word)
    int batch_bits = 0;
    while (batch_bits < 32 && (uint64_t(1) << batch_bits) < (uint64_t)num_batches) batch_bits++;
    const uint32_t* words[3] = {w, w + N, w + 2 * N};
    const int bits[3] = {32, 31, batch_bits};
    GVC_CUDA(radix_sort_words(ctx->ts_sort, N, words, bits, batch_bits > 0 ? 3 : 2, st), "batch Morton sort");
    GVC_CUDA(launch_gather_points(N, ctx->ts_points.as<float>(), ctx->ts_sort.perm.as<int32_t>(), samples_out, st),
             "gather samples");
    if (!gt_out) return GVC_OK;
    GVC_CUDA(sc->tmp_boxes.ensure(sizeof(float4) * 2 * C), "alloc cell boxes");
    GVC_CUDA(launch_tet_boxes(C, pts, conn4, sc->tmp_boxes.as<float4>(), st), "tet boxes");
    // the samples are Morton-sorted per batch already: locate them in that order
    LocateArgs la{};
    la.N = N;
    la.samples = samples_out;
    la.values = values;
    la.out32 = gt_out;
    return locate(ctx, la, C, pts, conn4, st);
}

int gvc_sample_cells(gvc_ctx* ctx, int64_t npts, const float* pts, int64_t C, const uint8_t* cell_types,
                     const int64_t* cell_offsets, const int32_t* conn, const double* values, int64_t N,
                     const float* samples, double* out, int64_t* cell_ids, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (npts < 0 || C < 0 || N < 0) return fail(ctx, GVC_ERR_ARG, "negative size");
    if (C > kMaxElems || N > kMaxElems) return fail(ctx, GVC_ERR_CAPACITY, "mesh or sample count out of range");
    if (N > 0 && (!samples || !out)) return fail(ctx, GVC_ERR_ARG, "null pointer");
    if (C > 0 && (!pts || !cell_types || !cell_offsets || !conn || !values))
        return fail(ctx, GVC_ERR_ARG, "null mesh pointer");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    if (N == 0) return GVC_OK;
    if (C > 0) {
        GVC_CUDA(sc->tmp_boxes.ensure(sizeof(float4) * 2 * C), "alloc cell boxes");
        GVC_CUDA(launch_cell_boxes(C, pts, cell_types, cell_offsets, conn, sc->tmp_boxes.as<float4>(), st),
                 "cell boxes");
    }
    GVC_CUDA(morton_sort_points(sc->msamp, N, samples, st), "sample order");
    LocateArgs la{};
    la.N = N;
    la.samples = samples;
    la.sperm = sc->msamp.perm.as<int32_t>();
    la.values = values;
    la.pts = pts;
    la.types = cell_types;
    la.offsets = cell_offsets;
    la.conn = conn;
    la.out = out;
    la.cell_ids = cell_ids;
    return locate(ctx, la, C, nullptr, nullptr, st);
}

int gvc_debug_lbvh(gvc_ctx* ctx, int64_t n, const float* boxes, uint32_t* keys_sorted, int32_t* perm,
                   int32_t* left, int32_t* right, float* node_boxes, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (n <= 0 || n > kMaxElems) return fail(ctx, GVC_ERR_ARG, "n out of range");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    GVC_CUDA(sc->tmp_boxes.ensure(sizeof(float4) * 2 * n), "alloc");
    k_boxes6_to_f4<<<nb(n, 256), 256, 0, st>>>(n, boxes, sc->tmp_boxes.as<float4>()); gvc::note_launch();
    GVC_CUDA(lbvh_build_boxes(sc->dbg, n, sc->tmp_boxes.as<float4>(), st), "LBVH");
    if (keys_sorted)
        GVC_CUDA(cudaMemcpyAsync(keys_sorted, sc->dbg.keys.ptr, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st),
                 "copy keys");
    if (perm)
        GVC_CUDA(cudaMemcpyAsync(perm, sc->dbg.perm.ptr, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st),
                 "copy perm");
    if (n > 1 && (left || right || node_boxes)) {
        k_karras_tree<<<nb(n - 1, 256), 256, 0, st>>>((int)n, sc->dbg.nodes.as<BvhNode>(), sc->dbg.keys.as<uint32_t>(),
                                                      left, right, node_boxes, nullptr); gvc::note_launch();
    }
    GVC_CUDA(cudaGetLastError(), "debug lbvh");
    return GVC_OK;
}

int gvc_debug_lbvh_escape(gvc_ctx* ctx, int32_t* escape, void* stream) {
    if (!ctx || !escape) return GVC_ERR_ARG;
    Scratch* sc = scratch_of(ctx);
    const int64_t n = sc->dbg.n;
    if (n <= 0) return fail(ctx, GVC_ERR_STATE, "gvc_debug_lbvh has not built a tree");
    cudaStream_t st = (cudaStream_t)stream;
    if (n == 1) {
        GVC_CUDA(cudaMemsetAsync(escape, 0xff, sizeof(int32_t), st), "debug lbvh escape");
        return GVC_OK;
    }
    k_karras_tree<<<nb(n - 1, 256), 256, 0, st>>>((int)n, sc->dbg.nodes.as<BvhNode>(), sc->dbg.keys.as<uint32_t>(),
                                                  nullptr, nullptr, nullptr, escape); gvc::note_launch();
    GVC_CUDA(cudaGetLastError(), "debug lbvh escape");
    return GVC_OK;
}

int gvc_debug_preprocess(gvc_ctx* ctx, int64_t P, const float* means3D, const float* scales, const float* rotations,
                         const float* weights, float scale_modifier, float* conics, float* aabbs, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (P <= 0 || P > kMaxElems) return fail(ctx, GVC_ERR_ARG, "P out of range");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch* sc = scratch_of(ctx);
    GVC_CUDA(sc->tmp_boxes.ensure(sizeof(float4) * 2 * P), "alloc");
    GVC_CUDA(launch_preprocess(P, means3D, scales, rotations, weights, scale_modifier, conics,
                               sc->tmp_boxes.as<float4>(), st),
             "preprocess");
    if (aabbs) k_f4_to_boxes6<<<nb(P, 256), 256, 0, st>>>(P, sc->tmp_boxes.as<float4>(), aabbs); gvc::note_launch();
    GVC_CUDA(cudaGetLastError(), "debug preprocess");
    return GVC_OK;
}

int gvc_debug_tc_gemm(gvc_ctx* ctx, const void* A, const void* B, int N, float* D, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (N < 32 || N > 256 || N % 32) return fail(ctx, GVC_ERR_ARG, "N must be a multiple of 32 in [32, 256]");
    if (!A || !B || !D) return fail(ctx, GVC_ERR_ARG, "null pointer");
    GVC_CUDA(launch_tc_gemm_test(A, B, N, D, ctx->d_status, (cudaStream_t)stream), "tc gemm");
    return GVC_OK;
}

int gvc_debug_wait_timeout(gvc_ctx* ctx, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    GVC_CUDA(launch_wait_timeout_test(ctx->d_status, (cudaStream_t)stream), "wait timeout");
    return GVC_OK;
}

int gvc_debug_sort_timeout(gvc_ctx* ctx, int64_t n, const float* pts, int32_t* perm, float* slots, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (n <= kRsTile || n > (1 << 20)) return fail(ctx, GVC_ERR_ARG, "n out of range");
    if (!pts || !perm || !slots) return fail(ctx, GVC_ERR_ARG, "null pointer");
    cudaStream_t st = (cudaStream_t)stream;
    Lbvh& L = scratch_of(ctx)->dbg;
    L.n = 0;
    GVC_CUDA(morton_sort_points_withheld(L, n, pts, st), "withheld sort");
    GVC_CUDA(launch_sample_slots(n, n, pts, L.perm.as<int32_t>(), reinterpret_cast<float4*>(slots), st), "slots");
    GVC_CUDA(cudaMemcpyAsync(perm, L.perm.ptr, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, st), "copy perm");
    return GVC_OK;
}

int gvc_debug_sample_order(gvc_ctx* ctx, int32_t* perm, uint32_t* keys, void* stream) {
    if (!ctx) return GVC_ERR_ARG;
    if (!ctx->samples_ready) return fail(ctx, GVC_ERR_STATE, "no samples");
    cudaStream_t st = (cudaStream_t)stream;
    if (ctx->S == 0) return GVC_OK;
    if (perm)
        GVC_CUDA(cudaMemcpyAsync(perm, ctx->s_sort.perm.ptr, sizeof(int32_t) * ctx->S, cudaMemcpyDeviceToDevice, st),
                 "copy perm");
    if (keys)
        GVC_CUDA(cudaMemcpyAsync(keys, ctx->s_sort.keys.ptr, sizeof(uint32_t) * ctx->S, cudaMemcpyDeviceToDevice, st),
                 "copy keys");
    return GVC_OK;
}

}  // extern "C"
