// mesh.cu -- point sampling of structured (uniform) and tetrahedral meshes.
//
// Replaces the Viskores Probe filter calls of gpu_sampling/sample_mesh.cu:155-167
// (uniform point field) and :380-390 (explicit cells).  Compiled with --fmad=false:
// the double-precision locate / interpolate arithmetic rounds after every operation,
// as the oracle does, so cell ids and values are reproducible bit for bit.
//
// Declared semantics (the reference's Viskores internals are not vendored):
//   uniform: f = (x - o) / sp per axis; inside iff 0 <= f <= n-1; cell
//            i = min(floor(f), n-2); trilinear lerp a + t (b - a) along x, y, z;
//            outside -> -1 converted to the value dtype.
//   tets:    orient(a,b,c,d) = det[b-a, c-a, d-a]; closed containment by sub-volume
//            signs; degenerate tets never contain; ties -> lowest cell id;
//            value = sum_k (V_k / V) f_k; outside -> -1, cell -1.
#include "render.cuh"
#include "traverse.cuh"

namespace gvc {

template <class T>
__device__ __forceinline__ double ld_val(const void* v, int64_t i) {
    return (double)reinterpret_cast<const T*>(v)[i];
}

__device__ __forceinline__ double load_value(const void* v, int dtype, int64_t i) {
    switch (dtype) {
        case GVC_F64: return ld_val<double>(v, i);
        case GVC_F32: return ld_val<float>(v, i);
        case GVC_U16: return ld_val<uint16_t>(v, i);
        default: return ld_val<uint8_t>(v, i);
    }
}

// Integer outputs round half up and saturate; invalid (-1) wraps like a C cast of -1
// to the unsigned type (255 / 65535).
__device__ __forceinline__ void store_value(void* out, int dtype, int64_t i, double v, bool valid) {
    switch (dtype) {
        case GVC_F64: reinterpret_cast<double*>(out)[i] = valid ? v : -1.0; break;
        case GVC_F32: reinterpret_cast<float*>(out)[i] = valid ? (float)v : -1.0f; break;
        case GVC_U16: {
            uint16_t r = 0xffffu;
            if (valid) {
                double t = floor(v + 0.5);
                r = t <= 0.0 ? 0u : (t >= 65535.0 ? 65535u : (uint16_t)t);
            }
            reinterpret_cast<uint16_t*>(out)[i] = r;
            break;
        }
        default: {
            uint8_t r = 0xffu;
            if (valid) {
                double t = floor(v + 0.5);
                r = t <= 0.0 ? 0u : (t >= 255.0 ? 255u : (uint8_t)t);
            }
            reinterpret_cast<uint8_t*>(out)[i] = r;
        }
    }
}

struct UniformGrid {
    int64_t n[3];
    float o[3], sp[3];
};

__device__ __forceinline__ double lerp_d(double a, double b, double t) { return a + t * (b - a); }

__global__ void __launch_bounds__(256) k_sample_uniform(UniformGrid g, const void* __restrict__ values, int dtype,
                                                        int64_t N, const float* __restrict__ samples, void* out) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= N) return;
    int64_t ci[3];
    double t[3];
    bool ok = true;
    for (int a = 0; a < 3; a++) {
        const double f = ((double)samples[3 * s + a] - (double)g.o[a]) / (double)g.sp[a];
        const int64_t n = g.n[a];
        if (!(f >= 0.0) || !(f <= (double)(n - 1))) {
            ok = false;
            break;
        }
        if (n == 1) {
            ci[a] = 0;
            t[a] = 0.0;
            continue;
        }
        int64_t i = (int64_t)floor(f);
        if (i > n - 2) i = n - 2;
        ci[a] = i;
        t[a] = f - (double)i;
    }
    if (!ok) {
        store_value(out, dtype, s, 0.0, false);
        return;
    }
    const int64_t nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const int64_t sx = nx > 1 ? 1 : 0, sy = ny > 1 ? nx : 0, sz = nz > 1 ? nx * ny : 0;
    const int64_t b = ci[0] + nx * (ci[1] + ny * ci[2]);
    const double v000 = load_value(values, dtype, b), v100 = load_value(values, dtype, b + sx);
    const double v010 = load_value(values, dtype, b + sy), v110 = load_value(values, dtype, b + sx + sy);
    const double v001 = load_value(values, dtype, b + sz), v101 = load_value(values, dtype, b + sx + sz);
    const double v011 = load_value(values, dtype, b + sy + sz), v111 = load_value(values, dtype, b + sx + sy + sz);
    const double c00 = lerp_d(v000, v100, t[0]), c10 = lerp_d(v010, v110, t[0]);
    const double c01 = lerp_d(v001, v101, t[0]), c11 = lerp_d(v011, v111, t[0]);
    const double c0 = lerp_d(c00, c10, t[1]), c1 = lerp_d(c01, c11, t[1]);
    store_value(out, dtype, s, lerp_d(c0, c1, t[2]), true);
}

// ---------------------------------------------------------------------------------
// Tetrahedra
// ---------------------------------------------------------------------------------
__device__ __forceinline__ double det3(double ux, double uy, double uz, double vx, double vy, double vz, double wx,
                                       double wy, double wz) {
    const double m0 = vy * wz - vz * wy;
    const double m1 = vx * wz - vz * wx;
    const double m2 = vx * wy - vy * wx;
    double r = ux * m0;
    r = r - uy * m1;
    r = r + uz * m2;
    return r;
}

__device__ __forceinline__ double orient(const float* a, const float* b, const float* c, const float* d) {
    const double ax = a[0], ay = a[1], az = a[2];
    return det3((double)b[0] - ax, (double)b[1] - ay, (double)b[2] - az, (double)c[0] - ax, (double)c[1] - ay,
                (double)c[2] - az, (double)d[0] - ax, (double)d[1] - ay, (double)d[2] - az);
}

__device__ __forceinline__ bool tet_contains(const float* a, const float* b, const float* c, const float* d,
                                             const float* p, double lam[4]) {
    const double V = orient(a, b, c, d);
    if (V == 0.0) return false;
    const double Va = orient(p, b, c, d), Vb = orient(a, p, c, d), Vc = orient(a, b, p, d), Vd = orient(a, b, c, p);
    if (V > 0) {
        if (Va < 0 || Vb < 0 || Vc < 0 || Vd < 0) return false;
    } else {
        if (Va > 0 || Vb > 0 || Vc > 0 || Vd > 0) return false;
    }
    lam[0] = Va / V;
    lam[1] = Vb / V;
    lam[2] = Vc / V;
    lam[3] = Vd / V;
    return true;
}

__global__ void __launch_bounds__(256) k_tet_boxes(int64_t C, const float* __restrict__ pts,
                                                   const int32_t* __restrict__ conn4, float4* __restrict__ boxes) {
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= C) return;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int k = 0; k < 4; k++) {
        const float* v = pts + 3 * (int64_t)conn4[4 * c + k];
        for (int a = 0; a < 3; a++) {
            lo[a] = fminf(lo[a], v[a]);
            hi[a] = fmaxf(hi[a], v[a]);
        }
    }
    boxes[2 * c] = make_float4(lo[0], lo[1], lo[2], 0.f);
    boxes[2 * c + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
}

constexpr int kPointStack = 96;

// One thread per sample, in the caller's order: point query of the cell LBVH with a
// per-thread stack; every containing tet is tested and the lowest id kept (noalloc.cu; samples
// in Morton order take k_locate).
__global__ void __launch_bounds__(128) k_sample_tets(int64_t N, const float* __restrict__ samples,
                                                     const int32_t* __restrict__ sperm, const float* __restrict__ pts,
                                                     const int32_t* __restrict__ conn4,
                                                     const double* __restrict__ values,
                                                     const BvhNode* __restrict__ nodes,
                                                     const int32_t* __restrict__ cperm, int64_t C,
                                                     double* __restrict__ out, int64_t* __restrict__ cell_ids,
                                                     int* status) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int64_t s = sperm ? sperm[i] : i;
    const float p[3] = {samples[3 * s], samples[3 * s + 1], samples[3 * s + 2]};
    int64_t best = -1;
    double best_v = -1.0;
    if (C > 0) {
        int stack[kPointStack];
        int sp = 0;
        stack[sp++] = 0;
        while (sp > 0) {
            const int node = stack[--sp];
            const float4* np = reinterpret_cast<const float4*>(nodes + node);
            const float4 a = __ldg(np), b = __ldg(np + 1), c = __ldg(np + 2), d = __ldg(np + 3);
            const uint32_t ch[2] = {__float_as_uint(a.w), __float_as_uint(d.w)};
            const bool hit[2] = {a.x <= p[0] && p[0] <= b.x && a.y <= p[1] && p[1] <= b.y && a.z <= p[2] && p[2] <= b.z,
                                 c.x <= p[0] && p[0] <= d.x && c.y <= p[1] && p[1] <= d.y && c.z <= p[2] && p[2] <= d.z};
            for (int k = 0; k < 2; k++) {
                if (!hit[k]) continue;
                if (ch[k] & kLeafBit) {
                    const int64_t cell = cperm[ch[k] & ~kLeafBit];
                    if (best >= 0 && cell > best) continue;
                    const int32_t* cv = conn4 + 4 * cell;
                    double lam[4];
                    if (tet_contains(pts + 3 * (int64_t)cv[0], pts + 3 * (int64_t)cv[1], pts + 3 * (int64_t)cv[2],
                                     pts + 3 * (int64_t)cv[3], p, lam)) {
                        double v = lam[0] * values[cv[0]];
                        v = v + lam[1] * values[cv[1]];
                        v = v + lam[2] * values[cv[2]];
                        v = v + lam[3] * values[cv[3]];
                        best = cell;
                        best_v = v;
                    }
                } else if (sp < kPointStack) {
                    stack[sp++] = (int)ch[k];
                } else {
                    atomicOr(status, kStatusStackOverflow);
                }
            }
        }
    }
    out[s] = best >= 0 ? best_v : -1.0;
    if (cell_ids) cell_ids[s] = best;
}

// ---------------------------------------------------------------------------------
// General explicit cells: VTK_TETRA (10), VTK_HEXAHEDRON (12), VTK_WEDGE (13),
// VTK_PYRAMID (14) with isoparametric shape functions in VTK node order; the point is
// mapped to parametric coordinates by Newton's method in double (same expressions, same
// iteration rule as the oracle); zero-volume cells (1, 3, 5, 9) never contain a point.
// ---------------------------------------------------------------------------------
constexpr int kNewtonIters = 20;
constexpr double kNewtonTol = 1e-13;
constexpr double kInsideEps = 1e-9;

__device__ __forceinline__ int cell_npts(int type) {
    return type == 10 ? 4 : (type == 12 ? 8 : (type == 13 ? 6 : (type == 14 ? 5 : 0)));
}

__device__ int shape_eval(int type, double r, double s, double t, double N[8], double dN[8][3]) {
    if (type == 12) {
        const double rm = 1.0 - r, sm = 1.0 - s, tm = 1.0 - t;
        N[0] = rm * sm * tm; N[1] = r * sm * tm; N[2] = r * s * tm; N[3] = rm * s * tm;
        N[4] = rm * sm * t;  N[5] = r * sm * t;  N[6] = r * s * t;  N[7] = rm * s * t;
        dN[0][0] = -(sm * tm); dN[0][1] = -(rm * tm); dN[0][2] = -(rm * sm);
        dN[1][0] = sm * tm;    dN[1][1] = -(r * tm);  dN[1][2] = -(r * sm);
        dN[2][0] = s * tm;     dN[2][1] = r * tm;     dN[2][2] = -(r * s);
        dN[3][0] = -(s * tm);  dN[3][1] = rm * tm;    dN[3][2] = -(rm * s);
        dN[4][0] = -(sm * t);  dN[4][1] = -(rm * t);  dN[4][2] = rm * sm;
        dN[5][0] = sm * t;     dN[5][1] = -(r * t);   dN[5][2] = r * sm;
        dN[6][0] = s * t;      dN[6][1] = r * t;      dN[6][2] = r * s;
        dN[7][0] = -(s * t);   dN[7][1] = rm * t;     dN[7][2] = rm * s;
        return 8;
    }
    if (type == 13) {
        const double u = 1.0 - r - s, tm = 1.0 - t;
        N[0] = u * tm; N[1] = r * tm; N[2] = s * tm; N[3] = u * t; N[4] = r * t; N[5] = s * t;
        dN[0][0] = -tm; dN[0][1] = -tm; dN[0][2] = -u;
        dN[1][0] = tm;  dN[1][1] = 0.0; dN[1][2] = -r;
        dN[2][0] = 0.0; dN[2][1] = tm;  dN[2][2] = -s;
        dN[3][0] = -t;  dN[3][1] = -t;  dN[3][2] = u;
        dN[4][0] = t;   dN[4][1] = 0.0; dN[4][2] = r;
        dN[5][0] = 0.0; dN[5][1] = t;   dN[5][2] = s;
        return 6;
    }
    if (type == 14) {
        const double rm = 1.0 - r, sm = 1.0 - s, tm = 1.0 - t;
        N[0] = rm * sm * tm; N[1] = r * sm * tm; N[2] = r * s * tm; N[3] = rm * s * tm; N[4] = t;
        dN[0][0] = -(sm * tm); dN[0][1] = -(rm * tm); dN[0][2] = -(rm * sm);
        dN[1][0] = sm * tm;    dN[1][1] = -(r * tm);  dN[1][2] = -(r * sm);
        dN[2][0] = s * tm;     dN[2][1] = r * tm;     dN[2][2] = -(r * s);
        dN[3][0] = -(s * tm);  dN[3][1] = rm * tm;    dN[3][2] = -(rm * s);
        dN[4][0] = 0.0;        dN[4][1] = 0.0;        dN[4][2] = 1.0;
        return 5;
    }
    return 0;
}

__device__ int iso_contains(int type, const float* __restrict__ pts, const int32_t* __restrict__ cv, const float* p,
                            double Nout[8]) {
    double r, s, t;
    if (type == 12) { r = 0.5; s = 0.5; t = 0.5; }
    else if (type == 13) { r = 1.0 / 3.0; s = 1.0 / 3.0; t = 0.5; }
    else { r = 0.5; s = 0.5; t = 0.25; }
    double N[8], dN[8][3];
    int n = 0;
    bool converged = false;
    for (int it = 0; it < kNewtonIters; it++) {
        n = shape_eval(type, r, s, t, N, dN);
        double f[3] = {0.0, 0.0, 0.0}, J[3][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
        for (int k = 0; k < n; k++) {
            const float* x = pts + 3 * (int64_t)cv[k];
            for (int a = 0; a < 3; a++) {
                f[a] = f[a] + N[k] * (double)x[a];
                for (int b = 0; b < 3; b++) J[a][b] = J[a][b] + dN[k][b] * (double)x[a];
            }
        }
        for (int a = 0; a < 3; a++) f[a] = f[a] - (double)p[a];
        const double det = det3(J[0][0], J[0][1], J[0][2], J[1][0], J[1][1], J[1][2], J[2][0], J[2][1], J[2][2]);
        if (det == 0.0 || det != det) return 0;
        const double d0 = det3(f[0], J[0][1], J[0][2], f[1], J[1][1], J[1][2], f[2], J[2][1], J[2][2]) / det;
        const double d1 = det3(J[0][0], f[0], J[0][2], J[1][0], f[1], J[1][2], J[2][0], f[2], J[2][2]) / det;
        const double d2 = det3(J[0][0], J[0][1], f[0], J[1][0], J[1][1], f[1], J[2][0], J[2][1], f[2]) / det;
        r = r - d0;
        s = s - d1;
        t = t - d2;
        double m = fabs(d0);
        if (fabs(d1) > m) m = fabs(d1);
        if (fabs(d2) > m) m = fabs(d2);
        if (!(m >= kNewtonTol)) {
            converged = true;
            break;
        }
    }
    // an unconverged iterate says nothing about the point: not contained
    if (!converged) return 0;
    const double e = kInsideEps;
    bool inside;
    if (type == 13) inside = r >= -e && s >= -e && r + s <= 1.0 + e && t >= -e && t <= 1.0 + e;
    else inside = r >= -e && r <= 1.0 + e && s >= -e && s <= 1.0 + e && t >= -e && t <= 1.0 + e;
    if (!inside) return 0;
    n = shape_eval(type, r, s, t, N, dN);
    for (int k = 0; k < n; k++) Nout[k] = N[k];
    return n;
}

__global__ void __launch_bounds__(256) k_cell_boxes(int64_t C, const float* __restrict__ pts,
                                                    const uint8_t* __restrict__ types,
                                                    const int64_t* __restrict__ offsets,
                                                    const int32_t* __restrict__ conn, float4* __restrict__ boxes) {
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= C) return;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    const int n = cell_npts(types[c]);
    for (int k = 0; k < n; k++) {
        const float* v = pts + 3 * (int64_t)conn[offsets[c] + k];
        for (int a = 0; a < 3; a++) {
            lo[a] = fminf(lo[a], v[a]);
            hi[a] = fmaxf(hi[a], v[a]);
        }
    }
    boxes[2 * c] = make_float4(lo[0], lo[1], lo[2], 0.f);
    boxes[2 * c + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
}

// ---------------------------------------------------------------------------------
// Point location by a wide tree (wide_tree.cuh) over the Morton-sorted cells.
//
// One warp owns up to 32 Morton-sorted samples.  It walks the tree once with their box and
// keeps the level-1 nodes (8 cells) that it meets in shared memory.  Every sample is tested
// against every node's box; the (sample, node) pairs that meet are queued and 32 at a time
// tested against the node's eight cells, and the (sample, cell) pairs that meet are queued in
// turn, 32 at a time, so that no lane idles where samples meet different cells.  Of a
// tetrahedron's pairs, seven in eight are told to be outside by its four planes in FP32 (an
// error bound decides: k_cell_leaves); what they leave takes the containment test in double.
// The lowest containing cell of each sample is kept in shared memory.  A run of samples that
// jumps across the mesh would meet a large part of it: a walk that has met 8 nodes per sample
// of the run is given up and the run halved, down to single samples.
//
// A thread per sample with a stack of its own took a chain of twenty dependent node loads and
// three dependent gathers per cell (id, vertex numbers, vertices; here one 64-byte record), and
// ran every containment test at the pace of the warp's slowest lane: 1.57M tetrahedra x 25M
// samples 16.7 ms against 9.1.  Testing each sample against every cell met instead took
// 11.3k instructions per warp there, 16.4 ms.
// ---------------------------------------------------------------------------------
struct LocateSmem {
    float4 lo[64], hi[64];  // met nodes: at most 31 before a step of the walk adds up to 32; lo.w: node
    int2 nodes[64];         // (node, sample): at most 31 before a node adds up to 32
    int2 cells[64];         // (leaf, sample): at most 31 before a leaf adds up to 32
    int2 close[64];         // those that the planes leave: at most 31 before 32 cells add to them
    float px[32], py[32], pz[32];
    unsigned best[32];
    double val[32];
    WideStack walk;
};

struct CellMesh {
    const float4* recs;      // tetrahedra: four vertices per leaf, .w their numbers, four planes
    const float* pts;        // other cells
    const uint8_t* types;
    const int64_t* offsets;
    const int32_t* conn;
    const int32_t* perm;     // leaf -> cell
    const double* values;
};

constexpr int kNodesPerSample = 8;

// A tetrahedron's plane k is the volume spanned by a point and its face k over the
// tetrahedron's own, as an affine function of the point relative to the box's low corner,
// scaled to at most one in size over the box.  Below minus this bound the double-precision
// test finds the point outside too: rounding of the planes, of the relative point and of the
// four products and sums is below 8 x 2^-24, the double-precision volumes' own errors are 1e-9
// of the scale (a face below 1e-6 of the box's square gets no plane).
constexpr float kPlaneBound = 4e-6f;

// The pairs [off, off + n) of sm.close (tetrahedra) or sm.cells.  Not inlined, nor is the next: the containment test is
// long, and a copy at every place that empties a queue thrashed the instruction cache.
template <bool TETS>
__device__ __noinline__ void contain(LocateSmem& sm, const CellMesh& mesh, int off, int n) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    bool c = false;
    unsigned cell = 0;
    int s = 0;
    double v = 0.0;
    if (lane < n) {
        const int2 q = TETS ? sm.close[off + lane] : sm.cells[off + lane];
        s = q.y;
        cell = (unsigned)__ldg(mesh.perm + q.x);
        if (cell < sm.best[s]) {
            const float p[3] = {sm.px[s], sm.py[s], sm.pz[s]};
            if (TETS) {
                const float4* r = mesh.recs + 8 * (int64_t)q.x;
                const float4 a4 = __ldg(r), b4 = __ldg(r + 1), c4 = __ldg(r + 2), d4 = __ldg(r + 3);
                const float a[3] = {a4.x, a4.y, a4.z}, b[3] = {b4.x, b4.y, b4.z}, e[3] = {c4.x, c4.y, c4.z},
                            d[3] = {d4.x, d4.y, d4.z};
                double lam[4];
                c = tet_contains(a, b, e, d, p, lam);
                if (c) {
                    v = lam[0] * mesh.values[__float_as_int(a4.w)];
                    v = v + lam[1] * mesh.values[__float_as_int(b4.w)];
                    v = v + lam[2] * mesh.values[__float_as_int(c4.w)];
                    v = v + lam[3] * mesh.values[__float_as_int(d4.w)];
                }
            } else {
                const int type = mesh.types[cell];
                const int32_t* cv = mesh.conn + mesh.offsets[cell];
                if (type == 10) {
                    double lam[4];
                    c = tet_contains(mesh.pts + 3 * (int64_t)cv[0], mesh.pts + 3 * (int64_t)cv[1],
                                     mesh.pts + 3 * (int64_t)cv[2], mesh.pts + 3 * (int64_t)cv[3], p, lam);
                    if (c) {
                        v = lam[0] * mesh.values[cv[0]];
                        v = v + lam[1] * mesh.values[cv[1]];
                        v = v + lam[2] * mesh.values[cv[2]];
                        v = v + lam[3] * mesh.values[cv[3]];
                    }
                } else if (type == 12 || type == 13 || type == 14) {
                    double Nf[8];
                    const int k = iso_contains(type, mesh.pts, cv, p, Nf);
                    c = k != 0;
                    if (c) {
                        v = Nf[0] * mesh.values[cv[0]];
                        for (int i = 1; i < k; i++) v = v + Nf[i] * mesh.values[cv[i]];
                    }
                }
            }
            if (c) atomicMin(&sm.best[s], cell);
        }
    }
    __syncwarp();
    if (c && sm.best[s] == cell) sm.val[s] = v;
    __syncwarp();
}

// The pairs [off, off + n) of sm.cells; n_close: the length of sm.close, returned.
template <bool TETS>
__device__ __forceinline__ int narrow(LocateSmem& sm, const WideTree& tree, const CellMesh& mesh, int off, int n,
                                      int n_close) {
    if (!TETS) {
        contain<false>(sm, mesh, off, n);
        return 0;
    }
    const int lane = threadIdx.x & 31;
    __syncwarp();
    bool keep = false;
    int2 q;
    if (lane < n) {
        q = sm.cells[off + lane];
        const float4* r = mesh.recs + 8 * (int64_t)q.x + 4;
        const float4 lo = __ldg(tree.box[0] + 2 * (int64_t)q.x);
        const float4 p0 = __ldg(r), p1 = __ldg(r + 1), p2 = __ldg(r + 2), p3 = __ldg(r + 3);
        const float dx = sm.px[q.y] - lo.x, dy = sm.py[q.y] - lo.y, dz = sm.pz[q.y] - lo.z;
        const float g0 = fmaf(p0.x, dx, fmaf(p0.y, dy, fmaf(p0.z, dz, p0.w)));
        const float g1 = fmaf(p1.x, dx, fmaf(p1.y, dy, fmaf(p1.z, dz, p1.w)));
        const float g2 = fmaf(p2.x, dx, fmaf(p2.y, dy, fmaf(p2.z, dz, p2.w)));
        const float g3 = fmaf(p3.x, dx, fmaf(p3.y, dy, fmaf(p3.z, dz, p3.w)));
        keep = !(g0 < -kPlaneBound || g1 < -kPlaneBound || g2 < -kPlaneBound || g3 < -kPlaneBound);
    }
    const uint32_t m = __ballot_sync(0xffffffffu, keep);
    if (keep) sm.close[n_close + __popc(m & lane_lt_mask())] = q;
    n_close += __popc(m);
    if (n_close >= 32) {
        n_close -= 32;
        contain<true>(sm, mesh, n_close, 32);
    }
    __syncwarp();
    return n_close;
}

// The pairs [off, off + n) of sm.nodes: tests the cells of each node and queues the pairs that
// meet; len: the lengths of sm.cells and sm.close, returned.
template <bool TETS>
__device__ __noinline__ int2 expand(LocateSmem& sm, const WideTree& tree, const CellMesh& mesh, int off, int n,
                                    int2 len) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = lane_lt_mask();
    __syncwarp();
    const int2 q = lane < n ? sm.nodes[off + lane] : make_int2(0, 0);
    const float x = sm.px[q.y], y = sm.py[q.y], z = sm.pz[q.y];
    // the eight loads together, then the pairs
    uint32_t hits = 0;
    const float4* p = tree.box[0] + 2 * (int64_t)(q.x * kWideLeaves);
    const int leaves = lane < n ? min(tree.n[0] - q.x * kWideLeaves, kWideLeaves) : 0;
#pragma unroll
    for (int k = 0; k < kWideLeaves; k++) {
        if (k < leaves) {
            const float4 lo = __ldg(p + 2 * k), hi = __ldg(p + 2 * k + 1);
            if (lo.x <= x && x <= hi.x && lo.y <= y && y <= hi.y && lo.z <= z && z <= hi.z) hits |= 1u << k;
        }
    }
#pragma unroll 1
    for (int k = 0; k < kWideLeaves; k++) {
        const int leaf = q.x * kWideLeaves + k;
        const bool h = (hits >> k) & 1u;
        const uint32_t m = __ballot_sync(0xffffffffu, h);
        if (h) sm.cells[len.x + __popc(m & lt)] = make_int2(leaf, q.y);
        len.x += __popc(m);
        if (len.x >= 32) {
            len.x -= 32;
            len.y = narrow<TETS>(sm, tree, mesh, len.x, 32, len.y);
        }
    }
    __syncwarp();
    return len;
}

template <bool TETS>
struct Locator {
    LocateSmem& sm;
    const CellMesh& mesh;
    float x, y, z;
    const WideTree& tree;
    bool in;  // this lane's sample is in the current run
    int n_nodes;
    int2 n_cells;  // and n_close

    // met nodes [off, off + n) against the run's samples
    __device__ __forceinline__ void operator()(int off, int n) {
        const int lane = threadIdx.x & 31;
        const uint32_t lt = lane_lt_mask();
        __syncwarp();
        for (int j = off; j < off + n; j++) {
            const float4 lo = sm.lo[j], hi = sm.hi[j];
            const bool h = in && lo.x <= x && x <= hi.x && lo.y <= y && y <= hi.y && lo.z <= z && z <= hi.z;
            const uint32_t m = __ballot_sync(0xffffffffu, h);
            if (m == 0) continue;
            if (h) sm.nodes[n_nodes + __popc(m & lt)] = make_int2(__float_as_int(lo.w), lane);
            n_nodes += __popc(m);
            if (n_nodes >= 32) {
                n_nodes -= 32;
                n_cells = expand<TETS>(sm, tree, mesh, n_nodes, 32, n_cells);
            }
        }
        __syncwarp();
    }
};

// `rows` samples per warp, a power of two up to 32.  Blocks per SM asked for: tetrahedra 28 (72
// registers; 32 and 24: 1 % and 6 % slower), other cells 16 (128 registers, for Newton's method;
// 12 or 10 5 % and 8 36 % slower).
template <bool TETS, class Out>
__global__ void __launch_bounds__(32, TETS ? 28 : 16)
    k_locate(int64_t N, int rows, const float* __restrict__ samples, int32_t* __restrict__ sperm,
             const __grid_constant__ WideTree tree, const __grid_constant__ CellMesh mesh, Out* __restrict__ out,
             int64_t* __restrict__ cell_ids) {
    __shared__ LocateSmem sm;
    const int lane = threadIdx.x;
    const int64_t i = (int64_t)blockIdx.x * rows + lane;
    const bool valid = lane < rows && i < N;
    int64_t s = 0;
    float x = NAN, y = NAN, z = NAN;
    if (valid) {
        s = sperm ? order_at(sperm, i, N) : i;
        x = samples[3 * s];
        y = samples[3 * s + 1];
        z = samples[3 * s + 2];
    }
    sm.px[lane] = x;
    sm.py[lane] = y;
    sm.pz[lane] = z;
    sm.best[lane] = 0xffffffffu;
    __syncwarp();
    const bool number = x == x && y == y && z == z;  // a NaN lies in no cell
    Locator<TETS> loc{sm, mesh, x, y, z, tree, false, 0, make_int2(0, 0)};
    int a = 0, len = rows;
    while (a < rows) {
        loc.in = number && lane >= a && lane < a + len;
        const Box6 b = warp_point_box(loc.in, x, y, z);
        const float3 lo = make_float3(b.lx, b.ly, b.lz), hi = make_float3(b.hx, b.hy, b.hz);
        int n_wait = 0, n_met = 0, n_tested = 0;
        bool given_up = false;
        wide_walk_nodes<false>(tree, lo, hi, sm.walk, n_tested, [&](int first, uint32_t m) -> bool {
            n_met += __popc(m);
            if (len > 1 && n_met > kNodesPerSample * len) {
                given_up = true;
                return false;
            }
            if ((m >> lane) & 1u) {
                const float4* q = tree.box[1] + 2 * (int64_t)(first + lane);
                const int k = n_wait + __popc(m & lane_lt_mask());
                float4 l = __ldg(q);
                l.w = __int_as_float(first + lane);
                sm.lo[k] = l;
                sm.hi[k] = __ldg(q + 1);
            }
            n_wait += __popc(m);
            __syncwarp();
            if (n_wait >= 32) {
                n_wait -= 32;
                loc(n_wait, 32);
            }
            return true;
        });
        __syncwarp();
        if (given_up) {
            len >>= 1;
            continue;
        }
        if (n_wait > 0) loc(0, n_wait);
        a += len;
        len = a & -a;
    }
    if (loc.n_nodes > 0) loc.n_cells = expand<TETS>(sm, tree, mesh, 0, loc.n_nodes, loc.n_cells);
    if (loc.n_cells.x > 0) loc.n_cells.y = narrow<TETS>(sm, tree, mesh, 0, loc.n_cells.x, loc.n_cells.y);
    if (TETS && loc.n_cells.y > 0) contain<TETS>(sm, mesh, 0, loc.n_cells.y);
    if (valid) {
        const bool found = sm.best[lane] != 0xffffffffu;
        out[s] = (Out)(found ? sm.val[lane] : -1.0);
        if (cell_ids) cell_ids[s] = found ? (int64_t)sm.best[lane] : -1;
    }
}

// Plane of a face: sign * (p - at) . m over `scale`, as (coefficients, value at p = 0).
__device__ __forceinline__ float4 face_plane(const double m[3], const double at[3], double sign, double L) {
    const double n1 = fabs(m[0]) + fabs(m[1]) + fabs(m[2]);
    if (n1 < 1e-6 * L * L) return make_float4(0.f, 0.f, 0.f, 0.f);
    const double k = sign / (n1 * L);
    return make_float4((float)(k * m[0]), (float)(k * m[1]), (float)(k * m[2]),
                       (float)(-k * (m[0] * at[0] + m[1] * at[1] + m[2] * at[2])));
}
__device__ __forceinline__ void cross_d(const double u[3], const double v[3], double m[3]) {
    m[0] = u[1] * v[2] - u[2] * v[1];
    m[1] = u[2] * v[0] - u[0] * v[2];
    m[2] = u[0] * v[1] - u[1] * v[0];
}

// The four planes of kPlaneBound's comment: tet_contains compares the signs of
// (b - p) . ((c - b) x (d - b)), (p - a) . ((c - a) x (d - a)), (p - a) . ((d - a) x (b - a))
// and (p - a) . ((b - a) x (c - a)) with the whole volume's.
__device__ __forceinline__ void tet_planes(const float* a, const float* b, const float* c, const float* d, float4 lo,
                                           float4 hi, float4* out) {
    const double V = orient(a, b, c, d);
    const double L = fmax(fmax((double)hi.x - lo.x, (double)hi.y - lo.y), (double)hi.z - lo.z);
    if (V == 0.0 || !(L >= 1e-30 && L <= 1e30)) {
        // a degenerate tetrahedron contains nothing; out of range, the planes say nothing
        const float w = V == 0.0 ? -1.f : 0.f;
        for (int k = 0; k < 4; k++) out[k] = make_float4(0.f, 0.f, 0.f, w);
        return;
    }
    const double sign = V > 0.0 ? 1.0 : -1.0;
    const float o[3] = {lo.x, lo.y, lo.z};
    double A[3], B[3], ab[3], ac[3], ad[3], bc[3], bd[3], m[3];
    for (int k = 0; k < 3; k++) {
        A[k] = (double)a[k] - o[k];
        B[k] = (double)b[k] - o[k];
        ab[k] = (double)b[k] - a[k];
        ac[k] = (double)c[k] - a[k];
        ad[k] = (double)d[k] - a[k];
        bc[k] = (double)c[k] - b[k];
        bd[k] = (double)d[k] - b[k];
    }
    cross_d(bc, bd, m);
    out[0] = face_plane(m, B, -sign, L);
    cross_d(ac, ad, m);
    out[1] = face_plane(m, A, sign, L);
    cross_d(ad, ab, m);
    out[2] = face_plane(m, A, sign, L);
    cross_d(ab, ac, m);
    out[3] = face_plane(m, A, sign, L);
}

// Leaves of the tree in Morton order (levels 0 and 1) and, of tetrahedra, their records.
template <bool TETS>
__global__ void __launch_bounds__(256) k_cell_leaves(int64_t C, int32_t* __restrict__ perm,
                                                     const float4* __restrict__ boxes, const float* __restrict__ pts,
                                                     const int32_t* __restrict__ conn4, float4* __restrict__ recs,
                                                     float4* __restrict__ leaf, float4* __restrict__ level1) {
    const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    Box6 b = empty_box();
    if (g < C) {
        const int64_t o = order_at(perm, g, C);
        const float4 lo = boxes[2 * o], hi = boxes[2 * o + 1];
        if (TETS) {
            float p[4][3];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int v = conn4[4 * o + k];
#pragma unroll
                for (int i = 0; i < 3; i++) p[k][i] = pts[3 * (int64_t)v + i];
                recs[8 * g + k] = make_float4(p[k][0], p[k][1], p[k][2], __int_as_float(v));
            }
            tet_planes(p[0], p[1], p[2], p[3], lo, hi, recs + 8 * g + 4);
        }
        b = Box6{lo.x, lo.y, lo.z, hi.x, hi.y, hi.z};
        store_box(leaf, g, b);
    }
    grow(b, shfl_xor_box(b, 1));
    grow(b, shfl_xor_box(b, 2));
    grow(b, shfl_xor_box(b, 4));
    if (g < C && (g & (kWideLeaves - 1)) == 0) store_box(level1, g / kWideLeaves, b);
}

static inline unsigned nbk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// ---------------------------------------------------------------------------------
// Validation of cells given as int64 arrays, as they come from the caller: one pass on the
// device, at the pace of its memory, in place of a dozen passes over host arrays (384k
// tetrahedra 21 ms on the host).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ int vtk_npts(int64_t type) {
    switch (type) {
        case 1: return 1;
        case 3: return 2;
        case 5: return 3;
        case 9: case 10: return 4;
        case 12: return 8;
        case 13: return 6;
        case 14: return 5;
        default: return 0;
    }
}

__global__ void k_check_init(int64_t* r) {
    if (threadIdx.x < 6) r[threadIdx.x] = threadIdx.x == 0 ? INT64_MAX : 0;
}

__global__ void __launch_bounds__(256) k_check_types(int64_t C, const int64_t* __restrict__ types,
                                                     const int64_t* __restrict__ offsets, int64_t n_conn,
                                                     uint8_t* __restrict__ types_out, int64_t* __restrict__ r) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= C) return;
    const int64_t t = types[i];
    const int want = vtk_npts(t);
    types_out[i] = (uint8_t)t;
    const int64_t start = offsets[i], end = i + 1 < C ? offsets[i + 1] : n_conn;
    if (want == 0) atomicMin((long long*)r, (long long)i);
    if ((int64_t)((uint64_t)end - (uint64_t)start) != want || start < 0 || end > n_conn) r[1] = 1;
    if (t != 10) r[2] = 1;
}

__global__ void __launch_bounds__(256) k_check_conn(int64_t n_conn, const int64_t* __restrict__ conn, int64_t npts,
                                                    const int64_t* __restrict__ offsets,
                                                    int32_t* __restrict__ conn_out, int64_t* __restrict__ r) {
    const int64_t first = offsets ? offsets[0] : 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_conn; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = conn[i];
        const int32_t w = (int32_t)v;
        conn_out[i] = w;
        if (w < 0 || w >= npts) {
            r[3] = 1;
            if (i >= first) r[4] = 1;
        }
        if (v < 0 || v >= npts) r[5] = 1;
    }
}

cudaError_t launch_check_cells(int64_t C, const int64_t* types, const int64_t* offsets, int64_t n_conn,
                               const int64_t* conn, int64_t npts, uint8_t* types_out, int32_t* conn_out,
                               int64_t* result, cudaStream_t st) {
    k_check_init<<<1, 32, 0, st>>>(result); gvc::note_launch();
    if (types && C > 0) {
        k_check_types<<<nbk(C, 256), 256, 0, st>>>(C, types, offsets, n_conn, types_out, result); gvc::note_launch();
    }
    if (n_conn > 0) {
        const int64_t b = (n_conn + 255) / 256;
        k_check_conn<<<(unsigned)(b < 148 * 8 ? b : 148 * 8), 256, 0, st>>>(
            n_conn, conn, npts, types && C > 0 ? offsets : nullptr, conn_out, result); gvc::note_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_cell_boxes(int64_t C, const float* pts, const uint8_t* types, const int64_t* offsets,
                              const int32_t* conn, float4* boxes, cudaStream_t st) {
    if (C <= 0) return cudaSuccess;
    k_cell_boxes<<<nbk(C, 256), 256, 0, st>>>(C, pts, types, offsets, conn, boxes); gvc::note_launch();
    return cudaGetLastError();
}

cudaError_t launch_cell_tree(int64_t C, int32_t* perm, const float4* boxes, const float* pts,
                             const int32_t* conn4, float4* recs, float4* tree_boxes, cudaStream_t st) {
    if (C <= 0) return cudaSuccess;
    const WideTreeSize z = wide_tree_size(C);
    float4* level1 = tree_boxes + 2 * z.n[0];
    if (conn4) {
        k_cell_leaves<true><<<nbk(C, 256), 256, 0, st>>>(C, perm, boxes, pts, conn4, recs, tree_boxes, level1);
    } else {
        k_cell_leaves<false><<<nbk(C, 256), 256, 0, st>>>(C, perm, boxes, pts, nullptr, nullptr, tree_boxes, level1);
    }
    gvc::note_launch();
    return launch_wide_levels(z, tree_boxes, st);
}

template <bool TETS>
static void launch_locate_as(const LocateArgs& a, cudaStream_t st) {
    const WideTree tree = wide_tree_at(wide_tree_size(a.C), a.tree_boxes);
    const CellMesh mesh{a.recs, a.pts, a.types, a.offsets, a.conn, a.cperm, a.values};
    // fewer samples per warp where 32 would leave the chip's 148 x 28 resident warps partly idle
    int rows = 32;
    while (rows > 1 && a.N < (int64_t)148 * 28 * rows) rows >>= 1;
    const unsigned n = nbk(a.N, rows);
    if (a.out32) {
        k_locate<TETS><<<n, 32, 0, st>>>(a.N, rows, a.samples, a.sperm, tree, mesh, a.out32, a.cell_ids);
    } else {
        k_locate<TETS><<<n, 32, 0, st>>>(a.N, rows, a.samples, a.sperm, tree, mesh, a.out, a.cell_ids);
    }
    gvc::note_launch();
}

cudaError_t launch_locate(const LocateArgs& a, cudaStream_t st) {
    if (a.N <= 0) return cudaSuccess;
    if (a.recs) launch_locate_as<true>(a, st);
    else launch_locate_as<false>(a, st);
    return cudaGetLastError();
}

cudaError_t launch_sample_uniform(const int64_t dims[3], const float origin[3], const float spacing[3],
                                  const void* values, int dtype, int64_t N, const float* samples, void* out,
                                  cudaStream_t st) {
    if (N <= 0) return cudaSuccess;
    UniformGrid g;
    for (int a = 0; a < 3; a++) {
        g.n[a] = dims[a];
        g.o[a] = origin[a];
        g.sp[a] = spacing[a];
    }
    k_sample_uniform<<<nbk(N, 256), 256, 0, st>>>(g, values, dtype, N, samples, out); gvc::note_launch();
    return cudaGetLastError();
}

cudaError_t launch_tet_boxes(int64_t C, const float* pts, const int32_t* conn4, float4* boxes, cudaStream_t st) {
    if (C <= 0) return cudaSuccess;
    k_tet_boxes<<<nbk(C, 256), 256, 0, st>>>(C, pts, conn4, boxes); gvc::note_launch();
    return cudaGetLastError();
}

cudaError_t launch_sample_tets(int64_t N, const float* samples, const int32_t* sperm, const float* pts,
                               const int32_t* conn4, const double* values, const BvhNode* cnodes,
                               const int32_t* cperm, int64_t C, double* out, int64_t* cell_ids, int* status,
                               cudaStream_t st) {
    if (N <= 0) return cudaSuccess;
    k_sample_tets<<<nbk(N, 128), 128, 0, st>>>(N, samples, sperm, pts, conn4, values, cnodes, cperm, C, out,
                                               cell_ids, status); gvc::note_launch();
    return cudaGetLastError();
}

}  // namespace gvc
