// render.cu -- the per-Gaussian end of the backward: the eleven sums of bwd_gauss.cu or
// bwd_tc.cu become the gradients of a Gaussian's parameters
// (diff-gaussian-rasterization/cuda_rasterizer/backward.cu:9-125).
#include "render.cuh"

namespace gvc {

// --------------------------------------------------------------------------------
// Finalize: gacc [P][16] (caller order) -> dmeans, dvalues, dweights and the
// covariance adjoint dconic -> dscales, drots (one thread per Gaussian).
// --------------------------------------------------------------------------------
__device__ __forceinline__ void rot_cols(float r, float x, float y, float z, float Rc[3][3]) {
    // Rc[col][row]: glm's column-major fill of forward.cu:40-44
    Rc[0][0] = 1.f - 2.f * (y * y + z * z);
    Rc[0][1] = 2.f * (x * y - r * z);
    Rc[0][2] = 2.f * (x * z + r * y);
    Rc[1][0] = 2.f * (x * y + r * z);
    Rc[1][1] = 1.f - 2.f * (x * x + z * z);
    Rc[1][2] = 2.f * (y * z - r * x);
    Rc[2][0] = 2.f * (x * z - r * y);
    Rc[2][1] = 2.f * (y * z + r * x);
    Rc[2][2] = 1.f - 2.f * (x * x + y * y);
}

// True gradient of conic = inv(Sigma + eps I), Sigma = M^T M, M = diag(s) Rg.
__device__ void cov_adjoint_true(const float s_in[3], const float q[4], float sm, const float c6[6],
                                 const float u[6], float ds[3], float dq[4]) {
    float Rc[3][3];
    rot_cols(q[0], q[1], q[2], q[3], Rc);
    float Rg[3][3];  // Rg[i][j] = row i, col j
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Rg[i][j] = Rc[j][i];
    const float sv[3] = {sm * s_in[0], sm * s_in[1], sm * s_in[2]};
    float M[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) M[i][j] = sv[i] * Rg[i][j];
    float Sd[3];
    for (int i = 0; i < 3; i++) Sd[i] = M[0][i] * M[0][i] + M[1][i] * M[1][i] + M[2][i] * M[2][i];
    const float C[3][3] = {{c6[0], c6[1], c6[2]}, {c6[1], c6[3], c6[4]}, {c6[2], c6[4], c6[5]}};
    const float G[3][3] = {{u[0], 0.5f * u[1], 0.5f * u[2]}, {0.5f * u[1], u[3], 0.5f * u[4]}, {0.5f * u[2], 0.5f * u[4], u[5]}};
    float T[3][3], H[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) T[i][j] = G[i][0] * C[0][j] + G[i][1] * C[1][j] + G[i][2] * C[2][j];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) H[i][j] = -(C[i][0] * T[0][j] + C[i][1] * T[1][j] + C[i][2] * T[2][j]);
    const float a0 = fabsf(Sd[0]), a1 = fabsf(Sd[1]), a2 = fabsf(Sd[2]);
    int kmax = 0;
    if (a1 > a0) kmax = 1;
    if (a2 > (kmax == 0 ? a0 : a1)) kmax = 2;
    const float trH = H[0][0] + H[1][1] + H[2][2];
    const float sk = Sd[kmax];
    const float sgn = sk > 0.f ? 1.f : (sk < 0.f ? -1.f : 0.f);
    H[kmax][kmax] += trH * 1e-5f * sgn;
    float dM[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) dM[i][j] = 2.f * (M[i][0] * H[0][j] + M[i][1] * H[1][j] + M[i][2] * H[2][j]);
    float GR[3][3];  // gradient wrt the textbook rotation R_std = Rg^T
    for (int k = 0; k < 3; k++) {
        ds[k] = (dM[k][0] * Rg[k][0] + dM[k][1] * Rg[k][1] + dM[k][2] * Rg[k][2]) * sm;
        for (int j = 0; j < 3; j++) GR[j][k] = sv[k] * dM[k][j];
    }
    const float r = q[0], x = q[1], y = q[2], z = q[3];
    dq[0] = 2.f * (-z * GR[0][1] + y * GR[0][2] + z * GR[1][0] - x * GR[1][2] - y * GR[2][0] + x * GR[2][1]);
    dq[1] = 2.f * (y * GR[0][1] + z * GR[0][2] + y * GR[1][0] - 2.f * x * GR[1][1] - r * GR[1][2] + z * GR[2][0] +
                   r * GR[2][1] - 2.f * x * GR[2][2]);
    dq[2] = 2.f * (-2.f * y * GR[0][0] + x * GR[0][1] + r * GR[0][2] + x * GR[1][0] + z * GR[1][2] - r * GR[2][0] +
                   z * GR[2][1] - 2.f * y * GR[2][2]);
    dq[3] = 2.f * (-2.f * z * GR[0][0] - r * GR[0][1] + x * GR[0][2] + r * GR[1][0] - 2.f * z * GR[1][1] +
                   y * GR[1][2] + x * GR[2][0] + y * GR[2][1]);
}

// Reference-compatible covariance adjoint: backward.cu:50-124 with glm's
// column-major conventions ((A*B)[c][r] = sum_k A[k][r] * B[c][k]).
__device__ void cov_adjoint_ref(const float s_in[3], const float q[4], float sm, const float c6[6],
                                const float u[6], float ds[3], float dq[4]) {
    float Rc[3][3];
    const float r = q[0], x = q[1], y = q[2], z = q[3];
    rot_cols(r, x, y, z, Rc);
    const float sv[3] = {sm * s_in[0], sm * s_in[1], sm * s_in[2]};
    auto mul = [](const float A[3][3], const float B[3][3], float O[3][3]) {
        for (int c = 0; c < 3; c++)
            for (int rr = 0; rr < 3; rr++) O[c][rr] = A[0][rr] * B[c][0] + A[1][rr] * B[c][1] + A[2][rr] * B[c][2];
    };
    float Sm[3][3] = {{sv[0], 0.f, 0.f}, {0.f, sv[1], 0.f}, {0.f, 0.f, sv[2]}};
    float M[3][3], Mt[3][3], Sigma[3][3];
    mul(Sm, Rc, M);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Mt[i][j] = M[j][i];
    mul(Mt, M, Sigma);
    const float C[3][3] = {{c6[0], c6[1], c6[2]}, {c6[1], c6[3], c6[4]}, {c6[2], c6[4], c6[5]}};
    const float G[3][3] = {{u[0], u[1], u[2]}, {u[1], u[3], u[4]}, {u[2], u[4], u[5]}};
    float negC[3][3], T1[3][3], dS[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) negC[i][j] = -C[i][j];
    mul(negC, G, T1);
    mul(T1, C, dS);
    const float dc[6] = {dS[0][0], dS[0][1], dS[0][2], dS[1][1], dS[1][2], dS[2][2]};
    const float a0 = fabsf(Sigma[0][0]), a1 = fabsf(Sigma[1][1]), a2 = fabsf(Sigma[2][2]);
    auto sgn = [](float v) { return v > 0.f ? 1.f : (v < 0.f ? -1.f : 0.f); };
    const float de0 = (a0 >= a1 && a0 >= a2) ? 1e-5f * sgn(Sigma[0][0]) : 0.f;
    const float de1 = (a1 >= a0 && a1 >= a2) ? 1e-5f * sgn(Sigma[1][1]) : 0.f;
    const float de2 = (a2 >= a0 && a2 >= a1) ? 1e-5f * sgn(Sigma[2][2]) : 0.f;
    const float tr = dc[0] + dc[3] + dc[5];
    const float dLdS[3][3] = {{dc[0] + tr * de0, dc[1], dc[2]}, {dc[1], dc[3] + tr * de1, dc[4]}, {dc[2], dc[4], dc[5] + tr * de2}};
    float dM[3][3], Rt[3][3], dSm[3][3];
    mul(dLdS, M, dM);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) dM[i][j] *= 2.f;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Rt[i][j] = Rc[j][i];
    mul(dM, Rt, dSm);
    ds[0] = dSm[0][0] * sm;
    ds[1] = dSm[1][1] * sm;
    ds[2] = dSm[2][2] * sm;
    for (int k = 0; k < 3; k++)
        for (int rr = 0; rr < 3; rr++) dM[k][rr] *= sv[k];
    dq[0] = 2 * z * (dM[1][0] - dM[0][1]) + 2 * y * (dM[0][2] - dM[2][0]) + 2 * x * (dM[2][1] - dM[1][2]);
    dq[1] = 2 * y * (dM[0][1] + dM[1][0]) + 2 * z * (dM[0][2] + dM[2][0]) + 2 * r * (dM[2][1] - dM[1][2]) -
            4 * x * (dM[2][2] + dM[1][1]);
    dq[2] = 2 * x * (dM[0][1] + dM[1][0]) + 2 * r * (dM[0][2] - dM[2][0]) + 2 * z * (dM[2][1] + dM[1][2]) -
            4 * y * (dM[2][2] + dM[0][0]);
    dq[3] = 2 * r * (dM[1][0] - dM[0][1]) + 2 * x * (dM[0][2] + dM[2][0]) + 2 * y * (dM[2][1] + dM[1][2]) -
            4 * z * (dM[1][1] + dM[0][0]);
}

__global__ void __launch_bounds__(256) k_finalize(int P, const float* __restrict__ gacc, const float* __restrict__ scales,
                                                  const float* __restrict__ rots, const float* __restrict__ conics,
                                                  float sm, int ref_compat, float* __restrict__ dmeans,
                                                  float* __restrict__ dscales, float* __restrict__ drots,
                                                  float* __restrict__ dvalues, float* __restrict__ dweights) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const float4* a = reinterpret_cast<const float4*>(gacc + 16 * (int64_t)i);
    const float4 a0 = a[0], a1 = a[1], a2 = a[2];
    dvalues[i] = a0.x;
    dweights[i] = a0.y;
    dmeans[3 * (int64_t)i] = a0.z;
    dmeans[3 * (int64_t)i + 1] = a0.w;
    dmeans[3 * (int64_t)i + 2] = a1.x;
    const float u[6] = {a1.y, a1.z, a1.w, a2.x, a2.y, a2.z};
    const float s[3] = {scales[3 * (int64_t)i], scales[3 * (int64_t)i + 1], scales[3 * (int64_t)i + 2]};
    const float q[4] = {rots[4 * (int64_t)i], rots[4 * (int64_t)i + 1], rots[4 * (int64_t)i + 2], rots[4 * (int64_t)i + 3]};
    float c6[6];
    for (int k = 0; k < 6; k++) c6[k] = conics[6 * (int64_t)i + k];
    float ds[3], dq[4];
    if (ref_compat) cov_adjoint_ref(s, q, sm, c6, u, ds, dq);
    else cov_adjoint_true(s, q, sm, c6, u, ds, dq);
    dscales[3 * (int64_t)i] = ds[0];
    dscales[3 * (int64_t)i + 1] = ds[1];
    dscales[3 * (int64_t)i + 2] = ds[2];
    drots[4 * (int64_t)i] = dq[0];
    drots[4 * (int64_t)i + 1] = dq[1];
    drots[4 * (int64_t)i + 2] = dq[2];
    drots[4 * (int64_t)i + 3] = dq[3];
}

// --------------------------------------------------------------------------------
// Launchers
// --------------------------------------------------------------------------------
static inline unsigned nblk(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

cudaError_t launch_finalize(int64_t P, const float* gacc, const float* scales, const float* rots, const float* conics,
                            float sm, int ref_compat, float* dmeans, float* dscales, float* drots, float* dvalues,
                            float* dweights, cudaStream_t st) {
    if (P <= 0) return cudaSuccess;
    k_finalize<<<nblk(P, 256), 256, 0, st>>>((int)P, gacc, scales, rots, conics, sm, ref_compat, dmeans, dscales,
                                             drots, dvalues, dweights); gvc::note_launch();
    return cudaGetLastError();
}

}  // namespace gvc
