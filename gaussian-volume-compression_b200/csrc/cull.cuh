// cull.cuh -- a box of samples against a Gaussian's power window.
//
// A pair counts only where d^T C d <= 28 (d = x - mu, C the conic; power >= -14,
// forward.cu:166,235).  The corners of a Gaussian's AABB lie well outside that ellipsoid
// (and the AABB is built from the transposed rotation, so it is not even aligned with it):
// of the (16-row unit, Gaussian) pairs whose boxes overlap, a third hold no point of it
// (2M x 16M: 4.2 evaluated rows per contributing pair with the box test alone, 2.7 with
// this one; 2.6 with the exact minimum of the form over the box).
#pragma once
#include "gvc_internal.cuh"

namespace gvc {

// The form is given by the staged power coefficients q = kHalfLog2e * conic (negative,
// off-diagonals doubled: pair.cuh), so 28 becomes kCullPower = 28 * 0.5 log2(e) and the
// signs of n and y^T C y turn around.  t is the rounding allowance per unit of trace.
constexpr float kCullPower = 20.197570572173914f;

struct CullGauss {
    float mx, my, mz;
    float q0, q1, q2, q3, q4, q5;
    float t;  // 1e-6 |q0 + q3 + q5|
};

// With `check`, a form that is not safely positive definite gets t = inf (nothing is
// culled): for conics handed in by a caller.
__device__ __forceinline__ float cull_allowance(float q0, float q1, float q2, float q3, float q4, float q5,
                                                bool check) {
    const float t = -1e-6f * (q0 + q3 + q5);
    if (check) {
        const float a = -q0, b = -0.5f * q1, c = -0.5f * q2, d = -q3, e = -0.5f * q4, f = -q5;
        const float m2 = a * d - b * b;
        const float det = a * (d * f - e * e) - b * (b * f - c * e) + c * (b * e - c * d);
        if (!(a > 0.f && m2 > 0.f && det > 0.f)) return INFINITY;
    }
    return t;
}

// True only if no point of the closed box [lo, hi] has a computed power inside the window.
// y is the point of the box nearest to mu, n = C y; by Cauchy-Schwarz in C every point of
// the box has (n.d)^2 <= (y^T C y)(d^T C d), so with n.d >= s > 0 over the box
// d^T C d >= s^2 / (y^T C y).  Rounding: |c_ij| <= trace, so n is off by at most 3 u tr |y|_1
// per component and s by 6 u tr |y|_1 D (D bounds |d|_1 over the box), y^T C y by
// 6 u tr |y|_1^2, and the evaluated form by 9 u tr |d|_1^2: all within t = 16 u tr.  Any NaN
// or infinity on the way makes a comparison false, and the box is kept.
__device__ __forceinline__ bool outside_window(const CullGauss& g, float4 lo, float4 hi) {
    const float ax = lo.x - g.mx, bx = hi.x - g.mx, ay = lo.y - g.my, by = hi.y - g.my, az = lo.z - g.mz,
                bz = hi.z - g.mz;
    const float yx = fmaxf(ax, fminf(bx, 0.f)), yy = fmaxf(ay, fminf(by, 0.f)), yz = fmaxf(az, fminf(bz, 0.f));
    const float hx = 0.5f * yx, hy = 0.5f * yy, hz = 0.5f * yz;
    // -n, -s and -y^T C y
    const float nx = g.q0 * yx + (g.q1 * hy + g.q2 * hz);
    const float ny = g.q3 * yy + (g.q1 * hx + g.q4 * hz);
    const float nz = g.q5 * yz + (g.q2 * hx + g.q4 * hy);
    const float s = fmaxf(nx * ax, nx * bx) + fmaxf(ny * ay, ny * by) + fmaxf(nz * az, nz * bz);
    const float q = nx * yx + ny * yy + nz * yz;
    const float Y = fabsf(yx) + fabsf(yy) + fabsf(yz);
    const float D = fmaxf(-ax, bx) + fmaxf(-ay, by) + fmaxf(-az, bz);
    const float l = s + g.t * Y * D;
    return l < 0.f && l * l > (kCullPower + g.t * D * D) * (g.t * Y * Y - q);
}

}  // namespace gvc
