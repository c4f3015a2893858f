// Per-triangle steps of the island solvers, shared by the conjugate-gradient
// path (solve.cu) and the direct path (direct.cu): packed slots, the ARAP
// local step, the flip-safe step bound and the fold test.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace uva {

// Packed slot column: island row in the low 24 bits, twice the LSCM
// boundary coupling (a small integer) in the high 8 bits.
__device__ __forceinline__ int slot_row(int x) { return x & 0xFFFFFF; }
__device__ __forceinline__ float slot_c2(int x) { return static_cast<float>(x >> 24); }

__device__ __forceinline__ long long global_ns() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned sm_id() {
    unsigned r;
    asm("mov.u32 %0, %%smid;" : "=r"(r));
    return r;
}

// ---- local step (per triangle): closest rotation + corner RHS terms.
// BATCH: engine/gpu.py:165-182. PARAM: engine/param.py:206-233, 457-474.
__device__ __forceinline__ void local_terms(const uva_batch& b, int v0, int f, const double2* U, bool batch,
                                            double& energy, int& flip) {
    const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
    const double4 fr = reinterpret_cast<const double4*>(b.frame)[f];
    const double4 wt = reinterpret_cast<const double4*>(b.wtri)[f];
    const double2 u0 = U[v0 + tv.x], u1 = U[v0 + tv.y], u2 = U[v0 + tv.z];
    const double x1 = fr.x, x2 = fr.y, y2 = fr.z;
    const double du1x = u1.x - u0.x, du1y = u1.y - u0.y, du2x = u2.x - u0.x, du2y = u2.y - u0.y;
    double c = 1.0, s = 0.0;
    const double sar = du1x * du2y - du2x * du1y;
    flip = sar <= 0.0 ? 1 : 0;
    energy = 0.0;
    if (batch) {
        if (wt.w != 0.0) {
            const double j00 = du1x / x1, j10 = du1y / x1;
            const double j01 = (du2x - j00 * x2) / y2, j11 = (du2y - j10 * x2) / y2;
            const double ca = j00 + j11, cb = j10 - j01;
            if (isfinite(ca) && isfinite(cb)) {
                const double h = hypot(ca, cb);
                if (h > 0.0) { c = ca / h; s = cb / h; }
            } else if (!isnan(ca) && !isnan(cb)) {
                const double th = atan2(cb, ca);
                c = cos(th); s = sin(th);
            }
        }
        const double sc = static_cast<double>(b.tscale[f]);
        c *= sc; s *= sc;
    } else if (fabs(x1 * y2) >= 1e-300) {
        const double j00 = du1x / x1, j10 = du1y / x1;
        const double j01 = (du2x - j00 * x2) / y2, j11 = (du2y - j10 * x2) / y2;
        double ca = j00 + j11, cb = j10 - j01;
        double h = sqrt(ca * ca + cb * cb);
        if (h < 1e-300) { ca = 1.0; cb = 0.0; h = 1.0; }
        c = ca / h; s = cb / h;
        const double qe = 0.5 * (j00 + j11), qh = 0.5 * (j10 - j01);
        const double rf = 0.5 * (j00 - j11), rg = 0.5 * (j10 + j01);
        const double q = sqrt(qe * qe + qh * qh), r = sqrt(rf * rf + rg * rg);
        energy = fr.w * ((q + r - 1.0) * (q + r - 1.0) + (q - r - 1.0) * (q - r - 1.0));
    }
    // edge k runs corner k+1 -> k+2; frame corners (0,0), (x1,0), (x2,y2)
    const double cxs[3] = {0.0, x1, x2}, cys[3] = {0.0, 0.0, y2};
    const double wk[3] = {wt.x, wt.y, wt.z};
    double vx[3], vy[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int i = (k + 1) % 3, j = (k + 2) % 3;
        const double dx = cxs[i] - cxs[j], dy = cys[i] - cys[j];
        vx[k] = wk[k] * (c * dx - s * dy);
        vy[k] = wk[k] * (s * dx + c * dy);
    }
    double2* rc = reinterpret_cast<double2*>(b.rc);
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
        const int kp = (cc + 2) % 3, km = (cc + 1) % 3;
        rc[3 * f + cc] = make_double2(vx[kp] - vx[km], vy[kp] - vy[km]);
    }
}

// Flip-safe step bound of one triangle (smallest positive root of the
// signed-area quadratic). BATCH: gpu.py:204-227, PARAM: param.py:259-291.
__device__ __forceinline__ double step_bound(const uva_batch& b, int v0, int f, const double2* U, const double2* X,
                                             bool batch) {
    const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
    const double2 u0 = U[v0 + tv.x], u1 = U[v0 + tv.y], u2 = U[v0 + tv.z];
    const int* vr = b.vert_row + v0;
    const double2 x0 = X[v0 + vr[tv.x]], x1 = X[v0 + vr[tv.y]], x2 = X[v0 + vr[tv.z]];
    const double2 d0 = make_double2(x0.x - u0.x, x0.y - u0.y), d1 = make_double2(x1.x - u1.x, x1.y - u1.y),
                  d2 = make_double2(x2.x - u2.x, x2.y - u2.y);
    const double ux1 = u1.x - u0.x, uy1 = u1.y - u0.y, ux2 = u2.x - u0.x, uy2 = u2.y - u0.y;
    const double dx1 = d1.x - d0.x, dy1 = d1.y - d0.y, dx2 = d2.x - d0.x, dy2 = d2.y - d0.y;
    const double C = ux1 * uy2 - ux2 * uy1;
    const double B = ux1 * dy2 + dx1 * uy2 - ux2 * dy1 - dx2 * uy1;
    const double A = dx1 * dy2 - dx2 * dy1;
    const double big = 1e30;
    if (!(C > 0.0)) return big;
    if (batch) {
        double t = big;
        if (fabs(A) < 1e-30) {
            if (B < 0.0) t = -C / B;
        } else {
            const double disc = B * B - 4.0 * A * C;
            if (disc >= 0.0) {
                const double sq = sqrt(disc);
                const double r1 = (-B - sq) / (2.0 * A), r2 = (-B + sq) / (2.0 * A);
                if (r1 > 0.0) t = fmin(t, r1);
                if (r2 > 0.0) t = fmin(t, r2);
            }
        }
        return isnan(t) ? big : t;
    }
    if (A == 0.0 || fabs(A) < 1e-30 * fmax(fabs(B), 1e-300)) return B < 0.0 ? -C / B : big;
    const double disc = B * B - 4.0 * A * C;
    if (disc < 0.0) return big;
    const double sq = sqrt(disc);
    const double r1 = (-B - sq) / (2.0 * A), r2 = (-B + sq) / (2.0 * A);
    double t = big;
    if (r1 > 0.0 && r1 < t) t = r1;
    if (r2 > 0.0 && r2 < t) t = r2;
    return t;
}

// 1 if triangle f is folded at U: negative signed UV area with a valid frame
// (engine/hier.py:549)
__device__ __forceinline__ int folded_tri(const uva_batch& b, int v0, int f, const double2* U) {
    if (reinterpret_cast<const double4*>(b.wtri)[f].w == 0.0) return 0;
    const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
    const double2 a = U[v0 + tv.x], c1 = U[v0 + tv.y], c2 = U[v0 + tv.z];
    return ((c1.x - a.x) * (c2.y - a.y) - (c2.x - a.x) * (c1.y - a.y)) < 0.0 ? 1 : 0;
}

}  // namespace uva
