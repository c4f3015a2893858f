// Distortion energies of engine/param.py:294-319 with hand-written backward
// passes, for every island of a batch.
//
//   kind 0 (ARAP):      E_f = area * ((q + r - 1)^2 + (q - r - 1)^2)
//                           = area * (|J|^2 - 4 q + 2),  dE/dJ = 2 area (J - R)
//   kind 1 (sym. Dir.): E_f = area * (|J|^2 + |J|^2 / det^2 - 4), inf if det <= 0
//                       dE/dJ = area * (2 J (1 + 1/det^2) - 2 |J|^2 / det^3 cof(J))
// J maps the triangle's isometric frame M = [[x1, x2], [0, y2]] to UV edges,
// J = [u1 - u0, u2 - u0] M^-1, with x1 = |e1|, x2 = e1.e2 / |e1|,
// y2 = |e1 x e2| / |e1|, area = |e1 x e2| / 2 (param.local_frames). The
// gradient with respect to the 3D positions goes through the frame:
// dE/dM = -J^T G M^-T, then x1, x2, y2 and area as functions of e1, e2.
// Triangles with |x1 y2| < 1e-300 contribute nothing (param.py:301-303).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"

using namespace uva;

namespace {

// Value of one triangle's energy, for the forward pass, by reciprocal square
// roots and products: FP64 issue bounds that pass as much as memory (5.1M
// triangles: 124 us with its launches, 139 with rounded roots and divisions), and
// the rounding of an island's sum covers theirs (24 charts, against 80 bits: 2e-16
// to 3e-16 either way). inf * rsqrt(inf) is not a number, so a squared normal that
// overflows counts as an infinite one.
__device__ __forceinline__ double en_value(const double* P, const double* U, int v0, int4 tv, int kind) {
    const double* p0 = P + 3 * (v0 + tv.x);
    const double* p1 = P + 3 * (v0 + tv.y);
    const double* p2 = P + 3 * (v0 + tv.z);
    double e1[3], e2[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) { e1[k] = p1[k] - p0[k]; e2[k] = p2[k] - p0[k]; }
    const double2* UU = reinterpret_cast<const double2*>(U);
    const double2 u0 = UU[v0 + tv.x], u1 = UU[v0 + tv.y], u2 = UU[v0 + tv.z];
    const double n0 = e1[1] * e2[2] - e1[2] * e2[1], n1 = e1[2] * e2[0] - e1[0] * e2[2], n2 = e1[0] * e2[1] - e1[1] * e2[0];
    const double l1sq = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
    const double nsq = n0 * n0 + n1 * n1 + n2 * n2;
    const double inn = rsqrt(nsq), nn = isinf(nsq) ? nsq : nsq * inn, il = rsqrt(l1sq);
    // x1 y2 = |n|; a zero normal or edge makes nn or il not a number, and a
    // first edge beyond 1e154 has no frame
    if (!(nn >= 1e-300 && il <= 1e300 && il > 0.0)) return 0.0;
    const double x2 = (e1[0] * e2[0] + e1[1] * e2[1] + e1[2] * e2[2]) * il;
    const double iy2 = l1sq * il * inn;   // y2 = e2 . (n/|n| x e1/|e1|) = |n| / |e1|
    const double j00 = (u1.x - u0.x) * il, j10 = (u1.y - u0.y) * il;
    const double j01 = ((u2.x - u0.x) - j00 * x2) * iy2, j11 = ((u2.y - u0.y) - j10 * x2) * iy2;
    const double area = 0.5 * nn;
    if (kind == 0) {
        const double qe = 0.5 * (j00 + j11), qh = 0.5 * (j10 - j01), rf = 0.5 * (j00 - j11), rg = 0.5 * (j10 + j01);
        const double q = sqrt(qe * qe + qh * qh), r = sqrt(rf * rf + rg * rg);
        return area * ((q + r - 1.0) * (q + r - 1.0) + (q - r - 1.0) * (q - r - 1.0));
    }
    const double det = j00 * j11 - j01 * j10;
    if (!(det > 0.0)) return area * INFINITY;
    const double fro = j00 * j00 + j01 * j01 + j10 * j10 + j11 * j11;
    return area * (fro + fro / (det * det) - 4.0);
}

// The backward pass: rounded roots and divisions in the frame, J and the
// energy's terms, which reciprocal roots in their place would put 4 % on the
// gradients' error (24 charts, against 80 bits: 1.67e-15 for 1.60e-15 in U,
// 1.94e-15 for 1.85e-15 in P); products of three reciprocals (1 / x1, 1 / y2,
// 1 / |n|) after that, which add nothing to it.
struct EnTri {
    double e1[3], e2[3], n[3];
    double l1, nn, il, x2, y2, area;
    double j00, j01, j10, j11;
    bool live;
};

__device__ __forceinline__ EnTri en_tri(const double* P, const double* U, int v0, int4 tv) {
    EnTri t;
    const double* p0 = P + 3 * (v0 + tv.x);
    const double* p1 = P + 3 * (v0 + tv.y);
    const double* p2 = P + 3 * (v0 + tv.z);
#pragma unroll
    for (int k = 0; k < 3; ++k) { t.e1[k] = p1[k] - p0[k]; t.e2[k] = p2[k] - p0[k]; }
    const double2* UU = reinterpret_cast<const double2*>(U);
    const double2 u0 = UU[v0 + tv.x], u1 = UU[v0 + tv.y], u2 = UU[v0 + tv.z];
    t.n[0] = t.e1[1] * t.e2[2] - t.e1[2] * t.e2[1];
    t.n[1] = t.e1[2] * t.e2[0] - t.e1[0] * t.e2[2];
    t.n[2] = t.e1[0] * t.e2[1] - t.e1[1] * t.e2[0];
    t.l1 = sqrt(t.e1[0] * t.e1[0] + t.e1[1] * t.e1[1] + t.e1[2] * t.e1[2]);   // x1
    t.nn = sqrt(t.n[0] * t.n[0] + t.n[1] * t.n[1] + t.n[2] * t.n[2]);
    t.il = 1.0 / fmax(t.l1, 1e-300);
    t.x2 = (t.e1[0] * t.e2[0] + t.e1[1] * t.e2[1] + t.e1[2] * t.e2[2]) * t.il;
    t.y2 = t.nn * t.il;   // e2 . (n/|n| x e1/|e1|) = |n| / |e1|
    t.area = 0.5 * t.nn;
    t.live = fabs(t.l1 * t.y2) >= 1e-300;
    if (t.live) {
        t.j00 = (u1.x - u0.x) / t.l1; t.j10 = (u1.y - u0.y) / t.l1;
        t.j01 = ((u2.x - u0.x) - t.j00 * t.x2) / t.y2; t.j11 = ((u2.y - u0.y) - t.j10 * t.x2) / t.y2;
    } else {
        t.j00 = t.j01 = t.j10 = t.j11 = 0.0;
    }
    return t;
}

// f(J) and dE/dJ per unit area; returns false for an inverted SD triangle.
__device__ __forceinline__ bool en_f(const EnTri& t, int kind, double& f, double (&G)[4]) {
    if (kind == 0) {
        const double qe = 0.5 * (t.j00 + t.j11), qh = 0.5 * (t.j10 - t.j01);
        const double rf = 0.5 * (t.j00 - t.j11), rg = 0.5 * (t.j10 + t.j01);
        const double q = sqrt(qe * qe + qh * qh), r = sqrt(rf * rf + rg * rg);
        f = (q + r - 1.0) * (q + r - 1.0) + (q - r - 1.0) * (q - r - 1.0);
        double c = 0.0, s = 0.0;
        if (q > 0.0) { c = qe / q; s = qh / q; }
        G[0] = 2.0 * (t.j00 - c); G[1] = 2.0 * (t.j01 + s); G[2] = 2.0 * (t.j10 - s); G[3] = 2.0 * (t.j11 - c);
        return true;
    }
    const double fro = t.j00 * t.j00 + t.j01 * t.j01 + t.j10 * t.j10 + t.j11 * t.j11;
    const double det = t.j00 * t.j11 - t.j01 * t.j10;
    if (!(det > 0.0)) {
        f = INFINITY;
        G[0] = G[1] = G[2] = G[3] = 0.0;
        return false;
    }
    const double id2 = 1.0 / (det * det);
    f = fro + fro * id2 - 4.0;
    const double a = 2.0 * (1.0 + id2), b = -2.0 * fro * id2 / det;
    G[0] = a * t.j00 + b * t.j11;
    G[1] = a * t.j01 - b * t.j10;
    G[2] = a * t.j10 - b * t.j01;
    G[3] = a * t.j11 + b * t.j00;
    return true;
}

// The forward pass gives a warp 32 * items consecutive triangles, lane by
// lane. A lane sums its triangles of the same island (island ids do not
// decrease along the triangles), then the warp folds runs of lanes with equal
// islands, so an island takes one FP64 atomic per run. 5.1M triangles: 166 -> 124 us
// with its launches (a thread's own run of eight strided its loads by 128 bytes).
__global__ void k_energy_fwd(const uva_batch b, const double* P, const double* U, int kind, int items, double* e_isl,
                             double* e_tri) {
    const int lane = threadIdx.x & 31;
    const int64_t f0 = (static_cast<int64_t>(blockIdx.x) * blockDim.x + (threadIdx.x & ~31)) * items + lane;
    int isl = -1;
    double acc = 0.0;
#pragma unroll 2
    for (int k = 0; k < items; ++k) {
        const int64_t f = f0 + 32 * k;
        if (f >= b.t) break;
        const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
        const double e = en_value(P, U, b.vofs[tv.w], tv, kind);
        if (e_tri) e_tri[f] = e;
        if (tv.w != isl) {   // a new island: flush the previous one
            if (isl >= 0 && acc != 0.0) atomicAdd(e_isl + isl, acc);
            isl = tv.w;
            acc = 0.0;
        }
        acc += e;
    }
    // Fold the lanes' last islands over contiguous runs of equal ids. In the
    // last warp of the triangles some lanes end a row of 32 before the others,
    // so one island can hold two runs (A A B B A A): each takes its own atomic.
    const int prev = __shfl_up_sync(0xffffffffu, isl, 1);
    const bool head = lane == 0 || prev != isl;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned above = lane == 31 ? 0u : heads & (0xfffffffeu << lane);
    const int end = above ? __ffs(above) - 1 : 32;   // one past the run's last lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_down_sync(0xffffffffu, acc, o);
        if (lane + o < end) acc += y;
    }
    if (isl >= 0 && head && acc != 0.0) atomicAdd(e_isl + isl, acc);
}

// The global FP64 additions bound the backward pass: L2 takes some 230 G of
// them a second, one operation per 32-byte sector that an instruction covers.
// The corner gradients therefore pass through shared memory, and the lanes of
// an addition take the components of a vertex side by side: one or two
// operations per corner instead of five. 512 islands of 5.1M triangles, UV and
// position gradients, with their launches: 350 -> 243 us. (Summing a block's
// corners by vertex in a shared hash table first took 281 us in place of 192
// without them: its lookups cost more than they save.)
constexpr int kBwdNT = 128;

template <bool POS>
__global__ void __launch_bounds__(kBwdNT) k_energy_bwd(const uva_batch b, const double* P, const double* U, int kind,
                                                       const double* gscale, double* gU, double* gP) {
    __shared__ double su[kBwdNT][6];
    __shared__ double sp[POS ? kBwdNT : 1][9];
    __shared__ int sv[kBwdNT][3];
    const int f = blockIdx.x * kBwdNT + threadIdx.x;
    int v[3] = {-1, -1, -1};
    if (f < b.t) {
        const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
        const int v0 = b.vofs[tv.w];
        const EnTri t = en_tri(P, U, v0, tv);
        double f_, G[4];
        if (t.live && en_f(t, kind, f_, G)) {
            v[0] = v0 + tv.x; v[1] = v0 + tv.y; v[2] = v0 + tv.z;
            const double sc = gscale ? gscale[tv.w] : 1.0;
            const double A = t.area * sc;
            // dE/dJ = A G; J = D M^-1 with D = [du1 du2]: dE/dD = dE/dJ M^-T
            // M^-1 = [[1/x1, -x2/(x1 y2)], [0, 1/y2]]
            const double g00 = A * G[0], g01 = A * G[1], g10 = A * G[2], g11 = A * G[3];
            const double il = t.il, iy2 = 1.0 / t.y2, m01 = -t.x2 * il * iy2;
            const double d1x = g00 * il + g01 * m01, d2x = g01 * iy2;
            const double d1y = g10 * il + g11 * m01, d2y = g11 * iy2;
            double* o = su[threadIdx.x];
            o[0] = -(d1x + d2x); o[1] = -(d1y + d2y);
            o[2] = d1x; o[3] = d1y;
            o[4] = d2x; o[5] = d2y;
            if constexpr (POS) {
                // dE/dM = -J^T (A G) M^-T; M^-T = [[1/x1, 0], [m01, 1/y2]]
                const double jg00 = t.j00 * g00 + t.j10 * g10, jg01 = t.j00 * g01 + t.j10 * g11;
                const double jg11 = t.j01 * g01 + t.j11 * g11;
                const double dM00 = -(jg00 * il + jg01 * m01);   // d/dx1
                const double dM01 = -(jg01 * iy2);                // d/dx2 (row 0, col 1)
                const double dM11 = -(jg11 * iy2);                // d/dy2
                // x1 = |e1|, x2 = e1.e2 / |e1|, y2 = |n| / |e1|, area = |n| / 2;
                // d|n|/de1 = e2 x nh, d|n|/de2 = nh x e1
                const double inn = 1.0 / t.nn, il2 = il * il;
                const double a1 = dM00 * il - il2 * (dM01 * t.x2 + dM11 * t.y2), a2 = dM01 * il;
                const double an = (dM11 * il + 0.5 * sc * f_) * inn;
                const double dn1[3] = {t.e2[1] * t.n[2] - t.e2[2] * t.n[1], t.e2[2] * t.n[0] - t.e2[0] * t.n[2],
                                       t.e2[0] * t.n[1] - t.e2[1] * t.n[0]};
                const double dn2[3] = {t.n[1] * t.e1[2] - t.n[2] * t.e1[1], t.n[2] * t.e1[0] - t.n[0] * t.e1[2],
                                       t.n[0] * t.e1[1] - t.n[1] * t.e1[0]};
                double* w = sp[threadIdx.x];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double ge1 = a1 * t.e1[k] + a2 * t.e2[k] + an * dn1[k], ge2 = a2 * t.e1[k] + an * dn2[k];
                    w[k] = -(ge1 + ge2);
                    w[3 + k] = ge1;
                    w[6 + k] = ge2;
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) sv[threadIdx.x][k] = v[k];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const int e = q * kBwdNT + threadIdx.x, c = e >> 1;
        const int vv = (&sv[0][0])[c];
        if (vv >= 0) atomicAdd(gU + 2 * static_cast<size_t>(vv) + (e & 1), (&su[0][0])[e]);
    }
    if constexpr (POS) {
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int e = q * kBwdNT + threadIdx.x, c = e / 3;
            const int vv = (&sv[0][0])[c];
            if (vv >= 0) atomicAdd(gP + 3 * static_cast<size_t>(vv) + (e - 3 * c), (&sp[0][0])[e]);
        }
    }
}

// ---- p95-stretch refinement: Jacobi-preconditioned descent on the
// symmetric Dirichlet energy, flip-safe and monotone per island.
__global__ void k_descent_dir(int n, const uva_batch b, const int32_t* vert_isl, const double* gU, double* Dd) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const int v0 = b.vofs[vert_isl[v]];
    const double d = b.wdiag[v0 + b.vert_row[v]];   // the diagonal is stored by solver row
    const double m = d > 1e-30 ? 1.0 / d : 0.0;
    Dd[2 * v] = -m * gU[2 * v];
    Dd[2 * v + 1] = -m * gU[2 * v + 1];
}

__device__ __forceinline__ void atomic_min_pos(double* addr, double v) {
    if (!(v >= 0.0)) return;
    atomicMin(reinterpret_cast<unsigned long long*>(addr), static_cast<unsigned long long>(__double_as_longlong(v)));
}

// Minimum over the warp's lanes of the same island (island ids do not
// decrease along the lanes), one atomic per island and warp.
__device__ __forceinline__ void island_min_fold(double* tmax, int isl, double t, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_down_sync(0xffffffffu, t, o);
        const int yi = __shfl_down_sync(0xffffffffu, isl, o);
        if (lane + o < 32 && yi == isl && y < t) t = y;
    }
    const int prev = __shfl_up_sync(0xffffffffu, isl, 1);
    if (isl >= 0 && (lane == 0 || prev != isl)) atomic_min_pos(tmax + isl, t);
}

// Per-island flip-safe bound (param.py:259-291 per island).
__global__ void k_island_max_step(const uva_batch b, const double* U, const double* Dd, double* tmax) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int isl = -1;          // idle lanes join the warp's fold with no island
    double t = 1e30;
    if (f < b.t) {
        const int4 tv = reinterpret_cast<const int4*>(b.tri4)[f];
        isl = tv.w;
        const int v0 = b.vofs[tv.w];
        const double2* UU = reinterpret_cast<const double2*>(U);
        const double2* DD = reinterpret_cast<const double2*>(Dd);
        const double2 u0 = UU[v0 + tv.x], u1 = UU[v0 + tv.y], u2 = UU[v0 + tv.z];
        const double2 d0 = DD[v0 + tv.x], d1 = DD[v0 + tv.y], d2 = DD[v0 + tv.z];
        const double ux1 = u1.x - u0.x, uy1 = u1.y - u0.y, ux2 = u2.x - u0.x, uy2 = u2.y - u0.y;
        const double dx1 = d1.x - d0.x, dy1 = d1.y - d0.y, dx2 = d2.x - d0.x, dy2 = d2.y - d0.y;
        const double C = ux1 * uy2 - ux2 * uy1;
        const double B = ux1 * dy2 + dx1 * uy2 - ux2 * dy1 - dx2 * uy1;
        const double A = dx1 * dy2 - dx2 * dy1;
        if (C > 0.0) {
            if (A == 0.0 || fabs(A) < 1e-30 * fmax(fabs(B), 1e-300)) {
                if (B < 0.0) t = -C / B;
            } else {
                const double disc = B * B - 4.0 * A * C;
                if (disc >= 0.0) {
                    const double sq = sqrt(disc);
                    const double r1 = (-B - sq) / (2.0 * A), r2 = (-B + sq) / (2.0 * A);
                    if (r1 > 0.0 && r1 < t) t = r1;
                    if (r2 > 0.0 && r2 < t) t = r2;
                }
            }
        }
    }
    island_min_fold(tmax, isl, t, lane);
}

__global__ void k_trial(int n, const uva_batch b, const double* U, const double* Dd, const double* alpha,
                        const int32_t* vert_isl, double* Ut) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const double a = alpha[vert_isl[v]];
    Ut[2 * v] = U[2 * v] + a * Dd[2 * v];
    Ut[2 * v + 1] = U[2 * v + 1] + a * Dd[2 * v + 1];
}

// Accept per island when the trial energy decreased (Armijo-free monotone
// test), else halve its step; islands that accepted stop shrinking.
__global__ void k_accept(int nc, const double* e_old, const double* e_new, double* alpha, int32_t* accepted) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc || accepted[i]) return;
    if (e_new[i] < e_old[i]) accepted[i] = 1;
    else alpha[i] *= 0.5;
}

__global__ void k_commit(int n, const int32_t* vert_isl, const int32_t* accepted, const double* Ut, double* U) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    if (accepted[vert_isl[v]]) { U[2 * v] = Ut[2 * v]; U[2 * v + 1] = Ut[2 * v + 1]; }
}

__global__ void k_init_alpha(int nc, const double* tmax, double* alpha, int32_t* accepted, double cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nc) return;
    alpha[i] = fmin(cap, 0.9 * tmax[i]);
    accepted[i] = 0;
}

__global__ void k_fill_d(double* p, int n, double v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

__global__ void k_vert_isl2(const int32_t* vofs, int nc, int32_t* vert_isl) {
    const int isl = blockIdx.x;
    if (isl >= nc) return;
    for (int v = vofs[isl] + threadIdx.x; v < vofs[isl + 1]; v += blockDim.x) vert_isl[v] = isl;
}

inline int nb(int x) { return std::max(1, (x + 255) / 256); }

}  // namespace

extern "C" int uva_energy_fwd(const uva_batch* b, const double* P, const double* U, int32_t kind, double* e_isl,
                              double* e_tri, void* stream) {
    if (!b || !P || !U || !e_isl || (kind != 0 && kind != 1)) { uva_set_error("uva_energy_fwd: bad arguments"); return UVA_E_ARG; }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaMemsetAsync(e_isl, 0, sizeof(double) * static_cast<size_t>(std::max(b->nc, 1)), s);
    // up to 8 triangles per thread once there are more than the GPU holds at a time
    const int items = std::min(8, std::max(1, b->t / (148 * 1024)));
    if (b->t > 0) k_energy_fwd<<<nb((b->t + items - 1) / items), 256, 0, s>>>(*b, P, U, kind, items, e_isl, e_tri);
    UVA_CHECK_LAUNCH("uva_energy_fwd");
    return UVA_OK;
}

extern "C" int uva_energy_bwd(const uva_batch* b, const double* P, const double* U, int32_t kind, const double* gscale,
                              double* gU, double* gP, void* stream) {
    if (!b || !P || !U || !gU || (kind != 0 && kind != 1)) { uva_set_error("uva_energy_bwd: bad arguments"); return UVA_E_ARG; }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaMemsetAsync(gU, 0, sizeof(double) * 2 * static_cast<size_t>(b->n), s);
    if (gP) cudaMemsetAsync(gP, 0, sizeof(double) * 3 * static_cast<size_t>(b->n), s);
    const int grid = (b->t + kBwdNT - 1) / kBwdNT;
    if (b->t > 0 && gP) k_energy_bwd<true><<<grid, kBwdNT, 0, s>>>(*b, P, U, kind, gscale, gU, gP);
    if (b->t > 0 && !gP) k_energy_bwd<false><<<grid, kBwdNT, 0, s>>>(*b, P, U, kind, gscale, gU, gP);
    UVA_CHECK_LAUNCH("uva_energy_bwd");
    return UVA_OK;
}

// `steps` iterations of descent on the symmetric Dirichlet energy for every
// island (after uva_batch_setup): direction -D^-1 grad (D: cotangent
// Laplacian diagonal), step = min(cap, 0.9 * flip-safe bound), halved up to
// `halvings` times until the island's energy decreases. U (b->U) is updated
// in place; e_isl (nc) receives the final energies. scratch: 8n + 7nc
// doubles + n ints.
extern "C" int uva_sd_refine(uva_batch* b, int32_t steps, int32_t halvings, double cap, double* e_isl, void* scratch,
                             void* stream) {
    if (!b || !e_isl || !scratch || steps < 0 || halvings < 0) { uva_set_error("uva_sd_refine: bad arguments"); return UVA_E_ARG; }
    if (b->nc == 0 || b->t == 0) return UVA_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int n = b->n, nc = b->nc;
    double* gU = static_cast<double*>(scratch);
    double* Dd = gU + 2 * static_cast<size_t>(n);
    double* Ut = Dd + 2 * static_cast<size_t>(n);
    double* tmax = Ut + 2 * static_cast<size_t>(n);
    double* alpha = tmax + nc;
    double* e_new = alpha + nc;
    int32_t* accepted = reinterpret_cast<int32_t*>(e_new + nc);
    int32_t* vert_isl = accepted + nc + (nc & 1);
    k_vert_isl2<<<nc, 256, 0, s>>>(b->vofs, nc, vert_isl);
    for (int it = 0; it < steps; ++it) {
        uva_energy_fwd(b, b->P, b->U, 1, e_isl, nullptr, s);
        uva_energy_bwd(b, b->P, b->U, 1, nullptr, gU, nullptr, s);
        k_descent_dir<<<nb(n), 256, 0, s>>>(n, *b, vert_isl, gU, Dd);
        k_fill_d<<<nb(nc), 256, 0, s>>>(tmax, nc, 1e30);
        k_island_max_step<<<nb(b->t), 256, 0, s>>>(*b, b->U, Dd, tmax);
        k_init_alpha<<<nb(nc), 256, 0, s>>>(nc, tmax, alpha, accepted, cap);
        for (int h = 0; h <= halvings; ++h) {
            k_trial<<<nb(n), 256, 0, s>>>(n, *b, b->U, Dd, alpha, vert_isl, Ut);
            uva_energy_fwd(b, b->P, Ut, 1, e_new, nullptr, s);
            k_accept<<<nb(nc), 256, 0, s>>>(nc, e_isl, e_new, alpha, accepted);
        }
        k_commit<<<nb(n), 256, 0, s>>>(n, vert_isl, accepted, Ut, b->U);
    }
    UVA_CHECK_LAUNCH("uva_sd_refine");
    return uva_energy_fwd(b, b->P, b->U, 1, e_isl, nullptr, s);
}
