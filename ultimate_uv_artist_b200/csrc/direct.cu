// Direct island solver: sparse LDL^T of every island's LSCM / ARAP operator
// in FP64, one CTA per island, in place of the conjugate gradients of
// solve.cu for islands of up to kDirectMaxN vertices.
//
// Why: in breadth-first order the matrix of a chart has a narrow skyline (about
// the square root of n columns on a regular grid, up to twice that on irregular
// triangulations). An 8,061-vertex disk has 3,779 blocks of 16 x 16 in its
// factor: 27 million multiply-adds and 7.7 MB, where the FP32 two-level CG needs
// 1,416 iterations of LSCM (and some 40 per ARAP step) whose cost is barriers and
// L2 round trips. The factor is exact to FP64 round-off, so one solve per global
// step meets the tolerance that the FP64 residual check asks for; ARAP factors
// once per call and only substitutes in its iterations.
//
//   k_band    (set-up) Cuthill-McKee order of an island from its far boundary
//             vertex: level-synchronous breadth-first search, levels ordered
//             by (first parent, row). Position of every solver row, first
//             block column of every block row, number of blocks.
//   k_direct  block LDL^H, left-looking by block columns of 16: S_IK = A_IK -
//             sum_M G_IM L_KM^H (G = L D kept in a ring of 16 x 16 blocks),
//             D_K inverted by the CTA, an element per thread, 2 x 2 pivots),
//             L_IK = S_IK D_K^-1. The products run on the FP64 tensor
//             instruction (m8n8k4). LSCM factors the
//             complex Hermitian n x n form of its (u, v) system, ARAP the
//             real one.
//   solves    forward and backward substitution with one barrier per block:
//             a group of 16 threads owns every sixteenth block row and keeps
//             its right-hand side in registers; the factor streams through a
//             ring of shared-memory stages (cp.async.bulk, mbarriers).
//
// What bounds it: the largest island, one CTA from end to end of the launch.
// Its factor is a chain of block columns with some 16 dependent L2 round trips
// (about 800 cycles each) a column: 8.1 ms of the 11.5 ms LSCM launch of 2,000
// islands (8,061 vertices the largest). Its substitutions are a chain of 504
// steps of 960 cycles, three fifths of them shared-memory loads and the FP64
// sums, the rest the hand-over of the block and its barrier: 11.7 ms of the
// 29.1 ms ARAP launch of 20 iterations; local step, right-hand side, residual
// and line search take 11.4, the factor some 4. With CG: 40.0 ms LSCM, 39.6 ARAP.
// Tried and slower: fragments of L prefetched in registers from global memory
// (45 ms ARAP), block x vector on the tensor instruction (36), the same layout
// with scalar sums and two feeding warps (29.9 ARAP, 29.9 then without them, but
// 12.7 LSCM).
//
// Blocks are stored column by column with an XOR swizzle (element (r, c) at
// 16 c + (r ^ c)): a forward step reads a column over 16 lanes, a backward
// step a row, both without bank conflicts and in full sectors.
//
// An island keeps the CG path (solve.cu, launched after this kernel) when it
// is above kDirectMaxN vertices, not connected, wider than kMaxW blocks, when
// its factor does not fit the CTA's scratch, or when a pivot or the residual
// check says that its operator is singular; all islands of a launch do when
// k_choose expects CG to be faster.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "direct.cuh"
#include "island.cuh"
#include "wait.cuh"

using namespace uva;

namespace {

constexpr int kNB = 16;                  // block edge
constexpr int kBE = kNB * kNB;           // elements of a block (one plane)
constexpr int kMaxW = 15;                // blocks left of the diagonal: the groups of a CTA less one
constexpr int kCT = 256;                 // compute threads: 16 groups of 16
constexpr int kCW = kCT / 32;
constexpr int kNT = kCT + 32;            // and one warp that feeds the solve's ring
constexpr int kNW = kNT / 32;
constexpr int kPitch = 20;               // pitch of a staged column: conflict-free m8n8k4 fragments
constexpr int kSB = kNB * kPitch;        // doubles of a staged block (one plane)
constexpr int kMaxBlk = kDirectMaxN / kNB;
constexpr int kRing = 94 * 1024;         // bytes of staged factor blocks (2 CTAs per SM)
constexpr int kMaxStages = 8;
constexpr int kLevelCap = 1024;          // vertices of one breadth-first level

// ------------------------------------------------------------------ order
// Cuthill-McKee order of one island per CTA. key[i]: position of row i's
// first placed neighbour (its lowest position, so also its skyline).
__global__ void __launch_bounds__(kNT) k_band(uva_batch b) {
    extern __shared__ int key[];
    __shared__ int cur[kLevelCap], comp[kLevelCap];
    __shared__ int nnew, total, maxw;
    const int isl = b.order[blockIdx.x], tid = threadIdx.x;
    const int v0 = b.vofs[isl], n = b.vofs[isl + 1] - v0, s0 = b.sofs[isl];
    int32_t* pos = b.band + v0;
    int32_t* first = band_first(b, v0, isl);
    int32_t* info = band_info(b, isl);
    if (n < 2 || n > kDirectMaxN) {
        if (tid == 0) info[0] = 0;
        return;
    }
    const int nblk = (n + kNB - 1) / kNB;
    for (int i = tid; i < n; i += kNT) key[i] = 0x7fffffff;
    for (int k = tid; k < nblk; k += kNT) first[k] = k;
    const int p0 = b.pins[3 * isl + 1];
    const int start = p0 >= 0 ? b.vert_row[v0 + p0] : 0;
    if (tid == 0) { cur[0] = start; nnew = 0; total = 0; maxw = 0; }
    __syncthreads();
    if (tid == 0) { key[start] = -1; pos[start] = 0; first[0] = 0; }
    __syncthreads();
    const int2* cw = reinterpret_cast<const int2*>(b.slot_cw);
    int base = 0, m = 1;     // the current level: positions [base, base + m), rows cur[0..m)
    while (m > 0) {
        for (int q = tid; q < 8 * m; q += kNT) {   // eight lanes per row
            const int i = cur[q >> 3], p = base + (q >> 3);
            const int s = s0 + (i >> 5);
            const int a = b.slice_ptr[s], w = (b.slice_ptr[s + 1] - a) >> 5;
            for (int k = q & 7; k < w; k += 8) {
                const int c = slot_row(cw[a + 32 * k + (i & 31)].x);
                if (c == i) continue;                  // padding and self loops
                if (atomicMin(&key[c], p) == 0x7fffffff) {
                    const int at = atomicAdd(&nnew, 1);
                    if (at < kLevelCap) comp[at] = c;
                }
            }
        }
        __syncthreads();
        const int m2 = nnew;
        __syncthreads();
        if (tid == 0) nnew = 0;
        if (m2 > kLevelCap) {       // uniform: every thread read the same count
            if (tid == 0) info[0] = 0;
            return;
        }
        // order of the next level: (first parent, row), both below 2^14
        for (int j = tid; j < m2; j += kNT) { const int c = comp[j]; comp[j] = (key[c] << 14) | c; }
        __syncthreads();
        for (int j = tid; j < m2; j += kNT) {
            const int mine = comp[j];
            int rank = 0;
            for (int k = 0; k < m2; ++k) rank += comp[k] < mine ? 1 : 0;
            const int row = mine & 16383, p = base + m + rank;
            cur[rank] = row;
            pos[row] = p;
            if (p % kNB == 0) first[p / kNB] = (mine >> 14) / kNB;   // keys grow with the position
        }
        __syncthreads();
        base += m;
        m = m2;
    }
    // blocks of the factor, widest row
    int t = 0, w = 0;
    for (int k = tid; k < nblk; k += kNT) {
        const int d = k - first[k];
        t += d + 1;
        w = max(w, d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
    }
    if ((tid & 31) == 0) { atomicAdd(&total, t); atomicMax(&maxw, w); }
    __syncthreads();
    if (tid == 0) {
        info[0] = base == n && maxw <= kMaxW ? 1 : 0;   // base < n: not connected
        info[1] = total;
        info[2] = maxw;
        info[3] = 0;
    }
}

// ------------------------------------------------------------------ small pieces
__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCT) : "memory"); }
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
constexpr int kWaitPolls = 1 << 18;      // about a second without the phase
__device__ __forceinline__ bool mbar_wait(int& bad, unsigned bar, unsigned parity) {
    return bounded_wait(
        [=]() {
            unsigned ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(bar), "r"(parity)
                : "memory");
            return ok != 0;
        },
        kWaitPolls, bad);
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ int sw(int r, int c) { return c * kNB + (r ^ c); }   // element (r, c) of a block

// Sums of up to 4 values over the CTA, the same bits on every thread.
struct Red {
    double* buf;   // 2 x 4 x kNW
    int phase;
};
template <int K>
__device__ __forceinline__ void cta_sum(Red& rd, double (&v)[K]) {
    static_assert(K <= 4, "four values at most");
    double* q = rd.buf + rd.phase * 4 * kNW;
    rd.phase ^= 1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) q[k * kNW + (threadIdx.x >> 5)] = x;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kNW; ++w) s += q[k * kNW + w];
        v[k] = s;
    }
}
__device__ __forceinline__ double cta_min(Red& rd, double v) {
    double* q = rd.buf + rd.phase * 4 * kNW;
    rd.phase ^= 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) q[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = q[0];
#pragma unroll
    for (int w = 1; w < kNW; ++w) s = fmin(s, q[w]);
    return s;
}

enum Op { OP_ARAP = 0, OP_LSCM = 1 };

// One island of the CTA.
struct Isl {
    int id, v0, n, f0, nt, s0, nblk;
    int pin, p0, p1;       // solver rows of the ARAP pin and of the LSCM pins
    double wpin;
    const int32_t* pos;    // band position of each solver row
    double* L;             // factor blocks, block rows one after the other
    double* G;             // ring of 16 x 16 blocks: G = L D of the active rows
    double2* rb;           // right-hand side / solution by band position
    double2 *y, *lu;       // A x of the last solution and of U, by solver row (ARAP)
    int stages;            // stages of the ring
    int q, ph;             // next stage and its phase (each thread its own: compute and feeding warps)
};

struct Shared {
    unsigned short first[kMaxBlk + 1];
    int off[kMaxBlk + 1];                     // first block of each block row
    double red[2 * 4 * kNW];
    double dsm[2 * kNB * (kNB + 1)];          // S_KK (two planes, padded rows)
    double dinv[2 * kSB];                     // D_K^-1 (staged layout)
    double2 prow[2][2][kNB], pcol[2][2][kNB]; // pivot rows and columns of the inversion
    double diag[kNB];                         // diagonal of A_KK
    double2 xk[2][kNB];                       // the block being substituted
    unsigned long long full[kMaxStages], empty[kMaxStages];
    int bad, rank, scan[kNW];
    int dead_q, dead_ph, dead_stages;         // the ring as the feeding warp left it when a wait ran out
};

// (A x)_i in FP64 from the FP32 slot weights, in difference form.
template <Op OP>
__device__ __forceinline__ double2 apply(const uva_batch& b, const Isl& I, int i, const double2* x) {
    const int s = I.s0 + (i >> 5);
    const int a = __ldg(b.slice_ptr + s), w = (__ldg(b.slice_ptr + s + 1) - a) >> 5;
    const int2* cw = reinterpret_cast<const int2*>(b.slot_cw) + a + (i & 31);
    const double2 xi = x[i];
    double ax = 0.0, ay = 0.0;
    for (int k = 0; k < w; k += 4) {   // slice widths are multiples of 4
        int2 q[4];
        double2 xj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) q[u] = __ldg(cw + 32 * (k + u));
#pragma unroll
        for (int u = 0; u < 4; ++u) xj[u] = x[slot_row(q[u].x)];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double wt = static_cast<double>(__int_as_float(q[u].y));
            ax += wt * (xi.x - xj[u].x);
            ay += wt * (xi.y - xj[u].y);
            if (OP == OP_LSCM) {
                const double c = 0.5 * static_cast<double>(slot_c2(q[u].x));
                ax += c * xj[u].y;
                ay -= c * xj[u].x;
            }
        }
    }
    if (OP == OP_ARAP && i == I.pin) { ax += I.wpin * xi.x; ay += I.wpin * xi.y; }
    return make_double2(ax, ay);
}

// ------------------------------------------------------------------ factor
// acc (8 rows x 16 columns: two m8n8 tiles, CP: real then imaginary) +-=
// A[8 mt ..][.] conj(B)^T for one block pair, B in the staged layout.
template <bool CP, bool SUB>
__device__ __forceinline__ void block_mma(double (&acc)[CP ? 4 : 2][2], const double (&a)[4], const double (&ai)[CP ? 4 : 1],
                                          const double* B, int lane) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const int k = (lane & 3) + 4 * ks;
        const double ar = SUB ? -a[ks] : a[ks];
        double aim = 0.0;
        if constexpr (CP) aim = SUB ? -ai[ks] : ai[ks];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int e = k * kPitch + (lane >> 2) + 8 * nt;
            const double br = B[e];
            dmma(acc[nt], ar, br);
            if constexpr (CP) {
                const double bi = B[kSB + e];
                dmma(acc[nt], aim, bi);
                dmma(acc[2 + nt], aim, br);
                dmma(acc[2 + nt], -ar, bi);
            }
        }
    }
}
template <bool CP>
__device__ __forceinline__ void load_a(const double* A, int mt, int lane, double (&a)[4], double (&ai)[CP ? 4 : 1]) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        const int e = sw((lane >> 2) + 8 * mt, (lane & 3) + 4 * ks);
        a[ks] = A[e];
        if constexpr (CP) ai[ks] = A[kBE + e];
    }
}

// Scatter the island's matrix into its factor blocks (lower part), zeros
// elsewhere; LSCM: pinned rows and columns become the identity.
template <Op OP>
__device__ void assemble(const uva_batch& b, const Isl& I, const Shared& S) {
    constexpr bool CP = OP == OP_LSCM;
    constexpr int BB = kBE * (CP ? 2 : 1);
    const int nd2 = S.off[I.nblk] * (BB / 2);
    double2* L2 = reinterpret_cast<double2*>(I.L);
    for (int k = threadIdx.x; k < nd2; k += kNT) L2[k] = make_double2(0.0, 0.0);
    __syncthreads();
    const int2* cw = reinterpret_cast<const int2*>(b.slot_cw);
    for (int i = threadIdx.x; i < I.nblk * kNB; i += kNT) {
        if (i >= I.n) {   // padding rows of the last block: the identity
            const int K = i / kNB;
            I.L[static_cast<size_t>(S.off[K + 1] - 1) * BB + sw(i % kNB, i % kNB)] = 1.0;
            continue;
        }
        const int p = I.pos[i], K = p / kNB, r = p % kNB;
        const bool pinned = OP == OP_LSCM && (i == I.p0 || i == I.p1);
        double d = 0.0;
        if (!pinned) {
            const int s = I.s0 + (i >> 5);
            const int a = __ldg(b.slice_ptr + s), w = (__ldg(b.slice_ptr + s + 1) - a) >> 5;
            for (int k = 0; k < w; ++k) {
                const int2 q = __ldg(cw + a + 32 * k + (i & 31));
                const int c = slot_row(q.x);
                if (c == i) continue;
                const double wt = static_cast<double>(__int_as_float(q.y));
                d += wt;
                if (OP == OP_LSCM && (c == I.p0 || c == I.p1)) continue;
                const int pc = I.pos[c];
                if (pc > p) continue;
                double* B = I.L + static_cast<size_t>(S.off[K] + pc / kNB - S.first[K]) * BB;
                const int e = sw(r, pc % kNB);
                B[e] = -wt;
                if (CP) B[kBE + e] = -0.5 * static_cast<double>(slot_c2(q.x));
                if (pc / kNB == K) {   // the diagonal block is kept whole (Hermitian)
                    const int et = sw(pc % kNB, r);
                    B[et] = -wt;
                    if (CP) B[kBE + et] = 0.5 * static_cast<double>(slot_c2(q.x));
                }
            }
            if (OP == OP_ARAP && i == I.pin) d += I.wpin;
        } else {
            d = 1.0;
        }
        I.L[static_cast<size_t>(S.off[K + 1] - 1) * BB + sw(r, r)] = d;
    }
    __syncthreads();
}

// D^-1 of the 16 x 16 (Hermitian) positive definite S_KK in S.dsm, one element
// per thread: Gauss-Jordan with 2 x 2 pivots, whose rows and columns pass
// through shared memory (one barrier per pivot pair). Into S.dinv and Dk. Sets
// S.bad when a pivot is not above 1e-13 of A's diagonal.
template <bool CP>
__device__ __forceinline__ void invert_block(Shared& S, double* Dk) {
    const int r = threadIdx.x >> 4, c = threadIdx.x & 15;
    double2 w = make_double2(S.dsm[r * (kNB + 1) + c], CP ? S.dsm[kNB * (kNB + 1) + r * (kNB + 1) + c] : 0.0);
    bool bad = false;
    auto mul = [](double2 x, double2 y) {
        return CP ? make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x) : make_double2(x.x * y.x, 0.0);
    };
    auto add = [](double2 x, double2 y) { return make_double2(x.x + y.x, CP ? x.y + y.y : 0.0); };
#pragma unroll
    for (int k = 0; k < kNB; k += 2) {
        double2(*row)[kNB] = S.prow[(k >> 1) & 1];
        double2(*col)[kNB] = S.pcol[(k >> 1) & 1];
        if ((r >> 1) == (k >> 1)) row[r & 1][c] = w;
        if ((c >> 1) == (k >> 1)) col[c & 1][r] = w;
        compute_sync();
        const double a = row[0][k].x, d = row[1][k + 1].x;
        const double2 b = row[0][k + 1];
        const double det = a * d - (CP ? b.x * b.x + b.y * b.y : b.x * b.x);
        bad |= !(a > 1e-13 * S.diag[k]) || !(det > 1e-13 * S.diag[k + 1] * a);
        const double id = 1.0 / det;
        const double2 p00 = make_double2(d * id, 0.0), p11 = make_double2(a * id, 0.0);
        const double2 p01 = make_double2(-b.x * id, -b.y * id), p10 = make_double2(p01.x, -p01.y);
        // the column's entry of the scaled pivot rows (its own columns: P^-1)
        const bool pc = (c >> 1) == (k >> 1);
        const double2 g0 = row[0][c], g1 = row[1][c];
        double2 t0 = add(mul(p00, g0), mul(p01, g1)), t1 = add(mul(p10, g0), mul(p11, g1));
        if (pc) { t0 = c & 1 ? p01 : p00; t1 = c & 1 ? p11 : p10; }
        if ((r >> 1) == (k >> 1)) {
            w = r & 1 ? t1 : t0;
        } else {
            const double2 u = add(mul(col[0][r], t0), mul(col[1][r], t1));
            w = make_double2((pc ? 0.0 : w.x) - u.x, (pc ? 0.0 : w.y) - u.y);
        }
    }
    if (bad) S.bad = 1;
    S.dinv[c * kPitch + r] = w.x;
    Dk[sw(r, c)] = w.x;
    if constexpr (CP) {
        S.dinv[kSB + c * kPitch + r] = w.y;
        Dk[kBE + sw(r, c)] = w.y;
    }
}

// Factor in place (the compute warps): on return block (K, K) holds D_K^-1 and
// (I, K) holds L_IK; S.bad is set when a pivot vanished.
template <Op OP>
__device__ __forceinline__ void factor(double* L, double* Gring, int nblk, Shared& S, double* stage) {
    constexpr bool CP = OP == OP_LSCM;
    constexpr int BB = kBE * (CP ? 2 : 1), SB = kSB * (CP ? 2 : 1);
    constexpr int kAhead = 3;   // blocks of G whose loads are in flight together
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sc = tid >> 4, sr = (tid & 15) ^ sc;   // the element at offset tid of a stored block
    for (int K = 0; K < nblk; ++K) {
        const int f = S.first[K], wl = K - f;
        // block rows below K that reach column K (first[] does not decrease)
        const int cnt = __popc(__ballot_sync(0xffffffffu, lane < kMaxW && K + 1 + lane < nblk &&
                                                              S.first[min(K + 1 + lane, kMaxBlk)] <= K));
        double* Lrow = L + static_cast<size_t>(S.off[K]) * BB;
        double* Dk = Lrow + static_cast<size_t>(wl) * BB;
        // L_K. of the earlier columns into shared memory
#pragma unroll 3
        for (int k = 0; k < wl; ++k) {
            stage[k * SB + sc * kPitch + sr] = Lrow[static_cast<size_t>(k) * BB + tid];
            if constexpr (CP) stage[k * SB + kSB + sc * kPitch + sr] = Lrow[static_cast<size_t>(k) * BB + kBE + tid];
        }
        if (tid < kNB) S.diag[tid] = Dk[sw(tid, tid)];
        compute_sync();
        // S_IK for I = K .. K + cnt, half a block (8 rows) per task
        for (int t = warp; t < 2 * (cnt + 1); t += kCW) {
            const int R = K + (t >> 1), mt = t & 1;
            double* blk = L + static_cast<size_t>(S.off[R] + K - S.first[R]) * BB;
            double acc[CP ? 4 : 2][2];
            const int row = (lane >> 2) + 8 * mt, col = 2 * (lane & 3);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int e = sw(row, 8 * nt + col + u);
                    acc[nt][u] = blk[e];
                    if constexpr (CP) acc[2 + nt][u] = blk[kBE + e];
                }
            const double* Gr = Gring + static_cast<size_t>((R & 15) * 16) * BB;
            for (int M = S.first[R]; M < K; M += kAhead) {
                double a[kAhead][4], ai[kAhead][CP ? 4 : 1];
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    load_a<CP>(Gr + static_cast<size_t>(min(M + u, K - 1) & 15) * BB, mt, lane, a[u], ai[u]);
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (M + u < K) block_mma<CP, true>(acc, a[u], ai[u], stage + (M + u - f) * SB, lane);
            }
            double* G = Gring + static_cast<size_t>((R & 15) * 16 + (K & 15)) * BB;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int c = 8 * nt + col + u;
                    if (R == K) {
                        S.dsm[row * (kNB + 1) + c] = acc[nt][u];
                        if constexpr (CP) S.dsm[kNB * (kNB + 1) + row * (kNB + 1) + c] = acc[2 + nt][u];
                    } else {
                        G[sw(row, c)] = acc[nt][u];
                        if constexpr (CP) G[kBE + sw(row, c)] = acc[2 + nt][u];
                    }
                }
        }
        compute_sync();
        invert_block<CP>(S, Dk);
        compute_sync();
        if (S.bad) return;
        for (int t = warp; t < 2 * cnt; t += kCW) {   // L_IK = S_IK D^-1
            const int R = K + 1 + (t >> 1), mt = t & 1;
            double acc[CP ? 4 : 2][2] = {};
            double a[4], ai[CP ? 4 : 1];
            load_a<CP>(Gring + static_cast<size_t>((R & 15) * 16 + (K & 15)) * BB, mt, lane, a, ai);
            block_mma<CP, false>(acc, a, ai, S.dinv, lane);
            double* blk = L + static_cast<size_t>(S.off[R] + K - S.first[R]) * BB;
            const int row = (lane >> 2) + 8 * mt, col = 2 * (lane & 3);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int e = sw(row, 8 * nt + col + u);
                    blk[e] = acc[nt][u];
                    if constexpr (CP) blk[kBE + e] = acc[2 + nt][u];
                }
        }
        compute_sync();
    }
}

// The real factor as a call of its own, its registers apart from the solve's:
// 4 % off ARAP (100 uneven islands, 12 iterations: 13.85 -> 13.21 ms). The complex
// one spills then and stays inline.
__device__ __noinline__ void factor_arap(double* L, double* Gring, int nblk, Shared& S, double* stage) {
    factor<OP_ARAP>(L, Gring, nblk, S, stage);
}

// ------------------------------------------------------------------ solve
// rb <- A^-1 rb. Group g = tid / 16 owns the block rows congruent to g: the
// right-hand side of its current row stays in registers until the row is
// final, then the group publishes it and takes the row 16 further on. The
// last warp feeds the ring: it copies a step's blocks once the compute warps
// have released the stage. A wait that runs out sets S.bad: the feeding warp
// stops copying and the compute warps go through their steps with hardly a wait
// (on whatever the stages hold). rb is then worthless and not used; the CTA
// takes no further island and waits for the copies in flight before it ends.
template <Op OP>
__device__ void solve(Isl& I, Shared& S, double* stage) {
    constexpr bool CP = OP == OP_LSCM;
    constexpr int BB = kBE * (CP ? 2 : 1);
    constexpr unsigned kBytes = BB * sizeof(double);
    const int tid = threadIdx.x, lane = tid & 31, g = tid >> 4, r = tid & 15;
    const int nblk = I.nblk, NS = I.stages;
    const int stage_d = kRing / 8 / NS / 2 * 2;    // doubles per stage (16-byte multiple)
    const unsigned full0 = smem_addr(S.full), empty0 = smem_addr(S.empty), st0 = smem_addr(stage);
    int q = I.q, ph = I.ph;
    auto next = [&]() {
        if (++q == NS) { q = 0; ph ^= 1; }
    };
    if (tid >= kCT) {
        bool run = true;
        for (int K = 0; K < nblk && run; ++K) {   // column K's blocks, one copy each
            const int R = K + 1 + lane;
            const bool on = lane < kMaxW && R < nblk && S.first[min(R, kMaxBlk)] <= K;
            const unsigned cnt = __popc(__ballot_sync(0xffffffffu, on));
            run = __all_sync(0xffffffffu, mbar_wait(S.bad, empty0 + 8 * q, ph ^ 1));
            if (!run) break;
            if (lane == 0) mbar_expect(full0 + 8 * q, cnt * kBytes);
            __syncwarp();
            if (on)
                bulk_copy(st0 + q * stage_d * 8 + lane * kBytes,
                          I.L + static_cast<size_t>(S.off[R] + K - S.first[R]) * BB, kBytes, full0 + 8 * q);
            next();
        }
        for (int K = nblk - 1; K >= 0 && run; --K) {   // row K's blocks are contiguous
            const unsigned bytes = (K - S.first[K]) * kBytes;
            run = __all_sync(0xffffffffu, mbar_wait(S.bad, empty0 + 8 * q, ph ^ 1));
            if (!run) break;
            if (lane == 0) {
                mbar_expect(full0 + 8 * q, bytes);
                if (bytes)
                    bulk_copy(st0 + q * stage_d * 8, I.L + static_cast<size_t>(S.off[K]) * BB, bytes, full0 + 8 * q);
            }
            __syncwarp();
            next();
        }
    } else {
        // ---- forward: r_I -= L_IK r_K
        int R = g;
        double2 acc = R < nblk ? I.rb[R * kNB + r] : make_double2(0.0, 0.0);
        double2 nxt = R + 16 < nblk ? I.rb[(R + 16) * kNB + r] : make_double2(0.0, 0.0);
        int fr = R < nblk ? S.first[R] : nblk;
        for (int K = 0; K < nblk; ++K) {
            if (R == K) {
                S.xk[K & 1][r] = acc;
                I.rb[K * kNB + r] = acc;
                R += 16;
                acc = nxt;
                fr = R < nblk ? S.first[R] : nblk;
                if (R + 16 < nblk) nxt = I.rb[(R + 16) * kNB + r];
            }
            compute_sync();   // r_K visible
            mbar_wait(S.bad, full0 + 8 * q, ph);
            if (fr <= K) {
                const double* B = stage + q * stage_d + (R - K - 1) * BB;
                const double2* x = S.xk[K & 1];
                double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
#pragma unroll
                for (int c = 0; c < kNB; c += 2) {
                    const double l0 = B[sw(r, c)], l1 = B[sw(r, c + 1)];
                    const double2 x0 = x[c], x1 = x[c + 1];
                    ax += l0 * x0.x; ay += l0 * x0.y;
                    bx += l1 * x1.x; by += l1 * x1.y;
                    if constexpr (CP) {
                        const double m0 = B[kBE + sw(r, c)], m1 = B[kBE + sw(r, c + 1)];
                        ax -= m0 * x0.y; ay += m0 * x0.x;
                        bx -= m1 * x1.y; by += m1 * x1.x;
                    }
                }
                acc.x -= ax + bx;
                acc.y -= ay + by;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * q);
            next();
        }
        compute_sync();
        // ---- z_K = D_K^-1 r_K, every block at once
        for (int K0 = 0; K0 < nblk; K0 += kCT / 16) {   // the same trip count on both groups of a warp
            const int K = min(K0 + g, nblk - 1);
            const double* B = I.L + static_cast<size_t>(S.off[K + 1] - 1) * BB;
            const double2 own = I.rb[K * kNB + r];
            double zx = 0.0, zy = 0.0;
#pragma unroll
            for (int c = 0; c < kNB; ++c) {
                const double l = B[sw(r, c)];
                const double xx = __shfl_sync(0xffffffffu, own.x, c, 16), xy = __shfl_sync(0xffffffffu, own.y, c, 16);
                zx += l * xx; zy += l * xy;
                if constexpr (CP) {
                    const double m = B[kBE + sw(r, c)];
                    zx -= m * xy; zy += m * xx;
                }
            }
            if (K0 + g < nblk) I.rb[K * kNB + r] = make_double2(zx, zy);
        }
        compute_sync();
        // ---- backward: z_J -= L_KJ^H x_K
        int J = nblk - 1 - ((nblk - 1 - g) & 15);          // the highest block row congruent to g
        acc = J >= 0 ? I.rb[J * kNB + r] : make_double2(0.0, 0.0);
        nxt = J - 16 >= 0 ? I.rb[(J - 16) * kNB + r] : make_double2(0.0, 0.0);
        for (int K = nblk - 1; K >= 0; --K) {
            if (J == K) {
                S.xk[K & 1][r] = acc;
                I.rb[K * kNB + r] = acc;
                J -= 16;
                acc = nxt;
                if (J - 16 >= 0) nxt = I.rb[(J - 16) * kNB + r];
            }
            const int f = S.first[K];
            compute_sync();
            mbar_wait(S.bad, full0 + 8 * q, ph);
            if (J >= f) {   // J < K
                const double* B = stage + q * stage_d + (J - f) * BB;
                const double2* x = S.xk[K & 1];
                double ax = 0.0, ay = 0.0, bx = 0.0, by = 0.0;
#pragma unroll
                for (int c = 0; c < kNB; c += 2) {
                    const double l0 = B[sw(c, r)], l1 = B[sw(c + 1, r)];
                    const double2 x0 = x[c], x1 = x[c + 1];
                    ax += l0 * x0.x; ay += l0 * x0.y;
                    bx += l1 * x1.x; by += l1 * x1.y;
                    if constexpr (CP) {
                        const double m0 = B[kBE + sw(c, r)], m1 = B[kBE + sw(c + 1, r)];
                        ax += m0 * x0.y; ay -= m0 * x0.x;
                        bx += m1 * x1.y; by -= m1 * x1.x;
                    }
                }
                acc.x -= ax + bx;
                acc.y -= ay + by;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty0 + 8 * q);
            next();
        }
    }
    I.q = q;
    I.ph = ph;
    __syncthreads();
}

// The copies in flight after a wait ran out, with a limit again (a stage that was
// never copied into counts as there).
__device__ __noinline__ void drain(Shared& S) {
    int late = 0, q = S.dead_q, ph = S.dead_ph;
    for (int k = 0; k < S.dead_stages; ++k) {
        if (--q < 0) { q = S.dead_stages - 1; ph ^= 1; }
        mbar_wait(late, smem_addr(S.full) + 8 * q, ph);
    }
}

// ------------------------------------------------------------------ ARAP
// gpu.py:230-249 / param.py:379-414. False (with U untouched) when the first
// global step does not reach the tolerance or a wait ran out in it: the CG path
// takes the island. A wait that runs out later leaves U as the iterations
// before it made it, with UVA_ST_TIMEOUT.
__device__ bool solve_arap(const uva_batch& b, const uva_solve_params& prm, Isl& I, Shared& S, Red& rd, double* stage) {
    const int tid = threadIdx.x;
    const bool batch = b.semantics == UVA_SEM_BATCH;
    double2* U = reinterpret_cast<double2*>(b.U);
    double2* x64 = reinterpret_cast<double2*>(b.x64) + I.v0;
    double2* b64 = reinterpret_cast<double2*>(b.b64) + I.v0;
    const double2* rc = reinterpret_cast<const double2*>(b.rc);
    uva_island_status st{};
    bool use_ls = prm.line_search != 0;
    double prev_e = 0.0;
    for (int i = tid; i < I.n; i += kNT) x64[i] = U[I.v0 + __ldg(b.row_vert + I.v0 + i)];
    __syncthreads();
    for (int i = tid; i < I.n; i += kNT) I.lu[i] = apply<OP_ARAP>(b, I, i, x64);
    for (int it = 0; it < prm.iters; ++it) {
        double ev[2] = {0.0, 0.0};
        for (int f = I.f0 + tid; f < I.f0 + I.nt; f += kNT) {
            double e; int fl;
            local_terms(b, I.v0, f, U, batch, e, fl);
            ev[0] += e; ev[1] += fl;
        }
        if (!batch) {
            cta_sum<2>(rd, ev);
            if (it == 0) {
                use_ls = prm.line_search != 0 && ev[1] == 0.0;
                prev_e = ev[0];
            } else if (prm.energy_tol > 0.0 && fabs(prev_e - ev[0]) <= prm.energy_tol * fmax(prev_e, 1e-300)) {
                st.flags |= UVA_ST_ENERGYSTOP;
                st.energy = ev[0];
                break;
            } else {
                prev_e = ev[0];
            }
            st.energy = ev[0];
        }
        __syncthreads();   // corner terms complete
        double bb[2] = {0.0, 0.0};
        for (int i = tid; i < I.n; i += kNT) {   // right-hand side and residual at U
            const int v = I.v0 + __ldg(b.row_vert + I.v0 + i);
            double bx = 0.0, by = 0.0;
            const int pe = __ldg(b.vt_ptr + v + 1);
            for (int p = __ldg(b.vt_ptr + v); p < pe; ++p) {
                const double2 c = rc[__ldg(b.vt + p)];
                bx += c.x; by += c.y;
            }
            const double2 u = U[v], lu = I.lu[i];
            if (i == I.pin) { bx += I.wpin * u.x; by += I.wpin * u.y; }
            b64[i] = make_double2(bx, by);
            x64[i] = u;
            I.rb[__ldg(I.pos + i)] = make_double2(bx - lu.x, by - lu.y);
            bb[0] += bx * bx; bb[1] += by * by;
        }
        for (int i = I.n + tid; i < I.nblk * kNB; i += kNT) I.rb[i] = make_double2(0.0, 0.0);
        cta_sum<2>(rd, bb);   // also publishes rb
        const double t0 = prm.tol * prm.tol * fmax(bb[0], 1e-300), t1 = prm.tol * prm.tol * fmax(bb[1], 1e-300);
        bool capped = false, bad = false;
        for (int ref = 0;; ++ref) {   // one solve unless the operator is nearly singular
            solve<OP_ARAP>(I, S, stage);
            for (int i = tid; i < I.n; i += kNT) {
                const double2 d = I.rb[__ldg(I.pos + i)];
                double2 x = x64[i];
                x.x += d.x; x.y += d.y;
                x64[i] = x;
            }
            __syncthreads();
            double rr[3] = {0.0, 0.0, 0.0};
            for (int i = tid; i < I.n; i += kNT) {
                const double2 y = apply<OP_ARAP>(b, I, i, x64), rhs = b64[i], x = x64[i];
                I.y[i] = y;
                const double rx = rhs.x - y.x, ry = rhs.y - y.y;
                I.rb[__ldg(I.pos + i)] = make_double2(rx, ry);
                rr[0] += rx * rx; rr[1] += ry * ry;
                if (!finite2(x)) rr[2] += 1.0;
            }
            cta_sum<3>(rd, rr);
            ++st.refinements;
            st.resid[0] = sqrt(rr[0] / fmax(bb[0], 1e-300));
            st.resid[1] = sqrt(rr[1] / fmax(bb[1], 1e-300));
            bad = rr[2] != 0.0;
            // an ill-conditioned island gets one more solve even within the tolerance
            const double few = ref == 0 ? 1e-11 / fmax(prm.tol, 1e-11) : 1.0;
            if (rr[0] <= t0 * few * few && rr[1] <= t1 * few * few) {
                capped = S.bad != 0;
                break;
            }
            if (ref >= min(prm.max_refine, 3) || !isfinite(rr[0] + rr[1]) || S.bad) {
                capped = !(rr[0] <= t0 && rr[1] <= t1);
                break;
            }
            for (int i = I.n + tid; i < I.nblk * kNB; i += kNT) I.rb[i] = make_double2(0.0, 0.0);
            __syncthreads();
        }
        if (capped) {
            if (it == 0 && (!bad || S.bad)) return false;
            if (S.bad) {
                st.flags |= UVA_ST_TIMEOUT;
                break;
            }
            st.flags |= UVA_ST_MAXITER;
        }
        st.outer_iters = it + 1;
        if (bad) {   // non-finite charts keep their layout (gpu.py:235-240)
            st.flags |= UVA_ST_NONFINITE;
            continue;
        }
        double step = 1.0;
        if (use_ls) {
            double tmin = 1e30;
            int folded = 0;
            for (int f = I.f0 + tid; f < I.f0 + I.nt; f += kNT) {
                tmin = fmin(tmin, step_bound(b, I.v0, f, U, reinterpret_cast<const double2*>(b.x64), batch));
                if (prm.fold_step) folded |= folded_tri(b, I.v0, f, U);
            }
            tmin = cta_min(rd, tmin);
            if (prm.fold_step) folded = __syncthreads_or(folded);   // folded islands: plain ARAP step
            step = folded ? 1.0 : fmin(0.9 * tmin, 1.0);
        }
        st.step = step;
        __syncthreads();   // all line-search reads of U done
        for (int i = tid; i < I.n; i += kNT) {
            const int v = I.v0 + __ldg(b.row_vert + I.v0 + i);
            const double2 x = x64[i], y = I.y[i];
            double2 u = U[v], lu = I.lu[i];
            if (use_ls) {
                u.x += (x.x - u.x) * step; u.y += (x.y - u.y) * step;
                lu.x += (y.x - lu.x) * step; lu.y += (y.y - lu.y) * step;
            } else {
                u = x; lu = y;
            }
            U[v] = u;
            I.lu[i] = lu;
        }
        __syncthreads();
    }
    if (tid == 0) b.status[I.id] = st;
    return true;
}

// ------------------------------------------------------------------ LSCM
// Hard pins p0 -> (0,0), p1 -> (|P[p1]-P[p0]|, 0), param.py:136-169. False
// when the residual stays above the tolerance or a wait ran out.
__device__ bool solve_lscm(const uva_batch& b, const uva_solve_params& prm, Isl& I, Shared& S, Red& rd, double* stage) {
    const int tid = threadIdx.x;
    double2* x64 = reinterpret_cast<double2*>(b.x64) + I.v0;
    double2* U = reinterpret_cast<double2*>(b.U);
    const double* pp0 = b.P + 3 * (I.v0 + b.pins[3 * I.id + 1]);
    const double* pp1 = b.P + 3 * (I.v0 + b.pins[3 * I.id + 2]);
    const double ax = pp1[0] - pp0[0], ay = pp1[1] - pp0[1], az = pp1[2] - pp0[2];
    const double dpin = sqrt(ax * ax + ay * ay + az * az);
    uva_island_status st{};
    for (int i = tid; i < I.n; i += kNT) x64[i] = make_double2(i == I.p1 ? dpin : 0.0, 0.0);
    __syncthreads();
    double bb = 0.0;
    bool done = false, bad = false;
    for (int ref = 0;; ++ref) {
        double rr[2] = {0.0, 0.0};
        for (int i = tid; i < I.n; i += kNT) {
            double2 r = make_double2(0.0, 0.0);
            const double2 x = x64[i];
            if (i != I.p0 && i != I.p1) {
                r = apply<OP_LSCM>(b, I, i, x64);
                r.x = -r.x; r.y = -r.y;
            }
            I.rb[__ldg(I.pos + i)] = r;
            rr[0] += r.x * r.x + r.y * r.y;
            if (!finite2(x)) rr[1] += 1.0;
        }
        for (int i = I.n + tid; i < I.nblk * kNB; i += kNT) I.rb[i] = make_double2(0.0, 0.0);
        cta_sum<2>(rd, rr);   // also publishes rb
        ++st.refinements;
        if (ref == 0) bb = rr[0];   // x = pins only: the residual is the right-hand side
        st.resid[0] = st.resid[1] = sqrt(rr[0] / fmax(bb, 1e-300));
        bad = rr[1] != 0.0;
        done = rr[0] <= prm.tol * prm.tol * fmax(bb, 1e-300);
        // an ill-conditioned island (a long strip) gets one more solve even
        // within the tolerance
        const bool good = rr[0] <= 1e-22 * fmax(bb, 1e-300);
        if ((done && (good || ref > 1)) || ref > min(prm.max_refine, 3) || !isfinite(rr[0]) || (ref > 0 && S.bad)) break;
        solve<OP_LSCM>(I, S, stage);
        for (int i = tid; i < I.n; i += kNT) {
            const double2 d = I.rb[__ldg(I.pos + i)];
            double2 x = x64[i];
            x.x += d.x; x.y += d.y;
            x64[i] = x;
        }
        __syncthreads();
    }
    if (!done || bad) return false;
    for (int i = tid; i < I.n; i += kNT) U[I.v0 + __ldg(b.row_vert + I.v0 + i)] = x64[i];
    st.outer_iters = 1;
    if (tid == 0) b.status[I.id] = st;
    return true;
}

// Bytes of an island's factor, ring of G and vectors.
template <Op OP>
__device__ __forceinline__ int64_t factor_bytes(int blocks, int nblk) {
    constexpr bool CP = OP == OP_LSCM;
    return (static_cast<int64_t>(blocks) + 256) * kBE * (CP ? 2 : 1) * 8 + static_cast<int64_t>(nblk) * kNB * 16 * (CP ? 1 : 3);
}

// ------------------------------------------------------------------ choice
// Factors or CG for a launch: estimates of both in microseconds, from the
// island sizes. Measured on disks of 32 to 16,000 vertices, 1 to 20,000 of
// them, alike and uneven, 3 to 20 ARAP iterations, at the default tolerances
// (70 batches): the estimates are within 15 % for factors, 30 % for CG, whose
// iterations depend on the shape.
//  * Factors: a chain of block columns and of substitutions per island,
//    proportional to its vertices (`lat`), two CTAs per SM; slower by up to a
//    third once the launch's factors exceed the L2.
//  * CG: a warp, a quarter CTA or a CTA per island by size class (up to 256,
//    2,048, 8,192 vertices, above: vectors in global memory), an SM's time per
//    vertex (`thr`) when there are more islands than teams.
// ARAP has the factors' chain in every iteration, so few islands of 5,000 to
// 8,000 vertices are faster by CG, whose CTA has 1,024 threads for them: 20
// iterations of 400 uneven islands (20 to 7,904 vertices) 24.3 ms by factors,
// 16.7 by CG; of 100 of them 20.6 and 13.2; but of 2,000 uneven ones
// 29.1 and 39.4, of 1,200 islands of 877 12.5 and 19.0. LSCM is slower by
// factors only for thousands of islands of some 60 vertices and fewer: 20,000
// of 24: 1.58 ms and 0.69.
// Islands without a factor take CG after the others: where one of them lasts as
// long as the launch by CG alone would, the factors' launch before it is time
// lost (60 irregular charts of 3,000 vertices, 10 with a factor: ARAP 19.9 ms, 11.9
// by CG alone). CG is taken when it is expected to save an eighth.
struct Cost {
    float lat, thr;
};
template <Op OP>
__device__ __forceinline__ Cost factor_cost(float n, float iters) {
    const float t = OP == OP_ARAP ? 15.f + 3.f * iters + n * (0.33f + 1.9e-5f * n + 0.093f * iters)
                                  : 8.f + n * (0.53f + 4.5e-5f * n);
    return {t, t * fminf(1.55f, 1.15f + 2e-4f * n)};
}
template <Op OP>
__device__ __forceinline__ Cost cg_cost(float n, float iters) {
    if (OP == OP_ARAP) {
        const float k = sqrtf(iters);   // later iterations start near their solution
        return {n <= UVA_CLASS_SMALL ? 9.f * k * n
                                     : (n <= UVA_CLASS_MID ? 0.95f * k * n : (n <= UVA_CLASS_BIG ? 1.f : 3.f) * k * (1300.f + 0.28f * n)),
                n <= 128.f ? n * (0.3f * iters - 0.3f) : 0.42f * k * n};
    }
    return {n * (n <= UVA_CLASS_SMALL ? 6.f : (n <= UVA_CLASS_BIG ? 3.2f : 8.6f)),
            n * (n <= 400.f ? 0.12f + 0.0032f * n : (n <= UVA_CLASS_MID ? 1.4f : 4.f))};
}

// work[kWorkCg] = 1: CG for the whole launch. Islands above kDirectMaxN have
// their own launch either way and are left out.
template <Op OP>
__global__ void __launch_bounds__(1024) k_choose(uva_batch b, uva_solve_params prm) {
    __shared__ float part[32][7];
    const int64_t* ofs = b.direct_ofs + (OP == OP_LSCM ? b.direct_slots + 1 : 0);
    const float iters = static_cast<float>(prm.iters);
    // 0 longest factor, 1 sum of factors, 2 their vertices, 3 longest of the
    // CG islands, 4 their sum, 5 longest of all by CG, 6 their sum
    float v[7] = {};
    for (int r = threadIdx.x; r < b.nc; r += 1024) {
        const int isl = b.order[r], n = b.vofs[isl + 1] - b.vofs[isl];
        if (n > kDirectMaxN) continue;
        const int32_t* info = band_info(b, isl);
        const int part_of = min(r, b.direct_slots - 1);
        const bool takes = (info[0] & 1) &&
                           factor_bytes<OP>(info[1], (n + kNB - 1) / kNB) <= ofs[part_of + 1] - ofs[part_of];
        const Cost cg = cg_cost<OP>(static_cast<float>(n), iters);
        v[5] = fmaxf(v[5], cg.lat);
        v[6] += cg.thr;
        if (takes) {
            const Cost f = factor_cost<OP>(static_cast<float>(n), iters);
            v[0] = fmaxf(v[0], f.lat);
            v[1] += f.thr;
            v[2] += static_cast<float>(n);
        } else {
            v[3] = fmaxf(v[3], cg.lat);
            v[4] += cg.thr;
        }
    }
    constexpr unsigned kMax = 1u | 8u | 32u;   // 0, 3, 5: maxima, the others sums
#pragma unroll
    for (int k = 0; k < 7; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float y = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = kMax >> k & 1 ? fmaxf(v[k], y) : v[k] + y;
        }
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][k] = v[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 7; ++k) {   // on every thread
        v[k] = part[0][k];
        for (int w = 1; w < 32; ++w) v[k] = kMax >> k & 1 ? fmaxf(v[k], part[w][k]) : v[k] + part[w][k];
    }
    constexpr float kSMs = 148.f;
    // a tighter tolerance takes CG more iterations; ARAP islands that could have
    // a factor are solved to half of it (solve.cu), an eighth more time
    const float tight = (OP == OP_ARAP ? 1.12f : 1.f) *
                        logf(fmaxf(static_cast<float>(prm.tol), 1e-30f)) / logf(OP == OP_ARAP ? 2e-7f : 1e-8f);
    auto both = [&](float lat, float sum) { return tight * sqrtf(lat * lat + sum * sum / (kSMs * kSMs)); };
    const float spill = fminf(1.f, v[2] / 4e5f);
    // CTAs beside one another: the launch's, or two per SM where each has one island
    const float ctas = b.direct_slots < b.nc ? static_cast<float>(b.direct_slots) : 2.f * kSMs;
    const float direct = fmaxf(v[0] * (1.f + (OP == OP_ARAP ? 0.35f : 0.2f) * spill), v[1] / ctas);
    // charts without a factor are irregular ones, on which CG takes longer than on
    // disks (ARAP some 1.5 times, LSCM 1.15); so rough an estimate counts from
    // half a millisecond
    const float shape = v[3] > 0.f ? (OP == OP_ARAP ? 1.5f : 1.15f) : 1.f;
    const float rest = shape * both(v[3], v[4]), all = shape * both(v[5], v[6]);
    const float gain = direct + rest - all;
    if (!(v[2] > 0.f && gain > 0.12f * (direct + rest) && (rest == 0.f || gain > 500.f))) return;
    for (int r = threadIdx.x; r < b.nc; r += 1024) band_info(b, r)[3] = 0;
    if (threadIdx.x == 0) {
        b.work[kWorkLeft] = b.nc;
        b.work[kWorkCg] = 1;
    }
}

// One CTA per island, largest first; CTA j starts with the j-th island (its
// scratch is sized for that one, the later ones are smaller). info[3] of an
// island tells the CG launch that follows whether it is done.
template <Op OP>
__global__ void __launch_bounds__(kNT, 2) k_direct(uva_batch b, uva_solve_params prm) {
    constexpr bool CP = OP == OP_LSCM;
    constexpr int BB = kBE * (CP ? 2 : 1);
    extern __shared__ __align__(128) double stage[];
    __shared__ Shared S;
    const int tid = threadIdx.x;
    if (b.work[kWorkCg]) return;   // every island is left
    const int64_t* ofs = b.direct_ofs + (CP ? b.direct_slots + 1 : 0);
    unsigned char* mem = b.direct + ofs[blockIdx.x];
    const int64_t room = ofs[blockIdx.x + 1] - ofs[blockIdx.x];
    Red rd{S.red, 0};
    int rank = blockIdx.x;
    bool dead = false;   // a wait ran out: the CTA leaves its further islands to CG
    while (rank < b.nc) {
        Isl I;
        I.id = b.order[rank];
        I.v0 = b.vofs[I.id]; I.n = b.vofs[I.id + 1] - I.v0;
        I.f0 = b.tofs[I.id]; I.nt = b.tofs[I.id + 1] - I.f0;
        I.s0 = b.sofs[I.id];
        I.wpin = b.wpin[I.id];
        I.nblk = (I.n + kNB - 1) / kNB;
        I.pos = b.band + I.v0;
        int32_t* info = band_info(b, I.id);
        const int total = info[1];
        const int npad = I.nblk * kNB;
        const int64_t need = factor_bytes<OP>(total, I.nblk);
        bool done = false;
        const long long t0 = global_ns();
        if (!dead && (info[0] & 1) && need <= room) {
            const int32_t* first = band_first(b, I.v0, I.id);
            I.pin = b.vert_row[I.v0 + b.pins[3 * I.id]];
            const int q0 = b.pins[3 * I.id + 1], q1 = b.pins[3 * I.id + 2];
            I.p0 = q0 >= 0 ? b.vert_row[I.v0 + q0] : -1;
            I.p1 = q1 >= 0 ? b.vert_row[I.v0 + q1] : -1;
            I.L = reinterpret_cast<double*>(mem);
            I.G = I.L + static_cast<size_t>(total) * BB;
            I.rb = reinterpret_cast<double2*>(I.G + static_cast<size_t>(256) * BB);
            I.y = I.rb + npad;
            I.lu = I.y + npad;
            const int w = max(info[2], 1);
            I.stages = max(1, min(kMaxStages, kRing / (w * BB * 8)));
            I.q = I.ph = 0;
            // skyline and block offsets
            constexpr int kPer = (kMaxBlk + kNT - 1) / kNT;
            int sum = 0, fs[kPer];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int k = tid * kPer + j;
                fs[j] = k < I.nblk ? first[k] : 0;
                if (k < I.nblk) { S.first[k] = static_cast<unsigned short>(fs[j]); sum += k - fs[j] + 1; }
            }
            int inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, inc, o);
                if ((tid & 31) >= o) inc += x;
            }
            if ((tid & 31) == 31) S.scan[tid >> 5] = inc;
            if (tid == 0) S.bad = 0;
            if (tid < I.stages) {
                mbar_init(smem_addr(S.full + tid), 1);
                mbar_init(smem_addr(S.empty + tid), kCW);
            }
            __syncthreads();
            int at = inc - sum;
            for (int k = 0; k < (tid >> 5); ++k) at += S.scan[k];
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int k = tid * kPer + j;
                if (k < I.nblk) { S.off[k] = at; at += k - fs[j] + 1; }
                if (k == I.nblk - 1) S.off[I.nblk] = at;
            }
            asm volatile("fence.proxy.async;" ::: "memory");   // mbarrier.init before the bulk copies
            __syncthreads();
            if (CP && I.p0 < 0) {   // closed surface: no far pair
                double2* U = reinterpret_cast<double2*>(b.U);
                for (int i = tid; i < I.n; i += kNT) U[I.v0 + i] = make_double2(0.0, 0.0);
                if (tid == 0) {
                    uva_island_status st{};
                    st.flags = UVA_ST_NOBOUNDARY;
                    b.status[I.id] = st;
                }
                done = true;
            } else {
                assemble<OP>(b, I, S);
                if (tid < kCT) {
                    if constexpr (CP) factor<OP>(I.L, I.G, I.nblk, S, stage);
                    else factor_arap(I.L, I.G, I.nblk, S, stage);
                }
                // the substitutions read the factor through the asynchronous proxy
                asm volatile("fence.proxy.async;" ::: "memory");
                __syncthreads();
                if (S.bad == 0) {
                    if (CP) done = solve_lscm(b, prm, I, S, rd, stage);
                    else done = solve_arap(b, prm, I, S, rd, stage);
                    if (S.bad == 2) {
                        dead = true;
                        if (tid == kCT) { S.dead_q = I.q; S.dead_ph = I.ph; S.dead_stages = I.stages; }
                    }
                }
            }
            __syncthreads();
            if (tid < I.stages && !dead) {
                asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(S.full + tid)) : "memory");
                asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(S.empty + tid)) : "memory");
            }
        }
        if (tid == 0) {
            info[3] = done ? 1 : 0;
            if (done) {
                uva_island_status& st = b.status[I.id];
                st.t_begin = t0;
                st.t_end = global_ns();
                st.sm = static_cast<int32_t>(sm_id());
                st.team = kCT;
            } else {
                atomicAdd(b.work + kWorkLeft, 1);
            }
            S.rank = static_cast<int>(gridDim.x) + atomicAdd(b.work + kWorkNext, 1);
        }
        __syncthreads();
        rank = S.rank;
        __syncthreads();
    }
    if (dead && tid >= kCT) drain(S);
}

template <Op OP>
cudaError_t direct_attr() {
    static std::mutex mu;
    static std::vector<char> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (static_cast<int>(done.size()) <= dev) done.resize(dev + 1, 0);
    if (done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_direct<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRing);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_band, cudaFuncAttributeMaxDynamicSharedMemorySize, kDirectMaxN * 4);
    if (e == cudaSuccess) done[dev] = 1;
    return e;
}

}  // namespace

cudaError_t uva_direct_attributes() {
    const cudaError_t e = direct_attr<OP_ARAP>();
    return e == cudaSuccess ? direct_attr<OP_LSCM>() : e;
}

int uva_direct_order(const uva_batch* b, cudaStream_t s) {
    const cudaError_t e = direct_attr<OP_ARAP>();
    if (e != cudaSuccess) return uva_cuda_status(e, "uva_batch_setup/band attribute");
    const int n = std::min(std::max(b->maxrows, 1), kDirectMaxN);
    k_band<<<b->nc, kNT, static_cast<size_t>(n) * 4, s>>>(*b);
    UVA_CHECK_LAUNCH("uva_batch_setup/band");
    return UVA_OK;
}

int uva_direct_launch(const uva_batch* b, const uva_solve_params* prm, bool lscm, cudaStream_t s) {
    const cudaError_t e = lscm ? direct_attr<OP_LSCM>() : direct_attr<OP_ARAP>();
    if (e != cudaSuccess) return uva_cuda_status(e, "uva_direct/cudaFuncSetAttribute");
    const int grid = std::min(b->nc, b->direct_slots);
    // few and small islands: factors won every measurement, and even irregular
    // charts of up to 700 vertices fit (the choice would cost 4 of some 120 us)
    if (b->maxrows > 700 || b->nc > 592) {
        if (lscm) k_choose<OP_LSCM><<<1, 1024, 0, s>>>(*b, *prm);
        else k_choose<OP_ARAP><<<1, 1024, 0, s>>>(*b, *prm);
        UVA_CHECK_LAUNCH("uva_direct/choose");
    }
    if (lscm) k_direct<OP_LSCM><<<grid, kNT, kRing, s>>>(*b, *prm);
    else k_direct<OP_ARAP><<<grid, kNT, kRing, s>>>(*b, *prm);
    UVA_CHECK_LAUNCH(lscm ? "uva_lscm/direct" : "uva_arap/direct");
    return UVA_OK;
}
