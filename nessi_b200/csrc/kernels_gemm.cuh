// Complex FP64 GEMM tiles on the FP64 tensor cores (mma.sync m16n8k8 .f64), the contraction
// engine of every Sigma-shared product of a time step:
//   Matsubara part of the tv row      Cmat = K_n . Gmat_all          (conv_impl :410-540)
//   les*adv                           gles = Sigma^<_dense . badv     (conv_impl :1244-1394)
//   tv*vt                             gles += Sigma^tv . btv          (conv_impl :1075-1242)
//   Volterra trailing updates         vacc += Sigma^R . vy            (dyson_impl :179-213, :983-1011)
// In all of them the rows are time indices (t, a) and the columns are the problems of a group
// (p, d), so one product serves every k-point that shares Sigma.
//
// Operands are read through loader objects, so that a product can read a triangle, a panel or a
// dense matrix in place; KC tells whether consecutive k are adjacent in memory (then consecutive
// threads load consecutive k, otherwise consecutive m / n).  Real and imaginary parts are
// accumulated separately (four real MMAs per complex fragment product).
#pragma once
#include "device_common.cuh"

namespace zg {
constexpr int BK = 8;        // complex k per stage (one m16n8k8 k-step)
constexpr int NTH = 128;     // threads of a tile group
}  // namespace zg

// D (16x8, fp64) += A (16x8) B (8x8); fragment layout of mma.m16n8k8 .f64: with g = lane/4,
// q = lane%4: a[v0 + 2 v1] = A[g + 8 v0][q + 4 v1], b[v] = B[q + 4 v][g],
// d[v0 + 2 v1] = D[g + 8 v1][2 q + v0].
__device__ __forceinline__ void dmma1688(double *d, const double *a, const double *b) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// ---- the standalone products --------------------------------------------------------------
// Loaders return the address of an operand element, or null outside the operand (zero): the tile
// kernels copy 16-byte elements global -> shared with cp.async (zero-filled where null).
// A(m, k) = p[m * ld + k] (row-major, k contiguous)
struct LdRowK {
    static constexpr bool KC = true;
    const double2 *p;
    long ld;
    int rows, cols;
    __device__ __forceinline__ const double2 *at(int m, int k) const {
        return (m < rows && k < cols) ? p + (long)m * ld + k : nullptr;
    }
};
// B(k, n) = p[k * ld + n] (row-major, n contiguous), read as at(n, k)
struct LdRowN {
    static constexpr bool KC = false;
    const double2 *p;
    long ld;
    int rows, cols;  // rows = K extent, cols = N extent
    __device__ __forceinline__ const double2 *at(int n, int k) const {
        return (n < cols && k < rows) ? p + (long)k * ld + n : nullptr;
    }
};
// Stores of a GEMM tile: accumulates() tells whether C's old value takes part, load(r, c) reads
// it (zero outside C), combine(old, v) forms the new value and store(r, c, x) writes it inside C.
// C[r][c] = alpha v (+ C[r][c] when accumulate), r < rows, c < cols
struct StRow {
    double2 *p;
    long ld;
    int rows, cols;
    double alpha;
    int accumulate;
    __device__ __forceinline__ bool accumulates() const { return accumulate != 0; }
    __device__ __forceinline__ double2 load(int r, int c) const {
        return (r < rows && c < cols) ? p[(long)r * ld + c] : cmk(0, 0);
    }
    __device__ __forceinline__ double2 combine(double2 old, double2 v) const { return cadd(old, cscale(v, alpha)); }
    __device__ __forceinline__ void store(int r, int c, double2 x) const {
        if (r < rows && c < cols) p[(long)r * ld + c] = x;
    }
};

// Shared-memory placement of one operand tile of a stage, R rows (m or n) x BK complex k: k-major
// rows of stride BK + 4 when consecutive k are adjacent in memory (KC), else n-major rows of
// stride R + 2.  Both strides make the 8 lanes of a 16-byte access phase (2 rows x 4 k) hit eight
// different bank groups, and the copies of consecutive threads land side by side.
template <int R, bool KC> struct ZgTile {
    static constexpr int total = KC ? R * (zg::BK + 4) : zg::BK * (R + 2);
    static __device__ __forceinline__ int at(int r, int k) { return KC ? r * (zg::BK + 4) + k : k * (R + 2) + r; }
};
namespace zg {
constexpr int STAGES = 3;
template <int BM, int BN, class LA, class LB> struct Pipe {
    static constexpr int stage = ZgTile<BM, LA::KC>::total + ZgTile<BN, LB::KC>::total;
    static constexpr int total = STAGES * stage;
};
}  // namespace zg

__device__ __forceinline__ void cp16(double2 *dst, const double2 *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int bytes = src ? 16 : 0;  // 0: the 16 bytes are zero-filled and nothing is read
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src ? src : dst), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// C tile (m0.., n0..) = A B over k = 0..K-1 by the 128 threads of a CTA: 2 x 2 warps of
// (16 MT) x (8 NT), operands through a ring of three cp.async stages of 8 k (one barrier per stage).
// Used with 32 x 32 tiles, four CTAs per SM, for short K (the last factor): 900 x 512 x 128 19.0
// TFLOP/s, the k-split form 17.5; 400 x 1024 x 128 20.2 against 16.9.  Larger tiles leave too few
// CTAs (64 x 64: 15.6 TFLOP/s on 400 x 1024 x 128).
template <int BM, int BN, class LA, class LB, class PUT>
__device__ __forceinline__ void zgemm_pipe(const LA &la, const LB &lb, const PUT &put, int m0, int n0, int K,
                                           double2 *sm) {
    using namespace zg;
    constexpr int MT = BM / 32, NT = BN / 16, AE = BM * BK / NTH, BE = BN * BK / NTH;
    using TA = ZgTile<BM, LA::KC>;
    using TB = ZgTile<BN, LB::KC>;
    constexpr int SG = Pipe<BM, BN, LA, LB>::stage;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, wm = (warp >> 1) * (16 * MT), wn = (warp & 1) * (8 * NT);
    const int g = lane >> 2, q = lane & 3;
    double acc[MT][NT][2][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[i][j][c][e] = 0.0;
    const int nk = (K + BK - 1) / BK;
    auto fill = [&](int kt) {
        if (kt < nk) {
            double2 *As = sm + (kt % STAGES) * SG, *Bs = As + TA::total;
#pragma unroll
            for (int i = 0; i < AE; i++) {
                const int idx = t + NTH * i;
                const int m = LA::KC ? idx / BK : idx % BM, k = LA::KC ? idx % BK : idx / BM;
                cp16(As + TA::at(m, k), la.at(m0 + m, kt * BK + k));
            }
#pragma unroll
            for (int i = 0; i < BE; i++) {
                const int idx = t + NTH * i;
                const int n = LB::KC ? idx / BK : idx % BN, k = LB::KC ? idx % BK : idx / BN;
                cp16(Bs + TB::at(n, k), lb.at(n0 + n, kt * BK + k));
            }
        }
        cp_commit();  // an empty group past the end keeps the count of the waits
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) fill(s);
    for (int kt = 0; kt < nk; kt++) {
        cp_wait<STAGES - 2>();
        __syncthreads();  // stage kt is complete, and every warp is done with stage kt - 1
        fill(kt + STAGES - 1);
        const double2 *As = sm + (kt % STAGES) * SG, *Bs = As + TA::total;
        double br[NT][2], bi[NT][2];
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int v = 0; v < 2; v++) {
                const double2 x = Bs[TB::at(wn + j * 8 + g, q + 4 * v)];
                br[j][v] = x.x;
                bi[j][v] = x.y;
            }
#pragma unroll
        for (int i = 0; i < MT; i++) {
            double ar[4], ai[4], an[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const double2 x = As[TA::at(wm + i * 16 + g + 8 * (v & 1), q + 4 * (v >> 1))];
                ar[v] = x.x;
                ai[v] = x.y;
                an[v] = -x.y;
            }
#pragma unroll
            for (int j = 0; j < NT; j++) {
                dmma1688(acc[i][j][0], ar, br[j]);
                dmma1688(acc[i][j][1], ar, bi[j]);
            }
#pragma unroll
            for (int j = 0; j < NT; j++) {
                dmma1688(acc[i][j][0], an, bi[j]);
                dmma1688(acc[i][j][1], ai, br[j]);
            }
        }
    }
    // epilogue: an accumulating store first reads the old values of a fragment row (independent
    // loads), then writes the sums
#pragma unroll
    for (int i = 0; i < MT; i++) {
        double2 old[NT][4];
        if (put.accumulates()) {
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    old[j][e] = put.load(m0 + wm + i * 16 + g + 8 * (e >> 1), n0 + wn + j * 8 + 2 * q + (e & 1));
        }
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const double2 v = cmk(acc[i][j][0][e], acc[i][j][1][e]);
                put.store(m0 + wm + i * 16 + g + 8 * (e >> 1), n0 + wn + j * 8 + 2 * q + (e & 1),
                          put.combine(put.accumulates() ? old[j][e] : cmk(0, 0), v));
            }
    }
}

// k-split products: a CTA of 8 warps computes a 32 x 8 tile, the k steps dealt to the warps and
// summed in warp order; operands straight from L1 / L2 into the fragments.  Grid (ceil(N / 8),
// ceil(M / 32)); two CTAs per SM (128 registers: with one CTA 812 us for 2002 x 512 x 2002, with three
// 687, with two 521).  Bound: the FP64 tensor pipe (16 warps per SM, each with two k steps of loads in
// flight), and for few tiles the K / 64 dependent rounds of loads of a warp.  Measured alone on a
// B200, complex M x N x K (8 flops each): 4804 x 128 x 4804 31.5 TFLOP/s (32 x 32 tiles through
// shared memory 25.4, 64 x 64 17.5: too few tiles, uneven last wave), 2002 x 512 x 2002 31.5
// (30.6, 29.0), 1002 x 64 x 1002 25 us (54, 172 us), 401 x 1 x 401 8.5 us (25, 72 us).
template <class LA, class LB, class PUT>
__device__ __forceinline__ void zgemm_split(const LA &la, const LB &lb, const PUT &put, int m0, int n0, int K,
                                            double2 *red) {
    constexpr int NT = 1, BN = 8 * NT;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, q = lane & 3;
    double acc[2][NT][2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[i][j][c][e] = 0.0;
    // Ordinary loads (ld.global.ca): a chained kernel is resident while its predecessor writes these
    // operands, and the read-only path (ld.global.nc) may only be used for data nobody writes while the
    // kernel lives.  __ldca and not *p: the pointers come out of a table, so that *p is a generic load
    // (step of one problem, n 200: 117.6 us, with __ldca 113.7, with read-only loads 114.1).
    auto ld = [](const double2 *p) { return p ? __ldca(p) : cmk(0, 0); };
#pragma unroll 2
    for (int k0 = warp * 8; k0 < K; k0 += 64) {
        double2 a[2][4], b[NT][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int v = 0; v < 4; v++) a[i][v] = ld(la.at(m0 + i * 16 + g + 8 * (v & 1), k0 + q + 4 * (v >> 1)));
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int v = 0; v < 2; v++) b[j][v] = ld(lb.at(n0 + j * 8 + g, k0 + q + 4 * v));
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const double ar[4] = {a[i][0].x, a[i][1].x, a[i][2].x, a[i][3].x};
            const double ai[4] = {a[i][0].y, a[i][1].y, a[i][2].y, a[i][3].y};
            const double an[4] = {-ai[0], -ai[1], -ai[2], -ai[3]};
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const double br[2] = {b[j][0].x, b[j][1].x}, bi[2] = {b[j][0].y, b[j][1].y};
                dmma1688(acc[i][j][0], ar, br);
                dmma1688(acc[i][j][1], ar, bi);
                dmma1688(acc[i][j][0], an, bi);
                dmma1688(acc[i][j][1], ai, br);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                red[(warp * 32 + i * 16 + g + 8 * (e >> 1)) * BN + j * 8 + 2 * q + (e & 1)] =
                    cmk(acc[i][j][0][e], acc[i][j][1][e]);
    __syncthreads();
#pragma unroll
    for (int x = t; x < 32 * BN; x += 256) {
        double2 v = red[x];
#pragma unroll
        for (int w = 1; w < 8; w++) v = cadd(v, red[w * 32 * BN + x]);
        const int r = m0 + x / BN, c = n0 + x % BN;
        put.store(r, c, put.combine(put.accumulates() ? put.load(r, c) : cmk(0, 0), v));
    }
}
