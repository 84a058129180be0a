// Volterra recursions of one Dyson / VIE2 time step for all problems of a Sigma group, as a blocked
// triangular solve: a diagonal kernel per block of 128 scalar rows, and one GEMM that carries the
// block into every later row.
//
//   ret  G^R(n, j), j = n-k-1 .. 0     dyson_impl :158-213, vie2_impl :60-140
//        x(j) M_j = h sum_{m>j} w(n-j, n-m) x(m) Sigma^R(m, j) - bdf(j)        (Dyson)
//        x(j) M_j = Q(n, j) - h sum_{m>j} w(n-j, n-m) x(m) Fcc^R(m, j)          (VIE2)
//   les  G^<(j, n), j = k+1 .. n       dyson_impl :983-1011, vie2_impl :847-990
//        M_j x(j) = gl(j) + h sum_{m<j} w(j, m) Sigma^R(j, m) x(m) - bdf(j)     (Dyson)
//        M_j x(j) = gl(j) + Q^<(j, n) - h sum_{m<j} w(j, m) F^R(j, m) x(m)      (VIE2)
//
// Both are written as one recursion in the solve order i = k+1 .. n (les: i = j; ret: i = n - j):
//   Y_i = D_i [ q_i + g h sum_{l<i} w(i, l) T(i, l) Y_l - sum_{p<=k+1} (i/h) bd_p Y_{i-p} ]
// with s x s blocks Y_i = x(i), T(i, l) = Sigma^R(i, l), D_i = M_i^-1 for les, and the transposes
// Y_i = x(n-i)^T, T(i, l) = Sigma^R(n-l, n-i)^T, D_i = (M_{n-i}^-1)^T for ret (g = +1; VIE2: g = -1
// and no bdf).  The columns of Y_i are independent: a group of P problems is a triangular system
// with P s right-hand sides whose off-diagonal part is shared and whose D_i are the problems' own.
//
// For i > k the Gregory weight is w(i, l) = a_l + a_{i-l} - 1 with a_j = omega_j (j <= k) or 1
// (integration.hpp:382-390, and the overlap rows k < i < 2k+2 below it).  So in the far field
// (i - l > k) it is a_l, a factor of the column l, and the block's contribution to all later rows
// is ONE complex GEMM over the group's columns (k_vol_trail, on the FP64 tensor cores) with the
// columns stored as a_l Y_l (`vy`); the k rows next to a block get (a_{i-l} - 1) T(i, l) Y_l added
// by the next diagonal kernel, which also adds the backward differences across the block edge.
//
// k_vol_block, one launch per block: the CTA stages the block's triangle g h a_{i-l} T(i, l) (128
// scalar rows, 130 KB) and the step inverses in shared memory; then one warp per column (p, d)
// solves the 128 rows right-looking from registers: a lane holds 4 scalar rows (lane + 32 t), and
// after a time row is solved every lane folds it into its own rows.  Per time row the critical path
// is the solve with D_l, the broadcast and the update of the next row.  128 scalar rows: the widest
// triangle that fits in shared memory, so that a step of n rows is n s / 128 launch pairs.
//
// Measured (ret + les of a step, ms; before = the best of the one-problem, multi-problem, cluster
// and whole-GPU forms that this replaces, which solved blocks of 8-32 rows and either kept a whole
// recursion on one SM or met at a barrier of all SMs 2 n s / 32 times): size1 2, 256 problems,
// n 1000: 3.4 (with the tv stream beside the retarded half), before 5.3; size1 4, 32 problems,
// n 1200: 5.7, before 13.2; sizes 1-8, 96 problems, n 600: 12.8, before 31; size1 2, 32 problems,
// n 500 (VIE2): 0.63, before 1.27; size1 1, one problem, n 200: 0.13, before 0.14.
#pragma once
#include "kernels_gemm.cuh"

#define NESSI_GSEL 64  // groups per launch
// The groups of a launch (blockIdx.z, or .y): index into the batch's group table, active problems
struct GroupSel {
    int ng;
    int gid[NESSI_GSEL], nact[NESSI_GSEL];
};

template <int S> struct VbCfg {
    static constexpr int NBT = 128 / S;              // time rows per block
    static constexpr int NR = NBT * S;               // scalar rows, at most 128
    static constexpr int NRP = NR | 1;               // odd stride of a column buffer
    static constexpr int TRI = S * S * (NBT * (NBT - 1) / 2);
    static constexpr int NEAR = NESSI_K1MAX * S;     // rows next to the block above, and their sources
    static constexpr int WMAX = 8;                   // columns (chain warps) per CTA
    static constexpr int SLOTS = (WMAX - 1 + S - 1) / S + 1;  // problems those columns can touch
    // shared memory in double2: triangle, near block, near values, step inverses, columns, q of a row
    static constexpr int near_ = TRI, ynear = near_ + NEAR * NEAR, dm = ynear + WMAX * NEAR, buf = dm + SLOTS * NR * S,
                         qs = buf + WMAX * NRP, total = qs + WMAX * S;
    static_assert(total * 16 <= 227 * 1024, "one CTA per SM");
    // packed column-major triangle: column l (s scalar columns) holds rows (l+1) s .. NR-1
    static __device__ __forceinline__ int off(int l) { return S * (l * NR - S * (l * (l + 1) / 2)); }
};

// T(i, l)[a][b]
template <int S, bool RET>
__device__ __forceinline__ const double2 *vol_t(const GroupDev &g, int n, int i, int l, int a, int b) {
    return RET ? g.rret + (tri(n - l) + n - i) * (S * S) + b * S + a : g.sret + (tri(i) + l) * (S * S) + a * S + b;
}
__device__ __forceinline__ double2 shfl2(double2 x, int src) {
    return cmk(__shfl_sync(0xffffffffu, x.x, src), __shfl_sync(0xffffffffu, x.y, src));
}
// acc - (i b) x
__device__ __forceinline__ double2 sub_ib(double2 acc, double b, double2 x) {
    return cmk(fma(b, x.y, acc.x), fma(-b, x.x, acc.y));
}

// One column of a block, solved by a warp: acc[t] = right-hand side of scalar row lane + 32 t on
// entry.  xs (shared, NR): the solved rows on exit.  bdx[delta] = bd / h for delta <= k+1, else 0.
template <int S, bool VIE>
__device__ __forceinline__ void vol_chain(double2 *acc, const double2 *coef, const double2 *D, const double *bdx, int K1,
                                          int nb, double2 *xs, double2 *qs, int lane) {
    using C = VbCfg<S>;
    if constexpr (S == 1) {
        double2 Dr[4];
#pragma unroll
        for (int t = 0; t < 4; t++) Dr[t] = lane + 32 * t < nb ? D[lane + 32 * t] : cmk(0, 0);
#pragma unroll
        for (int ph = 0; ph < 4; ph++) {
            const int lend = min(nb, 32 * ph + 32);
            for (int l = 32 * ph; l < lend; l++) {
                const int ll = l - 32 * ph;
                const double2 *cl = coef + C::off(l) - (l + 1);
                double2 cv[4];
#pragma unroll
                for (int t = ph; t < 4; t++) cv[t] = (t > ph || lane > ll) ? cl[lane + 32 * t] : cmk(0, 0);
                const double b0 = lane > ll ? bdx[lane - ll] : 0.0;
                const double2 x = shfl2(cmul(Dr[ph], acc[ph]), ll);
                if (lane > ll) {
                    acc[ph] = cfma(cv[ph], x, acc[ph]);
                    if (!VIE) acc[ph] = sub_ib(acc[ph], b0, x);
                }
                if (lane == ll) acc[ph] = x;
#pragma unroll
                for (int t = ph + 1; t < 4; t++) {
                    acc[t] = cfma(cv[t], x, acc[t]);
                    if (!VIE && t == ph + 1 && ll + K1 >= 32) acc[t] = sub_ib(acc[t], bdx[lane + 32 * t - l], x);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (lane + 32 * t < nb) xs[lane + 32 * t] = acc[t];
    } else if constexpr (S == 2) {
#pragma unroll
        for (int ph = 0; ph < 4; ph++) {
            const int lend = min(nb, 16 * ph + 16);
            for (int l = 16 * ph; l < lend; l++) {
                const int src = 2 * (l - 16 * ph), len = C::NR - 2 * (l + 1);
                const double2 *c0 = coef + C::off(l) - 2 * (l + 1), *c1 = c0 + len;
                double2 u[4], v[4];
#pragma unroll
                for (int t = ph; t < 4; t++) {
                    const bool in = t > ph || lane > src + 1;
                    u[t] = in ? c0[lane + 32 * t] : cmk(0, 0);
                    v[t] = in ? c1[lane + 32 * t] : cmk(0, 0);
                }
                const double2 d00 = D[l * 4], d01 = D[l * 4 + 1], d10 = D[l * 4 + 2], d11 = D[l * 4 + 3];
                const double b0 = lane > src + 1 ? bdx[(lane >> 1) - (l - 16 * ph)] : 0.0;
                const double2 q0 = shfl2(acc[ph], src), q1 = shfl2(acc[ph], src + 1);
                const double2 x0 = cfma(d01, q1, cmul(d00, q0)), x1 = cfma(d11, q1, cmul(d10, q0));
                const double2 xa = (lane & 1) ? x1 : x0;
                if (lane > src + 1) {
                    acc[ph] = cfma(v[ph], x1, cfma(u[ph], x0, acc[ph]));
                    if (!VIE) acc[ph] = sub_ib(acc[ph], b0, xa);
                }
                if ((lane & ~1) == src) acc[ph] = xa;
#pragma unroll
                for (int t = ph + 1; t < 4; t++) {
                    acc[t] = cfma(v[t], x1, cfma(u[t], x0, acc[t]));
                    if (!VIE && t == ph + 1 && src / 2 + K1 >= 16)
                        acc[t] = sub_ib(acc[t], bdx[((lane + 32 * t) >> 1) - l], xa);
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (lane + 32 * t < 2 * nb) xs[lane + 32 * t] = acc[t];
    } else {
        for (int l = 0; l < nb; l++) {
            const int r0 = l * S, r1 = r0 + S, len = C::NR - r1;
            // the row's right-hand side to shared memory, x = D_l q by lanes 0..s-1, then all lanes
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int r = lane + 32 * t;
                if (r >= r0 && r < r1) qs[r - r0] = acc[t];
            }
            __syncwarp();
            if (lane < S) {
                const double2 *dl = D + l * S * S + lane * S;
                double2 xe = cmk(0, 0), xo = cmk(0, 0);
#pragma unroll
                for (int b = 0; b < S; b += 2) xe = cfma(dl[b], qs[b], xe);
#pragma unroll
                for (int b = 1; b < S; b += 2) xo = cfma(dl[b], qs[b], xo);
                xs[r0 + lane] = cadd(xe, xo);
            }
            __syncwarp();
            double2 x[S];
#pragma unroll
            for (int b = 0; b < S; b++) x[b] = xs[r0 + b];
            const double2 *cl = coef + C::off(l) - r1;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                if (32 * t + 31 < r1 || 32 * t >= C::NR) continue;  // no row of this slot is left
                const int r = lane + 32 * t;
                if (r >= r1 && r < C::NR) {
                    double2 e = cmk(0, 0);
#pragma unroll
                    for (int b = 0; b < S; b += 2) acc[t] = cfma(cl[b * len + r], x[b], acc[t]);
#pragma unroll
                    for (int b = 1; b < S; b += 2) e = cfma(cl[b * len + r], x[b], e);
                    acc[t] = cadd(acc[t], e);
                    if (!VIE && r < r1 + K1 * S) acc[t] = sub_ib(acc[t], bdx[r / S - l], xs[r0 + r % S]);
                }
            }
        }
    }
}

// Grid (ceil(columns / wc), groups), 256 threads; wc = 1, 2, 4 or 8 columns per CTA.
template <int S, bool VIE, bool RET>
__global__ void __launch_bounds__(256) k_vol_block(const GroupDev *__restrict__ gt, GroupSel sel, int n, int blk, int wc) {
    extern __shared__ double2 smem[];
    using C = VbCfg<S>;
    constexpr int s2 = S * S, NR = C::NR;
    __shared__ double bdx[C::NBT + 1], wdx[C::NBT + 1];  // bd(delta) / h (0 beyond k+1), a_delta
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const int cols = sel.nact[blockIdx.y] * S, c0 = (int)blockIdx.x * wc;
    const int k = g.k, K1 = k + 1, i0 = K1 + blk * C::NBT, nb = min(C::NBT, n - i0 + 1);
    if (c0 >= cols || nb <= 0) return;
    const int ncol = min(wc, cols - c0), NRb = nb * S, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lw = wc == 8 ? 3 : (wc == 4 ? 2 : (wc == 2 ? 1 : 0)), p0 = c0 / S;
    const double h = g.h, gh = VIE ? -h : h;
    const long ldc = g.ldc;
    const ProbDev *probs = g.probs;
    double2 *coef = smem, *near_ = smem + C::near_, *ynear = smem + C::ynear, *dm = smem + C::dm, *buf = smem + C::buf;
    for (int e = tid; e <= C::NBT; e += 256) {
        bdx[e] = e <= K1 ? bd_w(k, e) / h : 0.0;
        wdx[e] = e <= k ? greg_omega(k, e) : 1.0;
    }
    __syncthreads();
    // ---- operands that do not depend on the solution: triangle, near block, step inverses
    if (RET) {  // memory is contiguous along the rows of a column
        for (int l = warp; l < nb - 1; l += 8)
            for (int b = 0; b < S; b++) {
                double2 v[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int r = (l + 1) * S + lane + 32 * t;
                    if (r < NRb) v[t] = *vol_t<S, RET>(g, n, i0 + r / S, i0 + l, r % S, b);
                }
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int x = lane + 32 * t, r = (l + 1) * S + x;
                    if (r < NRb) coef[C::off(l) + b * (NR - (l + 1) * S) + x] = cscale(v[t], gh * wdx[r / S - l]);
                }
            }
    } else {  // memory is contiguous along the columns of a row
        for (int r = S + warp; r < NRb; r += 8) {
            const int rt = r / S, a = r % S;
            double2 v[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int x = lane + 32 * t;
                if (x < rt * S) v[t] = *vol_t<S, RET>(g, n, i0 + rt, i0 + x / S, a, x % S);
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int x = lane + 32 * t, l = x / S, b = x % S;
                if (x < rt * S) coef[C::off(l) + b * (NR - (l + 1) * S) + r - (l + 1) * S] = cscale(v[t], gh * wdx[rt - l]);
            }
        }
    }
    if (blk > 0)
        for (int e = tid; e < K1 * S * K1 * S; e += 256) {
            const int x = RET ? e / (K1 * S) : e % (K1 * S), r = RET ? e % (K1 * S) : e / (K1 * S);
            const int rt = r / S, l = x / S, delta = rt + K1 - l;
            double2 v = cmk(0, 0);
            if (r < NRb && delta <= k)
                v = cscale(*vol_t<S, RET>(g, n, i0 + rt, i0 - K1 + l, r % S, x % S), gh * (wdx[delta] - 1.0));
            near_[x * C::NEAR + r] = v;
        }
    for (int q = p0; q <= (c0 + ncol - 1) / S; q++) {
        const double2 *mi = RET ? probs[q].minv_ret : probs[q].minv_les;
        for (int e = tid; e < nb * s2; e += 256) {
            const int l = e / s2, a = (e % s2) / S, b = e % S;
            dm[(q - p0) * NR * S + (RET ? l * s2 + b * S + a : e)] = mi[(long)(RET ? n - i0 - l : i0 + l) * s2 + a * S + b];
        }
    }
    // ---- right-hand sides: q_i + g h (far sum of the blocks above)
    for (int e = tid; e < NRb << lw; e += 256) {
        const int w = e & (wc - 1), r = e >> lw, i = i0 + r / S, a = r % S, c = c0 + w;
        if (w >= ncol) continue;
        double2 v = cmk(0, 0);
        if (!RET) v = __ldcg(g.gles + ((long)i * S + a) * ldc + c);
        if (VIE) {
            const ProbDev &p = probs[c / S];
            v = cadd(v, RET ? p.qret[(tri(n) + n - i) * s2 + (c % S) * S + a] : p.qles[(tri(n) + i) * s2 + a * S + c % S]);
        }
        if (blk > 0) {
            const double2 far = __ldcg(g.vacc + ((long)i * S + a) * ldc + c);
            v = cmk(fma(gh, far.x, v.x), fma(gh, far.y, v.y));
        }
        buf[w * C::NRP + r] = v;
    }
    if (blk > 0)
        for (int e = tid; e < (K1 * S) << lw; e += 256) {
            const int w = e & (wc - 1), x = e >> lw;
            if (w < ncol) ynear[w * C::NEAR + x] = __ldcg(g.vy + ((long)(i0 - K1) * S + x) * ldc + c0 + w);
        }
    __syncthreads();
    if (warp < ncol) {
        const int c = c0 + warp, d = c % S;
        double2 *xs = buf + warp * C::NRP;
        double2 acc[4];
#pragma unroll
        for (int t = 0; t < 4; t++) acc[t] = lane + 32 * t < NRb ? xs[lane + 32 * t] : cmk(0, 0);
        __syncwarp();
        if (blk > 0) {
            const double2 *y = ynear + warp * C::NEAR;
#pragma unroll
            for (int t = 0; t < (C::NEAR + 31) / 32; t++) {
                const int r = lane + 32 * t;
                if (r >= K1 * S || r >= NRb) continue;
                for (int x = (r / S) * S; x < K1 * S; x++) acc[t] = cfma(near_[x * C::NEAR + r], y[x], acc[t]);
                if (!VIE)
                    for (int l = r / S; l < K1; l++) acc[t] = sub_ib(acc[t], bdx[r / S + K1 - l], y[l * S + r % S]);
            }
        } else {
            // the start rows 0..k with exact weights
            const ProbDev &p = probs[c / S];
            for (int l = 0; l <= k; l++) {
                double2 y[S];
#pragma unroll
                for (int b = 0; b < S; b++)
                    y[b] = RET ? p.gret[(tri(n) + n - l) * s2 + d * S + b] : p.gles[(tri(n) + l) * s2 + b * S + d];
                const double al = greg_omega(k, l);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int r = lane + 32 * t, i = i0 + r / S, a = r % S, delta = i - l;
                    if (r >= NRb) continue;
                    const double w = gh * (al + (delta <= k ? greg_omega(k, delta) : 1.0) - 1.0);
                    double2 e = cmk(0, 0);
#pragma unroll
                    for (int b = 0; b < S; b++) e = cfma(*vol_t<S, RET>(g, n, i, l, a, b), y[b], e);
                    acc[t] = cmk(fma(w, e.x, acc[t].x), fma(w, e.y, acc[t].y));
                    if (!VIE && delta <= K1) {
                        double2 ya = y[0];
#pragma unroll
                        for (int b = 1; b < S; b++) ya = a == b ? y[b] : ya;
                        acc[t] = sub_ib(acc[t], bd_w(k, delta) / h, ya);
                    }
                }
            }
        }
        vol_chain<S, VIE>(acc, coef, dm + (c / S - p0) * NR * S, bdx, K1, nb, xs, smem + C::qs + warp * S, lane);
    }
    __syncthreads();
    // ---- results: vy (rows x columns, for the trailing GEMM), ret: the operand of les*adv
    //      badv(m) = h w(n, m) G^R(n, m)^dagger, and G's own row / column
    const bool more = i0 + nb <= n;
    for (int e = tid; e < NRb << lw; e += 256) {
        const int w = e & (wc - 1), r = e >> lw, i = i0 + r / S, a = r % S;
        if (w >= ncol) continue;
        const double2 x = buf[w * C::NRP + r];
        if (more) g.vy[((long)i * S + a) * ldc + c0 + w] = x;
        if (RET) g.badv[((long)(n - i) * S + a) * ldc + c0 + w] = cscale(cconj(x), h * greg_w(k, n, n - i));
    }
    for (int w = warp; w < ncol; w += 8) {
        const int c = c0 + w, d = c % S;
        double2 *out = RET ? probs[c / S].gret + tri(n) * s2 : probs[c / S].gles + tri(n) * s2;
        for (int r = lane; r < NRb; r += 32) {
            const int i = i0 + r / S, a = r % S;
            out[RET ? (long)(n - i) * s2 + d * S + a : (long)i * s2 + a * S + d] = buf[w * C::NRP + r];
        }
    }
}

// ---- trailing update: vacc(i, .) (+)= sum_l T(i, l) vy(l, .) for all rows i after the block -------
template <int S, bool RET> struct LdVolT {
    static constexpr bool KC = !RET;  // les: contiguous in l; ret: contiguous in i
    const double2 *t;
    int n, i1, l0, M, K;
    __device__ __forceinline__ const double2 *at(int r, int kk) const {
        if (r >= M || kk >= K) return nullptr;
        const int i = i1 + r / S, a = r % S, l = l0 + kk / S, b = kk % S;
        return RET ? t + (tri(n - l) + n - i) * (S * S) + b * S + a : t + (tri(i) + l) * (S * S) + a * S + b;
    }
};
template <int S, bool RET>
__device__ __forceinline__ bool vol_trail_operands(const GroupDev &g, int cols, int n, int blk, LdVolT<S, RET> &la,
                                                   LdRowN &lb, StRow &st, int &K) {
    using C = VbCfg<S>;
    const int i0 = g.k + 1 + blk * C::NBT, i1 = i0 + C::NBT, l0 = blk == 0 ? 0 : i0;
    const int M = (n - i1 + 1) * S;
    K = (i1 - l0) * S;
    la = LdVolT<S, RET>{RET ? g.rret : g.sret, n, i1, l0, M, K};
    lb = LdRowN{g.vy + (long)l0 * S * g.ldc, g.ldc, K, cols};
    st = StRow{g.vacc + (long)i1 * S * g.ldc, g.ldc, M, cols, 1.0, blk > 0};
    return M > 0;
}
// Grid (column tiles, row tiles, groups)
template <int S, bool RET>
__global__ void __launch_bounds__(128, 4) k_vol_trail(const GroupDev *__restrict__ gt, GroupSel sel, int n, int blk) {
    extern __shared__ double2 smem[];
    const GroupDev &g = gt[sel.gid[blockIdx.z]];
    const int cols = sel.nact[blockIdx.z] * S;
    LdVolT<S, RET> la;
    LdRowN lb;
    StRow st;
    int K;
    if (!vol_trail_operands<S, RET>(g, cols, n, blk, la, lb, st, K)) return;
    if ((int)blockIdx.x * 32 >= cols || (int)blockIdx.y * 32 >= la.M) return;
    zgemm_pipe<32, 32>(la, lb, st, blockIdx.y * 32, blockIdx.x * 32, K, smem);
}
template <int S, bool RET>
__global__ void __launch_bounds__(256) k_vol_trail_split(const GroupDev *__restrict__ gt, GroupSel sel, int n, int blk) {
    __shared__ double2 red[8 * 32 * 8];
    const GroupDev &g = gt[sel.gid[blockIdx.z]];
    const int cols = sel.nact[blockIdx.z] * S;
    LdVolT<S, RET> la;
    LdRowN lb;
    StRow st;
    int K;
    if (!vol_trail_operands<S, RET>(g, cols, n, blk, la, lb, st, K)) return;
    if ((int)blockIdx.x * 8 >= cols || (int)blockIdx.y * 32 >= la.M) return;
    zgemm_split(la, lb, st, blockIdx.y * 32, blockIdx.x * 8, K, red);
}

// ---- start rows i = 0..k, one CTA per problem (grid (problems, groups)) --------------------------
// ret: G(n, n) = -i (Dyson) or Q(n, n) (VIE2), then the k-block start G(n, n-1..n-k)
// (dyson_impl :112-157, vie2_impl :60-100)
template <int S, bool VIE>
__global__ void __launch_bounds__(256) k_ret_start(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    extern __shared__ double2 smem[];
    constexpr int s2 = S * S;
    if ((int)blockIdx.x >= sel.nact[blockIdx.y]) return;
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const ProbDev p = g.probs[blockIdx.x];
    const int k = g.k;
    const long ldc = g.ldc;
    double2 *grow = p.gret + tri(n) * s2;
    for (int e = threadIdx.x; e < s2; e += blockDim.x)
        grow[(long)n * s2 + e] = VIE ? p.qret[(tri(n) + n) * s2 + e] : (e / S == e % S ? cmk(0.0, -1.0) : cmk(0, 0));
    __syncthreads();
    if (VIE) ret_start_block_vie<S>(g, p, n, smem);
    else ret_start_block<S>(g, p, n, smem);
    __syncthreads();
    for (int e = threadIdx.x; e < (k + 1) * s2; e += blockDim.x) {
        const int l = e / s2, b = (e % s2) / S, d = e % S;  // Y_l[b][d] = G(n, n-l)[d][b]
        const double2 y = grow[(long)(n - l) * s2 + d * S + b];
        g.vy[((long)l * S + b) * ldc + p.col * S + d] = cscale(y, greg_omega(k, l));
        g.badv[((long)(n - l) * S + b) * ldc + p.col * S + d] = cscale(cconj(y), g.h * greg_w(k, n, n - l));
    }
}

// les: G^<(0, n) = -G^tv(n, 0)^dagger and the k-block start G^<(1..k, n) (dyson_impl :926-982), or
// the VIE2 start G^<(0..k, n) (vie2_impl :847-900); gl = the Sigma-shared products in g.gles.
template <int S, bool VIE>
__global__ void __launch_bounds__(256) k_les_start(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    extern __shared__ double2 smem[];
    constexpr int s2 = S * S;
    if ((int)blockIdx.x >= sel.nact[blockIdx.y]) return;
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const ProbDev p = g.probs[blockIdx.x];
    const int k = g.k;
    const long ldc = g.ldc;
    const double2 *gl = g.gles + (long)p.col * S;
    double2 *xcol = p.gles + tri(n) * s2;
    if (VIE) {
        les_start_block_vie<S>(g, p, n, gl, ldc, xcol, smem);
    } else {
        for (int ad = threadIdx.x; ad < s2; ad += blockDim.x) {
            const int a = ad / S, d = ad % S;
            xcol[ad] = cneg(cconj(p.gtv[((long)n * s2 + d * S + a) * (g.ntau + 1) + 0]));
        }
        __syncthreads();
        les_start_block<S>(g, p, n, gl, ldc, xcol, smem);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < (k + 1) * s2; e += blockDim.x) {
        const int l = e / s2, b = (e % s2) / S, d = e % S;
        g.vy[((long)l * S + b) * ldc + p.col * S + d] = cscale(xcol[e], greg_omega(k, l));
    }
}
