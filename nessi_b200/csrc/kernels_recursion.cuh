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
// columns stored as a_l Y_l (`vy`; the start rows 0..k first); the k rows next to a block get
// (a_{i-l} - 1) T(i, l) Y_l added by the next diagonal kernel, which also adds the backward
// differences across the block edge.
//
// k_vol_block, one launch per block: the CTA stages the block's triangle a_{i-l} T(i, l) (128
// scalar rows, 130 KB) and the step inverses in shared memory with asynchronous copies; then a warp
// (s >= 3: four warps, a slot of 32 rows each) solves a column (s = 2: two) (p, d), 128 rows
// right-looking from registers: a lane holds scalar rows lane + 32 t of a column, and after a time
// row is solved every lane folds it into its own rows.
// Bound: the chain of 128 / s dependent rows; per row the solve with D_l, the broadcast and the update
// of the next row (a dependent FP64 FMA takes 9 cycles, a shared-memory round trip 33), with the
// triangle's column of the next row loaded one row ahead.  Columns per warp: one for size1 1 (blocks of
// ret and les, 1024 problems, n 1000: 340 us; two that share the loads 475, their sums are longer than
// the chain).  Size1 2: two at eight columns per CTA, else one (256 problems, n 1000: 687 us, 512
// problems 1048; built for one only: 775 and 1004).
// 128 scalar rows: the widest triangle that fits in shared memory beside the tv stream's ring (size1 <= 4, see
// vol_beside_tv), so that a step of n rows is n s / 128 launch pairs.  The kernels of a recursion are launched with
// programmatic stream serialization: what does not depend on the solution (triangle, near block,
// step inverses) is staged while the previous kernel still runs.
//
// Measured on a B200, alone, ret + les of a step in us (blocks / trailing products / start rows):
// size1 1, 1024 problems, n 1000: 699 (340 / 389 / 33); size1 2, 256 problems, n 1000: 1402 (687 /
// 785 / 32); size1 4, 32 problems, n 1200: 2593 (1247 / 1450 / 64); size1 8, 18 problems, n 600: 3125
// (1275 / 1617 / 173); size1 1, one problem, n 400: 119.  Synchronous staging, without the overlap of
// launches, one warp per column for s >= 3: 957, 1842, 3774, 4175 and 238.
#pragma once
#include "kernels_dyson.cuh"

template <int S> struct VbCfg {
    static constexpr int TPS = 32 / S;               // time rows per slot (the 32 lanes of a warp)
    static constexpr int SR = TPS * S;               // scalar rows per slot
    static constexpr int NBT = 4 * TPS;              // time rows per block: four slots
    static constexpr int NR = NBT * S;               // scalar rows, at most 128
    static constexpr int NRP = NR | 1;               // odd stride of a column buffer
    static constexpr int TRI = S * S * (NBT * (NBT - 1) / 2);
    static constexpr int NEAR = NESSI_K1MAX * S;     // rows next to the block above, and their sources
    // s <= 2: a warp solves NC columns, all four slots; s >= 3: four warps per column, a slot each
    static constexpr int NTH = S <= 4 ? 256 : 512, NW = NTH / 32, WMAX = S <= 2 ? 8 : NTH / 128, NC = S == 2 ? 2 : 1;
    // shared memory in double2: 32 of padding (unpredicated loads of solved rows), triangle, near
    // block, then per column the near values, the column and (s >= 3) the row being solved, then the
    // step inverses of the problems touched
    static constexpr int coef = 32, near_ = coef + TRI, cols = near_ + NEAR * NEAR, QS = S >= 3 ? S : 0;
    static __host__ __device__ constexpr int slots(int wc) { return (wc - 1 + S - 1) / S + 1 < wc ? (wc - 1 + S - 1) / S + 1 : wc; }
    static __host__ __device__ constexpr int buf(int wc) { return cols + wc * NEAR; }
    static __host__ __device__ constexpr int qs(int wc) { return buf(wc) + wc * NRP; }
    static __host__ __device__ constexpr int dm(int wc) { return qs(wc) + wc * QS; }
    static __host__ __device__ constexpr int total(int wc) { return dm(wc) + (S == 1 ? 0 : slots(wc) * NR * S); }
    // packed column-major triangle: column l (s scalar columns) holds rows (l+1) s .. NR-1
    static __device__ __forceinline__ int off(int l) { return S * (l * NR - S * (l * (l + 1) / 2)); }
};
// Most columns per CTA with which k_vol_block and k_tv_ring share an SM (228 KB of shared memory, 1 KB of it
// reserved per CTA): 8 for size1 1 (219 KB for the pair), 4 for 2 (224; with 8 240), 2 for 3 (206), 1 for 4
// (218; with 2 228.4).  From size1 5 on the ring takes all registers of the SM and there is no limit.
// The retarded recursion keeps to it in an FP64 step with ntau >= 75 size1: with more columns a CTA its SMs wait
// for the stream's to finish, which costs more than a second wave of CTAs.  A step in ms, with the limit and
// with 8 (size1 4: 2) columns: size1 2, 310 problems, n 200, ntau 150 0.50 and 0.53; 1000, n 500, ntau 150 3.18
// and 3.35; 512, n 800, ntau 500 4.65 and 5.27; size1 4, 40 problems, n 200, ntau 300 0.70 and 0.71; 150, n 500,
// ntau 300 5.00 and 5.31; 40, n 1200, ntau 800 6.46 and 7.16.  A shorter stream has less to lose: size1 2, 310
// problems, n 900, ntau 40 2.51 and 2.41; size1 4, 45 problems, n 200, ntau 100 0.59 and 0.53.  The lesser
// recursion runs alone and has no limit (size1 2, 300 problems, n 800, ntau 500 3.08, limited too 3.19), nor has
// a mixed step, whose tv kernel does not leave room in any case (3.33 with it, 3.25 without).
template <int S> constexpr int vol_beside_tv() {
    int wc = VbCfg<S>::WMAX;
    if (S <= 4)
        while (wc > 1 && (VbCfg<S>::total(wc) + TvCfg<S>::total) * 16 + 2 * 1024 > 228 * 1024) wc /= 2;
    return wc;
}
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

// s <= 2: a column (s = 2: NC columns) of a block, solved by a warp.  acc[c][t] = right-hand side of scalar row
// lane + 32 t of column c on entry; xs (shared, stride NRP) receives the solved rows.  D: step
// inverses (s = 1: registers, rows lane + 32 t; s = 2: shared).  bdp[32 + delta] = bd / h for
// 1 <= delta <= k+1, else 0.  The accumulators of solved rows are not used again.
template <bool VIE>
__device__ __forceinline__ void vol_chain1(double2 *acc, const double2 *coef, const double2 *D, const double *bdp, double gh,
                                           int K1, int nb, double2 *xs, int lane) {
    using C = VbCfg<1>;
    const double2 *cl = coef - 1 + lane;  // column l: row lane + 32 t at cl[32 t]
    double2 cv[4];
#pragma unroll
    for (int t = 0; t < 4; t++) cv[t] = t > 0 || lane > 0 ? cl[32 * t] : cmk(0, 0);
#pragma unroll
    for (int ph = 0; ph < 4; ph++) {
        const int lend = min(32, nb - 32 * ph);
        const double *bp = bdp + 32 + lane;
#pragma unroll 2
        for (int ll = 0; ll < lend; ll++) {
            const double b0 = VIE ? 0.0 : bp[-ll], b1 = VIE ? 0.0 : bp[32 - ll];
            double2 nv[4];  // the next column of the triangle, one row ahead
            cl += C::NR - 2 - (32 * ph + ll);
#pragma unroll
            for (int t = ph; t < 4; t++) nv[t] = 32 * t + lane > 32 * ph + ll + 1 ? cl[32 * t] : cmk(0, 0);
            const double2 x = shfl2(cmul(D[ph], acc[ph]), ll), xg = cscale(x, gh);
            if (lane == ll) xs[32 * ph + ll] = x;
            double2 u = acc[ph];
            if (!VIE) u = sub_ib(u, b0, x);
            acc[ph] = cfma(cv[ph], xg, u);
#pragma unroll
            for (int t = ph + 1; t < 4; t++) {
                if (!VIE && t == ph + 1 && ll + K1 >= 32) acc[t] = sub_ib(acc[t], b1, x);
                acc[t] = cfma(cv[t], xg, acc[t]);
            }
#pragma unroll
            for (int t = ph; t < 4; t++) cv[t] = nv[t];
        }
    }
}

template <bool VIE, int NC>
__device__ __forceinline__ void vol_chain2(double2 (*acc)[4], const double2 *coef, const double2 *D, const double *bdp,
                                           double gh, int K1, int nb, double2 *xs, int lane) {
    using C = VbCfg<2>;
    const double2 *cl = coef - 2 + lane;  // column (l, 0): row lane + 32 t at cl[32 t]; (l, 1): len further
    double2 u[4], v[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        u[t] = t > 0 || lane > 1 ? cl[32 * t] : cmk(0, 0);
        v[t] = t > 0 || lane > 1 ? cl[C::NR - 2 + 32 * t] : cmk(0, 0);
    }
#pragma unroll
    for (int ph = 0; ph < 4; ph++) {
        const int lend = min(16, nb - 16 * ph);
        const double *bp = bdp + 32 + (lane >> 1);
#pragma unroll 1
        for (int ll = 0; ll < lend; ll++) {
            const int l = 16 * ph + ll, src = 2 * ll, len = C::NR - 2 * (l + 2);  // of the next column
            const double b0 = VIE ? 0.0 : bp[-ll], b1 = VIE ? 0.0 : bp[16 - ll];
            const double2 d00 = D[l * 4], d01 = D[l * 4 + 1], d10 = D[l * 4 + 2], d11 = D[l * 4 + 3];
            double2 nu[4], nv[4];
            cl += 2 * (C::NR - 2 * (l + 1)) - 2;
#pragma unroll
            for (int t = ph; t < 4; t++) {
                const bool open = 32 * t + lane > 32 * ph + src + 3;
                nu[t] = open ? cl[32 * t] : cmk(0, 0);
                nv[t] = open ? cl[len + 32 * t] : cmk(0, 0);
            }
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const double2 q0 = shfl2(acc[c][ph], src), q1 = shfl2(acc[c][ph], src + 1);
                const double2 x0 = cfma(d01, q1, cmul(d00, q0)), x1 = cfma(d11, q1, cmul(d10, q0));
                const double2 xa = (lane & 1) ? x1 : x0, g0 = cscale(x0, gh), g1 = cscale(x1, gh);
                if ((lane & ~1) == src) xs[c * C::NRP + 32 * ph + lane] = xa;
                double2 w = acc[c][ph];
                if (!VIE) w = sub_ib(w, b0, xa);
                acc[c][ph] = cfma(v[ph], g1, cfma(u[ph], g0, w));
#pragma unroll
                for (int t = ph + 1; t < 4; t++) {
                    if (!VIE && t == ph + 1 && ll + K1 >= 16) acc[c][t] = sub_ib(acc[c][t], b1, xa);
                    acc[c][t] = cfma(v[t], g1, cfma(u[t], g0, acc[c][t]));
                }
            }
#pragma unroll
            for (int t = ph; t < 4; t++) {
                u[t] = nu[t];
                v[t] = nv[t];
            }
        }
    }
}

// s >= 3: one column, solved by four warps, warp `slot` holding the SR scalar rows of its slot.  Per
// time row the warp that owns it forms x = D_l q (lanes 0..s-1, q through shared memory) and
// publishes it; one barrier of the warps still at work (named barrier `bar`), then every lane folds
// it into its row.
template <int S, bool VIE>
__device__ __forceinline__ void vol_chain_big(double2 acc, const double2 *coef, const double2 *D, const double *bdp,
                                              double gh, int nb, double2 *xs, double2 *qs, int slot, int lane, int bar) {
    using C = VbCfg<S>;
    const int row = slot * C::TPS + lane / S, ra = lane % S, r = slot * C::SR + lane;
    const bool live = lane < C::SR;
    const int lend = min(nb, (slot + 1) * C::TPS);
#pragma unroll 1
    for (int l = 0; l < lend; l++) {
        const int r0 = l * S, len = C::NR - r0 - S, own = l / C::TPS;
        const bool open = live && row > l;
        const double2 *cl = coef + C::off(l) - r0 - S + r;
        double2 cf[S];
#pragma unroll
        for (int b = 0; b < S; b++) cf[b] = open ? cl[b * len] : cmk(0, 0);
        const double bw = VIE || !open ? 0.0 : bdp[32 + min(row - l, NESSI_K1MAX + 1)];
        if (own == slot) {
            double2 dv[S];
            const double2 *dl = D + l * S * S + (lane < S ? lane : 0) * S;
#pragma unroll
            for (int b = 0; b < S; b++) dv[b] = dl[b];
            if (live && row == l) qs[ra] = acc;
            __syncwarp();
            double2 xe = cmul(dv[0], qs[0]), xo = cmul(dv[1], qs[1]);
#pragma unroll
            for (int b = 2; b < S; b += 2) xe = cfma(dv[b], qs[b], xe);
#pragma unroll
            for (int b = 3; b < S; b += 2) xo = cfma(dv[b], qs[b], xo);
            if (lane < S) xs[r0 + lane] = cadd(xe, xo);
        }
        asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(32 * (4 - own)) : "memory");
        double2 e = acc, o = cmk(0, 0);
        if (!VIE) e = sub_ib(e, bw, xs[r0 + ra]);
#pragma unroll
        for (int b = 0; b < S; b += 2) o = cfma(cf[b], cscale(xs[r0 + b], gh), o);
#pragma unroll
        for (int b = 1; b < S; b += 2) e = cfma(cf[b], cscale(xs[r0 + b], gh), e);
        if (open) acc = cadd(e, o);
    }
}

// Grid (ceil(columns / wc), groups), VbCfg<S>::NTH threads; wc = 1, 2, 4 or 8 columns per CTA (at most
// WMAX), VbCfg<S>::total(wc) complex of dynamic shared memory.
template <int S, bool VIE, bool RET>
__global__ void __launch_bounds__(VbCfg<S>::NTH, VbCfg<S>::NTH == 256 ? 2 : 1) k_vol_block(const GroupDev *__restrict__ gt, GroupSel sel, int n, int blk,
                                                             int wc) {
    extern __shared__ double2 smem[];
    using C = VbCfg<S>;
    constexpr int s2 = S * S, NR = C::NR, NTH = C::NTH;
    __shared__ double bdp[32 + C::NBT + 1], wdx[NESSI_K1MAX + 1];  // [32 + delta]: bd(delta) / h; a_delta
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const int cols = sel.nact[blockIdx.y] * S, c0 = (int)blockIdx.x * wc;
    const int k = g.k, K1 = k + 1, i0 = K1 + blk * C::NBT, nb = min(C::NBT, n - i0 + 1);
    if (c0 >= cols || nb <= 0) return;
    const int ncol = min(wc, cols - c0), NRb = nb * S, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lw = wc == 8 ? 3 : (wc == 4 ? 2 : (wc == 2 ? 1 : 0)), p0 = c0 / S;
    const int nc = wc == 8 ? C::NC : 1;  // columns per warp (s <= 2): two share the loads of the triangle
    const double h = g.h, gh = VIE ? -h : h;
    const long ldc = g.ldc;
    const ProbDev *probs = g.probs;
    double2 *coef = smem + C::coef, *near_ = smem + C::near_, *ynear = smem + C::cols, *dm = smem + C::dm(wc),
            *buf = smem + C::buf(wc);
    pdl_trigger();
    // ---- operands that do not depend on the solution, all copies in flight at once: triangle, near
    //      block, step inverses
    if (RET) {  // memory is contiguous along the rows of a column
        for (int l = warp; l < nb - 1; l += C::NW)
            for (int b = 0; b < S; b++) {
                double2 *dst = coef + C::off(l) + b * (NR - (l + 1) * S);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int x = lane + 32 * t, r = (l + 1) * S + x;
                    if (r < NRb) cp16(dst + x, vol_t<S, RET>(g, n, i0 + r / S, i0 + l, r % S, b));
                }
            }
    } else {  // memory is contiguous along the columns of a row
        for (int r = S + warp; r < NRb; r += C::NW) {
            const int rt = r / S, a = r % S;
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int x = lane + 32 * t, l = x / S, b = x % S;
                if (x < rt * S)
                    cp16(coef + C::off(l) + b * (NR - (l + 1) * S) + r - (l + 1) * S, vol_t<S, RET>(g, n, i0 + rt, i0 + l, a, b));
            }
        }
    }
    for (int e = tid; e < K1 * S * K1 * S; e += NTH) {
        const int x = RET ? e / (K1 * S) : e % (K1 * S), r = RET ? e % (K1 * S) : e / (K1 * S);
        const bool in = r < NRb && r / S + K1 - x / S <= k;
        cp16(near_ + x * C::NEAR + r, in ? vol_t<S, RET>(g, n, i0 + r / S, i0 - K1 + x / S, r % S, x % S) : nullptr);
    }
    double2 Dr[C::NC][4];  // s = 1: the step inverses of the warp's columns
    if constexpr (S == 1) {
#pragma unroll
        for (int c = 0; c < C::NC; c++)
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int q = c0 + warp * nc + c, i = i0 + lane + 32 * t;
                Dr[c][t] = cmk(0, 0);
                if (warp * nc + c < ncol && c < nc && i <= n) Dr[c][t] = RET ? probs[q].minv_ret[n - i] : probs[q].minv_les[i];
            }
    } else {
        for (int q = p0; q <= (c0 + ncol - 1) / S; q++) {
            const double2 *mi = RET ? probs[q].minv_ret : probs[q].minv_les;
            for (int e = tid; e < nb * s2; e += NTH) {
                const int l = e / s2, a = (e % s2) / S, b = e % S;
                cp16(dm + (q - p0) * NR * S + (RET ? l * s2 + b * S + a : e), mi + (long)(RET ? n - i0 - l : i0 + l) * s2 + a * S + b);
            }
        }
    }
    cp_commit();
    for (int e = tid; e < 32 + C::NBT + 1; e += NTH) bdp[e] = e > 32 && e - 32 <= K1 ? bd_w(k, e - 32) / h : 0.0;
    if (tid <= NESSI_K1MAX) wdx[tid] = tid <= k ? greg_omega(k, tid) : 1.0;
    cp_wait<0>();
    __syncthreads();
    // weights: a_delta on the k rows below the diagonal, g h (a_delta - 1) on the near block
    for (int l = warp; l < nb - 1; l += C::NW) {
        const int len = NR - (l + 1) * S;
        double2 *col = coef + C::off(l);
        for (int b = 0; b < S; b++)
            for (int x = lane; x < k * S; x += 32)
                if ((l + 1) * S + x < NRb) col[b * len + x] = cscale(col[b * len + x], wdx[x / S + 1]);
    }
    for (int e = tid; e < K1 * S * K1 * S; e += NTH) {
        const int x = e / (K1 * S), r = e % (K1 * S), delta = r / S + K1 - x / S;
        if (delta <= k) near_[x * C::NEAR + r] = cscale(near_[x * C::NEAR + r], gh * (wdx[delta] - 1.0));
    }
    pdl_wait();  // from here on the results of the kernels before
    // ---- right-hand sides: q_i + g h (far sum of the rows above)
    constexpr int RI = (NR * C::WMAX + NTH - 1) / NTH;
    {
        double2 far[RI], q[RI];
#pragma unroll
        for (int x = 0; x < RI; x++) {
            const int e = tid + x * NTH, w = e & (wc - 1), r = e >> lw, i = i0 + r / S, a = r % S, c = c0 + w;
            far[x] = q[x] = cmk(0, 0);
            if (r >= NRb || w >= ncol) continue;
            far[x] = __ldcg(g.vacc + ((long)i * S + a) * ldc + c);
            if (!RET) q[x] = __ldcg(g.gles + ((long)i * S + a) * ldc + c);
            if (VIE) {
                const ProbDev &p = probs[c / S];
                q[x] = cadd(q[x], RET ? p.qret[(tri(n) + n - i) * s2 + (c % S) * S + a] : p.qles[(tri(n) + i) * s2 + a * S + c % S]);
            }
        }
        const double2 *ysrc = blk > 0 ? g.vy + (long)(i0 - K1) * S * ldc : g.vst;
        for (int e = tid; e < (K1 * S) << lw; e += NTH) {
            const int w = e & (wc - 1), x = e >> lw;
            if (w < ncol) ynear[w * C::NEAR + x] = __ldcg(ysrc + (long)x * ldc + c0 + w);
        }
#pragma unroll
        for (int x = 0; x < RI; x++) {
            const int e = tid + x * NTH, w = e & (wc - 1), r = e >> lw;
            if (r < NRb && w < ncol) buf[w * C::NRP + r] = cmk(fma(gh, far[x].x, q[x].x), fma(gh, far[x].y, q[x].y));
        }
    }
    __syncthreads();
    // row r of column w: the right-hand side with the near rows (weights and backward differences)
    auto rhs = [&](int w, int r) {
        double2 v = buf[w * C::NRP + r];
        if (r < K1 * S) {
            const double2 *y = ynear + w * C::NEAR;
            const int l0 = r / S;
            double2 o = cmk(0, 0);
            for (int x = l0 * S; x < K1 * S; x++) o = cfma(near_[x * C::NEAR + r], y[x], o);
            v = cadd(v, o);
            if (!VIE)
                for (int l = l0; l < K1; l++) v = sub_ib(v, bdp[32 + l0 + K1 - l], y[l * S + r % S]);
        }
        return v;
    };
    if constexpr (S <= 2) {
        if (warp * nc < ncol) {
            double2 acc[C::NC][4];
            double2 *xs = buf + warp * nc * C::NRP;
#pragma unroll
            for (int cc = 0; cc < C::NC; cc++)
#pragma unroll
                for (int t = 0; t < 4; t++)
                    acc[cc][t] = cc < nc && warp * nc + cc < ncol && lane + 32 * t < NRb ? rhs(warp * nc + cc, lane + 32 * t) : cmk(0, 0);
            __syncwarp();
            if constexpr (S == 1) {
                vol_chain1<VIE>(acc[0], coef, Dr[0], bdp, gh, K1, nb, xs, lane);
            } else {  // two columns of a warp are one problem's
                const double2 *D = dm + ((c0 + warp * nc) / S - p0) * NR * S;
                if (nc == 2) vol_chain2<VIE, 2>(acc, coef, D, bdp, gh, K1, nb, xs, lane);
                else vol_chain2<VIE, 1>(acc, coef, D, bdp, gh, K1, nb, xs, lane);
            }
        }
    } else {
        const int w = warp >> 2, slot = warp & 3, r = slot * C::SR + lane;
        double2 acc = w < ncol && lane < C::SR && r < NRb ? rhs(w, r) : cmk(0, 0);
        __syncthreads();
        if (w < ncol)
            vol_chain_big<S, VIE>(acc, coef, dm + ((c0 + w) / S - p0) * NR * S, bdp, gh, nb, buf + w * C::NRP,
                                  smem + C::qs(wc) + w * S, slot, lane, 1 + w);
    }
    __syncthreads();
    // ---- results: vy (rows x columns, for the trailing GEMM), ret: the operand of les*adv
    //      badv(m) = h w(n, m) G^R(n, m)^dagger, and G's own row / column
    const bool more = i0 + nb <= n;
#pragma unroll
    for (int x = 0; x < RI; x++) {
        const int e = tid + x * NTH, w = e & (wc - 1), r = e >> lw, i = i0 + r / S, a = r % S;
        if (r >= NRb || w >= ncol) continue;
        const double2 v = buf[w * C::NRP + r];
        if (more) g.vy[((long)i * S + a) * ldc + c0 + w] = v;
        if (RET) g.badv[((long)(n - i) * S + a) * ldc + c0 + w] = cscale(cconj(v), h * greg_w(k, n, n - i));
    }
    for (int w = warp; w < ncol; w += C::NW) {
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
    // blk = -1: the start rows 0..k
    const int l0 = blk < 0 ? 0 : g.k + 1 + blk * VbCfg<S>::NBT, i1 = g.k + 1 + (blk + 1) * VbCfg<S>::NBT;
    const int M = (n - i1 + 1) * S;
    K = (i1 - l0) * S;
    la = LdVolT<S, RET>{RET ? g.rret : g.sret, n, i1, l0, M, K};
    lb = LdRowN{g.vy + (long)l0 * S * g.ldc, g.ldc, K, cols};
    st = StRow{g.vacc + (long)i1 * S * g.ldc, g.ldc, M, cols, 1.0, blk >= 0};
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
    pdl_trigger();
    if (!vol_trail_operands<S, RET>(g, cols, n, blk, la, lb, st, K)) return;
    if ((int)blockIdx.x * 32 >= cols || (int)blockIdx.y * 32 >= la.M) return;
    pdl_wait();
    zgemm_pipe<32, 32>(la, lb, st, blockIdx.y * 32, blockIdx.x * 32, K, smem);
}
template <int S, bool RET>
__global__ void __launch_bounds__(256, 2) k_vol_trail_split(const GroupDev *__restrict__ gt, GroupSel sel, int n, int blk) {
    __shared__ double2 red[8 * 32 * 8];
    const GroupDev &g = gt[sel.gid[blockIdx.z]];
    const int cols = sel.nact[blockIdx.z] * S;
    LdVolT<S, RET> la;
    LdRowN lb;
    StRow st;
    int K;
    pdl_trigger();
    if (!vol_trail_operands<S, RET>(g, cols, n, blk, la, lb, st, K)) return;
    if ((int)blockIdx.x * 8 >= cols || (int)blockIdx.y * 32 >= la.M) return;
    pdl_wait();
    zgemm_split(la, lb, st, blockIdx.y * 32, blockIdx.x * 8, K, red);
}

// ---- start rows i = 0..k, one CTA per problem (grid (problems, groups)) --------------------------
// ret: G(n, n) = -i (Dyson) or Q(n, n) (VIE2), then the k-block start G(n, n-1..n-k)
// (dyson_impl :112-157, vie2_impl :60-100)
template <int S, bool VIE>
__global__ void __launch_bounds__(256) k_ret_start(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    extern __shared__ double2 smem[];
    constexpr int s2 = S * S;
    pdl_wait();     // before the trigger: k_vol_block reads the step matrices without waiting again
    pdl_trigger();
    if ((int)blockIdx.x >= sel.nact[blockIdx.y]) return;
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const ProbDev p = g.probs[blockIdx.x];
    const int k = g.k;
    const long ldc = g.ldc;
    double2 *grow = p.gret + tri(n) * s2;
    for (int e = threadIdx.x; e < s2; e += blockDim.x)
        grow[(long)n * s2 + e] = VIE ? p.qret[(tri(n) + n) * s2 + e] : (e / S == e % S ? cmk(0.0, -1.0) : cmk(0, 0));
    __syncthreads();
    ret_start_block<S, VIE>(g, p, n, smem);
    for (int e = threadIdx.x; e < (k + 1) * s2; e += blockDim.x) {
        const int l = e / s2, b = (e % s2) / S, d = e % S;  // Y_l[b][d] = G(n, n-l)[d][b]
        const double2 y = grow[(long)(n - l) * s2 + d * S + b];
        g.vy[((long)l * S + b) * ldc + p.col * S + d] = cscale(y, greg_omega(k, l));
        g.vst[((long)l * S + b) * ldc + p.col * S + d] = y;
        g.badv[((long)(n - l) * S + b) * ldc + p.col * S + d] = cscale(cconj(y), g.h * greg_w(k, n, n - l));
    }
}

// les: G^<(0, n) = -G^tv(n, 0)^dagger and the k-block start G^<(1..k, n) (dyson_impl :926-982), or
// the VIE2 start G^<(0..k, n) (vie2_impl :847-900); gl = the Sigma-shared products in g.gles.
template <int S, bool VIE>
__global__ void __launch_bounds__(256) k_les_start(const GroupDev *__restrict__ gt, GroupSel sel, int n) {
    extern __shared__ double2 smem[];
    constexpr int s2 = S * S;
    pdl_wait();     // before the trigger: k_vol_block reads the step matrices without waiting again
    pdl_trigger();
    if ((int)blockIdx.x >= sel.nact[blockIdx.y]) return;
    const GroupDev &g = gt[sel.gid[blockIdx.y]];
    const ProbDev p = g.probs[blockIdx.x];
    const int k = g.k;
    const long ldc = g.ldc;
    const double2 *gl = g.gles + (long)p.col * S;
    double2 *xcol = p.gles + tri(n) * s2;
    if (!VIE) {
        for (int ad = threadIdx.x; ad < s2; ad += blockDim.x) {
            const int a = ad / S, d = ad % S;
            xcol[ad] = cneg(cconj(p.gtv[((long)n * s2 + d * S + a) * (g.ntau + 1) + 0]));
        }
        __syncthreads();
    }
    les_start_block<S, VIE>(g, p, n, gl, ldc, xcol, smem);
    for (int e = threadIdx.x; e < (k + 1) * s2; e += blockDim.x) {
        const int l = e / s2, b = (e % s2) / S, d = e % S;
        g.vy[((long)l * S + b) * ldc + p.col * S + d] = cscale(xcol[e], greg_omega(k, l));
        g.vst[((long)l * S + b) * ldc + p.col * S + d] = xcol[e];
    }
}
